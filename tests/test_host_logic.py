"""Host-side rules that need no GPU: the decode split-size rule and its environment override, the padded
capacity of moe_align_block_size."""


def test_decode_split_size_rule(monkeypatch):
    from dlcompiler_b200.kernels import paged_attention as pa

    monkeypatch.delenv("DLBLAS_B200_DECODE_CHUNK", raising=False)
    # C5: 64 sequences x 8 kv heads x up to 32768 tokens -> the longest split the rule allows
    assert pa._pick_chunk(64, 8, 32768, 64) == 4096
    # 16 sequences: about 4 waves of CTAs
    assert pa._pick_chunk(16, 8, 32768, 64) == 2048
    # tiny problems: never below one 256-token split, never below a page
    assert pa._pick_chunk(1, 1, 100, 16) == 256
    assert pa._pick_chunk(1, 1, 100, 1024) == 1024
    for b, h, c, p in [(3, 2, 5000, 32), (128, 8, 2048, 16), (7, 1, 70000, 128)]:
        chunk = pa._pick_chunk(b, h, c, p)
        assert chunk & (chunk - 1) == 0 and chunk % 64 == 0 and chunk % min(p, chunk) == 0
    monkeypatch.setenv("DLBLAS_B200_DECODE_CHUNK", "300")
    assert pa._pick_chunk(64, 8, 32768, 64) == 512          # rounded up to a power of two
    monkeypatch.setenv("DLBLAS_B200_DECODE_CHUNK", "64")
    assert pa._pick_chunk(64, 8, 32768, 256) == 256         # never below a page


def test_align_capacity_covers_the_worst_case():
    from dlcompiler_b200.kernels.fused_moe import _align_capacity

    for numel, experts, block in [(8192, 8, 128), (1, 4, 128), (0, 3, 16), (1000, 256, 64), (77, 7, 1)]:
        cap = _align_capacity(numel, experts, block)
        assert cap % block == 0
        assert cap >= numel + experts * (block - 1)          # every expert may waste block - 1 entries
        assert cap - (numel + experts * (block - 1)) < block



def test_decode_attention_refuses_what_names_no_row(monkeypatch):
    """Before any launch: a two-dimensional b_req_idx, too few of them, a table without columns."""
    import pytest
    import torch

    from dlcompiler_b200 import _lib
    from dlcompiler_b200.kernels.decode_attention import decode_attention_fwd

    monkeypatch.setattr(_lib, "require_cuda", lambda *t: torch.device("cpu"))
    monkeypatch.setattr(_lib, "load", lambda: pytest.fail("not refused"))
    q, kv, table = torch.zeros(4, 8, 64), torch.zeros(16, 2, 64), torch.zeros(3, 16, dtype=torch.int32)
    lens = torch.ones(4, dtype=torch.int32)
    for t, idx in ((table, torch.zeros(2, 2, dtype=torch.int32)), (table, torch.zeros(3, dtype=torch.int32)),
                   (table[:, :0], torch.zeros(4, dtype=torch.int32))):
        with pytest.raises(AssertionError, match="b_req_idx|columns"):
            decode_attention_fwd(q, kv, kv, q, t, idx, None, lens, None, 16, 0.125)


def test_gate_capacity_is_the_tensor_arithmetic():
    """The fp32 product of the tensor form, rounding, infinities, NaN and refusals included."""
    import math
    import random

    import pytest
    import torch

    from dlcompiler_b200.kernels.topk_gating import _capacity

    def tensor_form(tokens, experts, factor, least):
        return max(int(torch.ceil((tokens / experts) * torch.tensor(factor)).to(torch.int64)), int(least))

    r = random.Random(0)
    cases = [(64, 8, f, 4) for f in (math.inf, -math.inf, math.nan, 1e30, -1e30, 1e300, 2.0**31, 9.3e18, -3.0, 0.0, 2, True)]
    cases += [(r.randint(1, 1 << r.randint(1, 21)), r.randint(1, 512), r.choice([r.random() * 8, r.randint(1, 32) * 1.1,
                                                                                r.randint(1, 32) / 3, 1.25]), 2)
              for _ in range(3000)]
    for case in cases:
        assert _capacity(*case) == tensor_form(*case), case
    with pytest.raises(ValueError):
        _capacity(64, 8, 2**70, 4)
