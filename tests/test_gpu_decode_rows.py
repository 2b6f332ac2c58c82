"""GPU: decode_attention_fwd through its table's rows: any order, repeated, either index type, a table that is a view."""
import pytest
import torch

from dlcompiler_b200 import check_device_status, decode_attention_fwd
from dlcompiler_b200._lib import DlblasError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idx_dtype", [torch.int32, torch.int64, torch.int16])
@pytest.mark.parametrize("transposed", [False, True])
def test_rows_of_the_table(cuda_device, idx_dtype, transposed):
    """Bit for bit what a table gathered beforehand and read in order gives."""
    g = torch.Generator().manual_seed(3)
    rows, ctx, hq, hkv, dim = 7, 700, 8, 2, 64
    pool = torch.randperm(rows * ctx, generator=g).to(torch.int32).view(rows, ctx).to(cuda_device)
    k, v = (torch.randn(rows * ctx, hkv, dim, generator=g).to(torch.bfloat16).to(cuda_device) for _ in range(2))
    idx = torch.tensor([6, 0, 3, 3, 5])
    lens = torch.tensor([700, 1, 65, 512, 256], dtype=torch.int32, device=cuda_device)
    q = torch.randn(5, hq, dim, generator=g).to(torch.bfloat16).to(cuda_device)
    table = pool.t().contiguous().t() if transposed else pool
    out, ref = torch.empty_like(q), torch.empty_like(q)
    decode_attention_fwd(q, k, v, out, table, idx.to(idx_dtype).to(cuda_device), None, lens, None, ctx, 0.125)
    decode_attention_fwd(q, k, v, ref, pool[idx.to(cuda_device)].contiguous(), torch.arange(5, device=cuda_device), None,
                         lens, None, ctx, 0.125)
    assert torch.isfinite(out.float()).all() and torch.equal(out, ref)


@pytest.mark.parametrize("ctx", [64, 4000])             # one split, and the merge of several
@pytest.mark.parametrize("bad,idx_dtype", [(-1, torch.int32), (7, torch.int32), (-1, torch.int64), (7, torch.int64),
                                           (2 ** 32 + 3, torch.int64), (-2 ** 40, torch.int64)])
def test_row_outside_the_table(cuda_device, bad, idx_dtype, ctx):
    """No other request's tokens: zeros for that request, an error for the call, the other requests as without it."""
    g = torch.Generator().manual_seed(5)
    rows, hq, hkv, dim = 7, 8, 2, 64
    pool = torch.randint(0, 5000, (rows, ctx), generator=g, dtype=torch.int32).to(cuda_device)
    k, v = (torch.randn(5000, hkv, dim, generator=g).to(torch.bfloat16).to(cuda_device) for _ in range(2))
    q = torch.randn(3, hq, dim, generator=g).to(torch.bfloat16).to(cuda_device)
    lens = torch.tensor([ctx, ctx - 1, ctx // 2], dtype=torch.int32, device=cuda_device)
    outs = []
    for idx in ([6, 3, 0], [6, bad, 0]):
        o = torch.full_like(q, 7.0)
        decode_attention_fwd(q, k, v, o, pool, torch.tensor(idx, dtype=idx_dtype, device=cuda_device), None, lens, None,
                             ctx, 0.125)
        outs.append(o)
        if bad in idx:
            with pytest.raises(DlblasError, match="request 1 .* table of 7"):
                check_device_status()
        check_device_status()
    assert torch.equal(outs[1][1], torch.zeros_like(q[1]))
    assert torch.equal(outs[1][[0, 2]], outs[0][[0, 2]])


@pytest.mark.parametrize("kind", ["int16", "transposed", "every other column"])
def test_table_that_needs_a_copy(cuda_device, kind):
    """Bit for bit the table in its plain form, only the rows and columns in use copied: less new memory than the pool."""
    g = torch.Generator().manual_seed(9)
    rows, ctx, cols = 512, 300, 4096
    pool = torch.randint(0, 5000, (rows, cols), generator=g, dtype=torch.int32).to(cuda_device)
    table = {"int16": pool.to(torch.int16), "transposed": pool.t().contiguous().t(),
             "every other column": pool.repeat_interleave(2, 1)[:, ::2]}[kind]
    k, v = (torch.randn(5000, 2, 64, generator=g).to(torch.bfloat16).to(cuda_device) for _ in range(2))
    q = torch.randn(4, 8, 64, generator=g).to(torch.bfloat16).to(cuda_device)
    lens = torch.tensor([ctx, 1, 65, 257], dtype=torch.int32, device=cuda_device)
    idx = torch.tensor([511, 0, -1, 511], device=cuda_device)
    outs = []
    for t in (pool, table):
        o = torch.empty_like(q)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        held = torch.cuda.memory_allocated()
        decode_attention_fwd(q, k, v, o, t, idx, None, lens, None, ctx, 0.125)
        assert torch.cuda.max_memory_allocated() - held < rows * cols
        with pytest.raises(DlblasError, match="request 2 "):
            check_device_status()
        outs.append(o)
    assert torch.equal(outs[0], outs[1]) and not outs[0][2].any()
