"""GPU: the orders in which the prefill kernel goes through its tiles, each at the edge of its rule."""
import pytest
import torch

from dlcompiler_b200 import context_attention_fwd, paged_attention_fwd
from oracle import dlblas_oracle as oracle

pytestmark = pytest.mark.gpu

RTOL = ATOL = 2e-2      # bf16 attention outputs


def _case(lens, hq, hkv, dim, seed):
    g = torch.Generator().manual_seed(seed)
    total = sum(lens)
    q, k, v = (torch.randn(total, h, dim, generator=g).to(torch.bfloat16) for h in (hq, hkv, hkv))
    ends = torch.tensor(lens).cumsum(0)
    return q, k, v, (ends - torch.tensor(lens)).to(torch.int32), torch.tensor(lens, dtype=torch.int32)


@pytest.mark.parametrize("lens,dim", [
    ([5, 900, 0, 130, 1, 257, 128, 640, 33, 129, 400, 64, 0], 128),     # ragged, tiles that do not exist
    ([7 * i % 300 + 1 for i in range(31)] + [1500], 64),                # ragged, one sequence per lane
    ([7 * i % 300 + 1 for i in range(32)] + [1500], 64),                # ragged, more than a warp can sort
    ([384, 384, 384, 300], 128),                                        # about the same length: row tiles first
    ([96], 128),                                                        # a tile whose last warp has no row
])
def test_varlen_orders(cuda_device, lens, dim):
    q, k, v, start, n = _case(lens, 6, 2, dim, len(lens))
    o = torch.full_like(q, float("nan")).to(cuda_device)
    lse = torch.full((6, q.shape[0]), float("nan"), device=cuda_device)
    context_attention_fwd(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), o, start.to(cuda_device),
                          n.to(cuda_device), max(lens), lse=lse)
    ref, rlse = oracle.context_attention(q, k, v, start, n, return_lse=True)
    torch.testing.assert_close(o.cpu().float(), ref.float(), rtol=RTOL, atol=ATOL)
    torch.testing.assert_close(lse.cpu(), rlse, rtol=1e-3, atol=1e-3)


@pytest.mark.parametrize("dim", [128, 64, 72, 24])
@pytest.mark.parametrize("rows", [1, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 192, 193])
def test_epilogue_by_rows_of_the_tile(cuda_device, rows, dim):
    """Both ways out of a tile at their edges (at most 64 rows: a row per lane; more: staged), into a strided output
    whose other columns and rows stay as they are."""
    q, k, v, start, n = _case([rows], 4, 2, dim, rows)
    wide = torch.full((rows + 3, 4, dim + 8), 7.0, dtype=torch.bfloat16, device=cuda_device)
    o = wide[:rows, :, :dim]
    context_attention_fwd(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), o, start.to(cuda_device),
                          n.to(cuda_device), rows)
    ref = oracle.context_attention(q, k, v, start, n)
    torch.testing.assert_close(o.cpu().float(), ref.float(), rtol=RTOL, atol=ATOL)
    assert (wide[rows:] == 7).all() and (wide[:, :, dim:] == 7).all()


def _each_as_if_alone(cuda_device, batch, history):
    """A sequence attends to its own keys only, so every one must equal a launch of its own (which starts all tiles at
    once)."""
    hq, hkv, dim, page = 32, 8, 64, 16
    lens = [150 if i % 3 else 40 for i in range(batch)]
    full = [n + history(i) for i, n in enumerate(lens)]
    q, _, _, start, n = _case(lens, hq, hkv, dim, batch)
    g = torch.Generator().manual_seed(1)
    pages = [(m + page - 1) // page for m in full]
    kc, vc = (torch.randn(sum(pages), page, hkv, dim, generator=g).to(torch.bfloat16).to(cuda_device) for _ in range(2))
    table = torch.zeros(batch, max(pages), dtype=torch.int32)
    order = torch.randperm(sum(pages), generator=g).to(torch.int32)
    for b in range(batch):
        table[b, :pages[b]] = order[sum(pages[:b]):sum(pages[:b + 1])]
    q, table, kv = q.to(cuda_device), table.to(cuda_device), torch.tensor(full, dtype=torch.int32, device=cuda_device)
    o = torch.full_like(q, float("nan"))
    paged_attention_fwd(q, kc, vc, o, table, start.to(cuda_device), n.to(cuda_device), kv, max(lens))
    for b in range(batch):
        rows = slice(int(start[b]), int(start[b]) + lens[b])
        alone = torch.empty_like(q[rows])
        paged_attention_fwd(q[rows], kc, vc, alone, table[b:b + 1], torch.zeros(1, dtype=torch.int32, device=cuda_device),
                            n[b:b + 1].to(cuda_device), kv[b:b + 1], lens[b])
        assert torch.equal(o[rows], alone)


@pytest.mark.parametrize("batch", [5, 32, 33])
def test_paged_sequences_by_length(cuda_device, batch):
    """More tiles than the GPU holds at once, in the order of the batch (short histories)."""
    _each_as_if_alone(cuda_device, batch, lambda i: (37 * i) % 200)


@pytest.mark.parametrize("batch", [5, 31, 32, 33])
@pytest.mark.parametrize("history", ["about the same", "far apart", "equal pairs"])
def test_paged_long_histories(cuda_device, batch, history):
    """A table with room for long histories: up to 32 sequences by descending key count, or as they are when their lengths
    are within a quarter."""
    _each_as_if_alone(cuda_device, batch, {"about the same": lambda i: 900 + i, "far apart": lambda i: (397 * i) % 1700,
                                           "equal pairs": lambda i: 1200 * (i // 2 % 2)}[history])
