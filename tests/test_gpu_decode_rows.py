"""GPU: decode_attention_fwd through its table's rows: any order, repeated, either index type, a table that is a view."""
import pytest
import torch

from dlcompiler_b200 import decode_attention_fwd

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
