"""GPU: fused_moe with few rows per expert, at the edges of its row boxes (32), tile widths and of the rule itself."""
import pytest
import torch

from dlcompiler_b200 import fused_moe
from oracle import dlblas_oracle as oracle

pytestmark = pytest.mark.gpu


# rows per expert around 32 / 64 / 96 / 128; intermediate and hidden sizes that leave ragged tiles at every width;
# 16 experts x 4000 columns take a narrower tile, 2 experts x 1000 rows are past the rule (whole boxes, zero padding)
@pytest.mark.parametrize("rows,hidden,inter,dtype", [
    ([1, 31, 32, 33, 0, 64, 65, 97], 128, 200, torch.bfloat16),
    ([128, 129, 2, 96, 127, 63, 0, 5], 136, 328, torch.float16),
    ([3] * 16, 64, 4000, torch.bfloat16),
    ([1], 512, 1160, torch.bfloat16),                     # a handful of tiles: the narrowest width
    ([1000, 1000], 64, 72, torch.bfloat16),
])
def test_rows_and_widths(cuda_device, rows, hidden, inter, dtype):
    g = torch.Generator().manual_seed(len(rows) + hidden)
    E, T = len(rows), sum(rows)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(T, generator=g)].view(T, 1)
    x = torch.randn(T, hidden, generator=g).to(dtype)
    w1 = (torch.randn(E, 2 * inter, hidden, generator=g) * 0.1).to(dtype)
    w2 = (torch.randn(E, hidden, inter, generator=g) * 0.1).to(dtype)
    weights = torch.rand(T, 1, generator=g)
    out = fused_moe(*(t.to(cuda_device) for t in (x, w1, w2, weights, ids)), 1)
    ref = oracle.fused_moe_rounding_faithful(x, w1, w2, weights, ids)
    # stated bound of the block in 16 bits: 4 ulp of bf16 against the rounding-faithful oracle
    torch.testing.assert_close(out.cpu().float(), ref.float(), rtol=2e-2, atol=2e-2 * float(ref.float().std()))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_silu_over_its_range(cuda_device, dtype):
    """The activation from one end of its range to the other: hidden state 1, gate weights the values, up weights 1 and
    an identity behind it give silu(value).  Two roundings to the type; below 2^-24 only the size is left to compare."""
    values = torch.cat([torch.linspace(-104, 104, 833), torch.tensor([-6e4, -500., -88.8, -87.4, 0., 1e-4, 500., 6e4])])
    n = values.numel() // 8 * 8
    values = values[-n:].to(dtype)
    w1 = torch.zeros(1, 2 * n, 8)
    w1[0, :n, 0], w1[0, n:, 0] = values.float(), 1.0
    x = torch.zeros(1, 8)
    x[0, 0] = 1.0
    one = torch.ones(1, 1, device=cuda_device)
    out = fused_moe(x.to(dtype).to(cuda_device), w1.to(dtype).to(cuda_device),
                    torch.eye(n).unsqueeze(0).to(dtype).to(cuda_device), one, one.long() * 0, 1)
    ref = torch.nn.functional.silu(values.double())
    torch.testing.assert_close(out[0].cpu().double(), ref, rtol=2 * torch.finfo(dtype).eps, atol=2.0 ** -24)
