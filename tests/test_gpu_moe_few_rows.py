"""GPU: fused_moe with few rows per expert, at the edges of its row boxes (32), tile widths and of the rule itself."""
import pytest
import torch

from dlcompiler_b200 import _lib, fused_moe
from dlcompiler_b200.kernels.fused_moe import _grouped_gemm
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
    """The activation from -6e4 to 6e4 through the whole block: hidden state 1, gate weights the values, up weights 1 and
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


@pytest.mark.parametrize("few", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_silu_of_every_value(cuda_device, dtype, few):
    """The activation of all 65536 gates of the type, straight from the GEMM that fuses it, up = 1.  Where e^-x leaves
    fp32 (x < -88.73) the quotient is -0, whatever the size of x, and NaN at -inf; elsewhere two roundings to the type and
    the relative error of exp's fp32 argument (|x| 2^-24, below 2^-17)."""
    gates = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(dtype)
    n = gates.numel()
    w1 = torch.zeros(1, 2 * n, 8, dtype=dtype)
    w1[0, :n, 0], w1[0, n:, 0] = gates, 1.0
    a = torch.zeros(128, 8, dtype=dtype)
    a[0, 0] = 1.0
    numel = 1 if few else 128            # the padding's share picks the kernel's form
    ids = torch.full((128,), numel, dtype=torch.int32)
    ids[0] = 0
    out = torch.zeros(128, n, dtype=dtype, device=cuda_device)
    _grouped_gemm(a.to(cuda_device), w1.to(cuda_device), out, n, ids.to(cuda_device),
                  torch.tensor([0, 1], dtype=torch.int32, device=cuda_device), None, numel,
                  _lib.GEMM_FUSE_SILU | _lib.GEMM_SLOTS_ONLY)
    got, x = out[0].cpu().double(), gates.double()
    ref = torch.nn.functional.silu(x)
    gone = x < -88.73
    assert torch.equal(got[gone & torch.isfinite(x)], ref.new_zeros(int((gone & torch.isfinite(x)).sum())))
    assert torch.isnan(got[x == -torch.inf]).all() and torch.isnan(got[torch.isnan(x)]).all()
    assert (got[x == torch.inf] == torch.inf).all()
    rest = torch.isfinite(x) & ~gone
    # the smallest normal number as the floor: the tensor cores may take a subnormal operand as zero
    torch.testing.assert_close(got[rest], ref[rest], rtol=2 * torch.finfo(dtype).eps + 2.0 ** -17,
                               atol=torch.finfo(dtype).tiny)


def test_c_entries_keep_the_rows_of_no_slot(cuda_device):
    """Called without SLOTS_ONLY the GEMM stores every row of its blocks, whatever sorted_token_ids holds, and the permute
    writes zeros for the sentinel rows, however many there are."""
    g = torch.Generator().manual_seed(2)
    lib, stream = _lib.load(), _lib.stream_ptr(cuda_device)
    a = torch.randn(256, 64, generator=g).to(torch.bfloat16).to(cuda_device)
    w = (torch.randn(2, 2 * 40, 64, generator=g) * 0.2).to(torch.bfloat16).to(cuda_device)
    starts = torch.tensor([0, 1, 2], dtype=torch.int32, device=cuda_device)
    nobody = torch.full((256,), 1 << 30, dtype=torch.int32, device=cuda_device)
    out = torch.full((256, 40), float("nan"), dtype=torch.bfloat16, device=cuda_device)
    _grouped_gemm(a, w, out, 40, nobody, starts, None, 1, _lib.GEMM_FUSE_SILU)
    h = torch.einsum("erk,enk->ern", a.view(2, 128, 64).float(), w.float()).to(torch.bfloat16).float()
    gate = torch.nn.functional.silu(h[..., :40]).to(torch.bfloat16).float()
    ref = (gate * h[..., 40:]).view(256, 40)
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2 * float(ref.std()))
    ids = torch.full((256,), 9, dtype=torch.int32, device=cuda_device)
    ids[3], ids[130] = 8, 0
    post = torch.tensor([256], dtype=torch.int32, device=cuda_device)
    for entry, untouched in ((lib.dlb_moe_permute_rows, False), (lib.dlb_moe_permute_slots, True)):
        dst = torch.full((256, 64), 7.0, dtype=torch.bfloat16, device=cuda_device)
        _lib.check(entry(a.data_ptr(), dst.data_ptr(), ids.data_ptr(), post.data_ptr(), 9, 1, 64, 64, 256, 2, stream), "permute")
        assert torch.equal(dst[3], a[8]) and torch.equal(dst[130], a[0])
        dst[3] = dst[130] = 7.0 if untouched else 0.0
        assert (dst == (7.0 if untouched else 0.0)).all()
