"""GPU: the cluster-wide slot sort at the edges of its cluster sizes, segments and expert counts (integers: exact)."""
import pytest
import torch

from dlcompiler_b200 import topk_gating
from dlcompiler_b200.kernels.fused_moe import _moe_align
from oracle import dlblas_oracle as oracle

pytestmark = pytest.mark.gpu


# one CTA up to 2048 slots, then 2, 4 and 8; segments are whole rounds of 32 slots per warp
@pytest.mark.parametrize("numel", [1, 31, 33, 2048, 2049, 4096, 4097, 8192, 8193, 33000])
@pytest.mark.parametrize("E,block", [(1, 16), (33, 1), (256, 128), (1024, 8)])
def test_sort_at_cluster_edges(cuda_device, numel, E, block):
    g = torch.Generator().manual_seed(numel + E)
    ids = torch.randint(-1, E + 2, (numel,), generator=g, dtype=torch.int32)      # some belong to no expert here
    got = _moe_align(ids.to(cuda_device), block, E)
    for a, b in zip(got, oracle.moe_align_block_size(ids, block, E)):
        assert torch.equal(a.cpu(), b)


@pytest.mark.parametrize("S,E,k,cf", [(1, 4, 1, 1.0), (7, 8, 8, 1.0), (2049, 4, 1, 2.0), (5000, 16, 4, 2.0),
                                      (3001, 512, 2, 1.25), (16384, 8, 2, 1.25)])
def test_gate_at_cluster_edges(cuda_device, S, E, k, cf):
    """Half-empty capacity lists (cf = 2), a ragged last CTA, one and eight CTAs, four warps per CTA (E > 256)."""
    g = torch.Generator().manual_seed(S + E)
    logits = torch.randn(S, E, generator=g)
    l_aux, ec, w, sel = topk_gating(logits.to(cuda_device), k, cf, 1)
    rl, rec, rw, rsel, _ = oracle.topk_gating(logits, k, cf, 1)
    assert torch.equal(ec.cpu(), rec) and torch.equal(sel.cpu(), rsel)
    torch.testing.assert_close(l_aux.cpu(), rl, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(w.cpu(), rw, rtol=1e-5, atol=1e-7)
