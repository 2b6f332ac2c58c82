"""GPU: the cluster-wide slot sort at the edges of its cluster sizes, segments and expert counts (integers: exact)."""
import threading
from ctypes import c_int, c_int64, c_void_p

import pytest
import torch

from dlcompiler_b200 import _lib, topk_gating
from dlcompiler_b200.kernels.fused_moe import _align_capacity, _moe_align
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


@pytest.mark.parametrize("S,E,k,capacity,blocks", [(1, 4, 1, 1, 1), (37, 8, 8, 5, 7), (4096, 64, 8, 640, 64), (3001, 512, 2, 3, 3001),
                                                   (20000, 40, 4, 3000, 256)])
def test_gate_then_assign_is_the_forward(cuda_device, S, E, k, capacity, blocks):
    """The two-step C entries against the one the wrapper calls: the same choices, queues, lists and weights; the column
    means are added in another order (fp32 sums of S values in [0, 1])."""
    lib, stream = _lib.load(), _lib.stream_ptr(cuda_device)
    x = torch.randn(S, E, generator=torch.Generator().manual_seed(S)).to(cuda_device)

    def buffers():
        new = lambda n, dt: torch.full((n,), -7, dtype=dt, device=cuda_device)      # noqa: E731
        return [new(k * S, torch.int32), new(E, torch.float32), new(E, torch.float32), new(1, torch.float32),
                new(k * S, torch.int32), new(k * S, torch.float32), new(E * capacity, torch.int64)]

    gates, gates2 = torch.empty_like(x), torch.empty_like(x)
    ids, ids_km = (torch.empty(S * k, dtype=torch.int32, device=cuda_device) for _ in range(2))
    scratch = torch.empty(S * max(k, E), device=cuda_device)
    one, two = buffers(), buffers()
    _lib.check(lib.dlb_gshard_forward(x.data_ptr(), S, E, k, capacity, gates.data_ptr(), ids_km.data_ptr(),
                                      scratch.data_ptr(), scratch.numel(), *[t.data_ptr() for t in one], stream), "forward")
    _lib.check(lib.dlb_gshard_gate(x.data_ptr(), S, E, k, gates2.data_ptr(), ids.data_ptr(), scratch.data_ptr(), stream), "gate")
    choices = ids.view(S, k).t().contiguous()
    colsum = torch.empty(blocks * E, device=cuda_device)
    _lib.check(lib.dlb_gshard_assign(gates2.data_ptr(), choices.data_ptr(), None, None, S, E, k, capacity,
                                     colsum.data_ptr(), blocks, *[t.data_ptr() for t in two], stream), "assign")
    assert torch.equal(gates, gates2) and torch.equal(ids_km, choices.view(-1))
    for i, (a, b) in enumerate(zip(one, two)):
        if i in (1, 3):      # me, l_aux
            torch.testing.assert_close(a, b, rtol=1e-5, atol=0)
        else:
            assert torch.equal(a, b), i


@pytest.mark.parametrize("E,k", [(8, 8), (5, 3), (40, 20)])
def test_gate_of_a_negative_nan(cuda_device, E, k):
    """The fillers of a ragged gate rank above it: no id outside the experts, forward and backward (nothing reads or
    writes outside the gates), and the other tokens' gradients stay finite."""
    logits = torch.randn(37, E, generator=torch.Generator().manual_seed(E))
    logits[3] = torch.tensor(-1, dtype=torch.int32).view(torch.float32)
    logits[36, ::2] = torch.tensor(-4194304, dtype=torch.int32).view(torch.float32)
    x = logits.to(cuda_device).requires_grad_()
    _, ec, w, sel = topk_gating(x, k, 1.0, 2, True)
    ids = w.grad_fn.saved_tensors[2]
    assert ((ids >= 0) & (ids < E)).all()
    w.nan_to_num().sum().backward()
    assert ((ec >= 0) & (ec < sel.numel())).all() and ((sel >= 0) & (sel < 37)).all()
    assert torch.isfinite(x.grad[[i for i in range(36) if i != 3]]).all()


def test_threads_with_different_expert_counts(cuda_device):
    """The kernel's shared-memory limit is one for the process: a thread with few experts must not lower it for a launch
    with many (1024 experts take 148 KB, 8 take 1.4).  The entry point itself in a tight loop, which holds no lock."""
    lib = _lib.load()
    codes = []

    def work(E):
        cap = _align_capacity(64, E, 8)
        buf = torch.zeros(2 * cap + E + 2 + 64, dtype=torch.int32, device=cuda_device)
        at = [buf.data_ptr() + 4 * o for o in (0, 64, 64 + cap, 64 + 2 * cap, 65 + 2 * cap)]
        call = [c_void_p(at[0]), c_int(0), c_int64(64), c_int(E), c_int(8), c_void_p(at[1]), c_int64(cap), c_void_p(at[2]),
                c_int64(cap), c_void_p(at[3]), c_void_p(at[4]), c_void_p(stream.cuda_stream)]
        start.wait()
        codes.extend({fn(*call) for _ in range(20000)})
        stream.synchronize()

    stream, start = torch.cuda.Stream(), threading.Barrier(4)
    fn = lib.dlb_moe_align_block_size
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(E,)) for E in (8, 1024, 16, 1000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert set(codes) == {0}
