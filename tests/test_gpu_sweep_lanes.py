"""Plain sweep with two of a walker's lanes per thread (many walkers) against one lane per
thread (one walker less): positions, records and counters of the common walkers bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sweep(lemc, pos, N, G, K, probes):
    import torch
    W = pos.shape[0]
    pos = pos.clone()
    rec_p = torch.zeros(K, W, 2, device="cuda")
    rec_w = torch.zeros(4 + 2 * len(probes), W, device="cuda")
    acc = torch.zeros(W, dtype=torch.int32, device="cuda")
    pr = np.asarray(probes, np.int32)
    st = lemc.load().lemc_sweep_device(
        C.c_void_p(pos.data_ptr()), W, N, 3, 0.6, 77, 5, 3, K, np.sqrt(6.0 * N), G, 1,
        pr.ctypes.data_as(C.POINTER(C.c_int32)), len(probes), C.c_void_p(rec_p.data_ptr()),
        C.c_void_p(rec_w.data_ptr()), C.c_void_p(acc.data_ptr()), None)
    assert st == 0
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in (pos, rec_p, rec_w, acc)]


# W is the smallest that takes two lanes a thread: 13 warps on each of 148 SMs; N below and
# above a row of the lanes, odd and even slot counts, the longest record of eight lanes
@pytest.mark.parametrize("N, G, W", [(5, 8, 15392), (8, 8, 15392), (65, 8, 15392), (896, 8, 15392),
                                     (31, 16, 7696), (150, 16, 7696), (33, 32, 3848), (200, 32, 3848)])
def test_two_lanes_a_thread(lemc, cuda_ctx, N, G, W):
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    pos = torch.randn(W, N, 2, device="cuda", generator=g) * np.sqrt(1.5 * N)
    two = _sweep(lemc, pos, N, G, 7, [1, 3])
    one = _sweep(lemc, pos[:-1].contiguous(), N, G, 7, [1, 3])
    n = W - 1
    assert one[3].sum() > 0
    for a, b in ((two[0][:n], one[0]), (two[1][:, :n], one[1]), (two[2][:, :n], one[2]),
                 (two[3][:n], one[3])):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
