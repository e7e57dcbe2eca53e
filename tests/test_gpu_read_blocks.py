"""Read-back of Gram and cross blocks, small (one piece) and large (plane by plane), with
planes left out, after reset and repeated, against the same sums in numpy."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 3])
def test_read_blocks(lemc, cuda_ctx, mode):
    torch, lib = cuda_ctx, lemc.load()
    # 1, 77 and 490 states: 8, 35 k and 1.4 M doubles
    sectors, W = [0, 12, 19], 64
    g = np.random.default_rng(1)
    smp = lemc.Sampler(lemc.SamplerConfig(20, 3, W, gram_mode=mode), sectors, probes=[7])
    V = g.standard_normal((2 * smp.total_dim, W)).astype(np.float32)
    w = np.ones((lemc._lib.N_WEIGHTS, W), np.float32)
    w[1], w[2], w[3] = 2.0, 3.0, 0.5
    dV, dw = torch.from_numpy(V).cuda(), torch.from_numpy(w).cuda()

    def add():
        assert lib.lemc_gram_device(smp._h, C.c_void_p(dV.data_ptr()), C.c_void_p(dw.data_ptr()), W, W, mode,
                                    None) == 0
        torch.cuda.synchronize()

    vals, f = [], 0
    for d in smp.dims:
        vals.append((V[2 * f:2 * f + d] + 1j * V[2 * f + d:2 * f + 2 * d]).astype(complex))
        f += d
    tol = 1e-12 if mode == 0 else 1e-6

    def same(got, a, b, x):
        assert np.max(np.abs(got - x * a.conj() @ b.T)) < tol * x * 2 * W * 4

    for times in (1, 2):  # the sums continue after a read
        add()
        for _ in range(2):
            for s, v in enumerate(vals):
                for got, x in zip(smp.gram(s)[:3], (1, 2, 3)):
                    same(got, v, v, x * times)
    d = smp.dims[2]
    only = np.zeros(2 * d * d)
    assert lib.lemc_read_gram(smp._h, 2, None, lemc._lib.dptr(only), None, None) == 0
    same(only.view(complex).reshape(d, d), vals[2], vals[2], 4)
    for i, j in ((1, 2), (2, 1), (0, 2)):
        cu, cc, _ = smp.cross(i, j)
        assert np.max(np.abs(cu - 2 * 0.5 * vals[i].conj() @ vals[j].T)) < 1e-9
        if {i, j} == {1, 2}:
            assert np.max(np.abs(cc - 2 * vals[i].conj() @ vals[j].T)) < 1e-9
    smp.reset()
    add()
    same(smp.gram(1)[0], vals[1], vals[1], 1)
    smp.close()
