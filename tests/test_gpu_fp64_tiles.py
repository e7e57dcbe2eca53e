"""FP64 SIMT accumulation at the edges of its tile shapes: sector sizes on both
sides of 8, 16 and 32 rows and their remainders, every sector pair, ragged
walker counts, one and three weight planes, against numpy on the same V."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sectors, W", [
    ([0, 2, 5, 6, 7], 1),               # 1, 2, 7, 11, 15 states; one walker
    ([4, 6, 8, 9], 333),                # 5, 11, 22, 30
    ([10, 1, 11], 1000),                # 42 = 32 + 16 rows, 1, 56 = 32 + 32
    ([13, 5, 7], 257),                  # 101 = 3 x 32 + 8, 7, 15
])
def test_fp64_tiles(lemc, cuda_ctx, sectors, W):
    torch, lib = cuda_ctx, lemc.load()
    probes = [abs(sectors[0] - sectors[1])]
    g = np.random.default_rng(7)
    Wpad = (W + 63) // 64 * 64
    smp = lemc.Sampler(lemc.SamplerConfig(20, 3, W), sectors, probes=probes)
    D = smp.total_dim
    V = np.zeros((2 * D, Wpad), np.float32)
    V[:, :W] = g.standard_normal((2 * D, W))
    w = np.zeros((lemc._lib.N_WEIGHTS, Wpad), np.float32)
    w[:6, :W] = g.uniform(0.5, 2.0, (6, W))
    dV, dw = torch.from_numpy(V).cuda(), torch.from_numpy(w).cuda()
    assert lib.lemc_gram_device(smp._h, C.c_void_p(dV.data_ptr()), C.c_void_p(dw.data_ptr()), W, Wpad,
                                lemc._lib.GRAM_FP64, None) == 0
    torch.cuda.synchronize()
    smp.synchronize()
    w32 = w[:, :W]
    plane = lambda p: (w32[0] * w32[p]).astype(np.float64)  # noqa: E731  (the product is FP32)
    V = V.astype(np.float64)[:, :W]
    vals, f = [], 0
    for d in smp.dims:
        vals.append(V[2 * f:2 * f + d] + 1j * V[2 * f + d:2 * f + 2 * d])
        f += d
    # an FP64 sum of W products against another order of the same sum
    tol = lambda a, b, x: 4e-16 * max(W, 16) * (np.abs(a) * x) @ np.abs(b).T  # noqa: E731

    def same(got, a, b, x):
        assert np.all(np.abs(got - (a.conj() * x) @ b.T) <= tol(a, b, x))

    for s, v in enumerate(vals):
        for got, x in zip(smp.gram(s)[:3], (w32[0].astype(np.float64), plane(1), plane(2))):
            same(got, v, v, x)
    for i, a in enumerate(vals):
        for j, b in enumerate(vals):
            cu, cc, cs = smp.cross(i, j)
            same(cu, a, b, plane(lemc._lib.W_USER))
            if abs(sectors[i] - sectors[j]) == probes[0]:
                same(cc, a, b, plane(4))
                same(cs, a, b, plane(5))
            else:
                assert not cc.any() and not cs.any()
    smp.close()
