"""tcgen05 contraction (FP16 hi/lo operands with power-of-two row scales) at the
edges of its ranges: rows of very large, very small and zero magnitude, uneven
weights, walker counts around a K-chunk, one tile a job and two.  Against numpy
in FP64 on the same V; the error measure and its 1e-6 bound are those of the
split (22 significant bits, FP32 sums)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sectors, W, spread", [
    ([0, 1, 2], 1, 0),                     # one walker
    ([1, 3, 5], 63, 12),
    ([1, 3, 5], 65, 12),                   # one walker past a K-chunk
    ([4, 6, 8], 1000, 30),                 # rows from 1e-30 to 1e30
    ([2, 7, 12], 4097, 6),                 # a sector of several A slices
    (list(range(0, 17, 2)), 20000, 8),     # two tiles a job
])
def test_scaled_rows(lemc, cuda_ctx, sectors, W, spread):
    torch, lib = cuda_ctx, lemc.load()
    g = np.random.default_rng(3)
    Wpad = (W + 63) // 64 * 64
    smp = lemc.Sampler(lemc.SamplerConfig(30, 3, W, gram_mode=lemc._lib.GRAM_TF32X3), sectors)
    D = smp.total_dim
    V = np.zeros((2 * D, Wpad), np.float32)
    V[:, :W] = g.standard_normal((2 * D, W)) * np.exp(g.standard_normal((1, W)))
    row = 10.0 ** g.uniform(-spread, spread, D)
    f = 0
    for d in smp.dims:  # a state's Re and Im rows at one magnitude
        V[2 * f:2 * f + d] *= row[f:f + d, None]
        V[2 * f + d:2 * f + 2 * d] *= row[f:f + d, None]
        f += d
    zero = 2 * (D - smp.dims[-1])  # the last sector's first state vanishes
    V[[zero, zero + smp.dims[-1]]] = 0.0
    w = np.zeros((lemc._lib.N_WEIGHTS, Wpad), np.float32)
    w[0, :W] = g.uniform(0.0, 2.0, W)
    w[1, :W] = 1e4 * g.uniform(0.5, 1.5, W)
    w[2, :W] = 1e7 * np.exp(g.standard_normal(W))
    dV, dw = torch.from_numpy(V).cuda(), torch.from_numpy(w).cuda()
    assert lib.lemc_gram_device(smp._h, C.c_void_p(dV.data_ptr()), C.c_void_p(dw.data_ptr()), W, Wpad,
                                lemc._lib.GRAM_TF32X3, None) == 0
    torch.cuda.synchronize()
    smp.synchronize()
    weights = [w[0, :W].astype(float), (w[0] * w[1])[:W].astype(float), (w[0] * w[2])[:W].astype(float)]
    f = 0
    for s, d in enumerate(smp.dims):
        v = V[2 * f:2 * f + d, :W] + 1j * V[2 * f + d:2 * f + 2 * d, :W].astype(float)
        f += d
        v = v.astype(complex)
        for got, x in zip(smp.gram(s)[:3], weights):
            ref = (v.conj() * x) @ v.T
            n = np.sqrt(np.real(np.diag(ref)))
            n[n == 0] = 1.0
            assert np.max(np.abs(got - ref) / np.outer(n, n)) < 1e-6
    smp.close()


def test_non_finite_rows_are_reported(lemc, cuda_ctx):
    torch, lib = cuda_ctx, lemc.load()
    W = 256
    for bad in (np.inf, np.nan):
        smp = lemc.Sampler(lemc.SamplerConfig(8, 3, W, gram_mode=lemc._lib.GRAM_TF32X3), [1, 2])
        V = torch.ones((2 * smp.total_dim, W), device="cuda")
        V[2, 17] = bad  # sector 2, first state
        w = torch.ones((lemc._lib.N_WEIGHTS, W), device="cuda")
        torch.cuda.synchronize()
        assert lib.lemc_gram_device(smp._h, C.c_void_p(V.data_ptr()), C.c_void_p(w.data_ptr()), W, W,
                                    lemc._lib.GRAM_TF32X3, None) == 0
        torch.cuda.synchronize()
        assert np.allclose(smp.gram(0)[0], 2 * W)
        with pytest.raises(lemc.LemcError):
            smp.gram(1)
        smp.close()
