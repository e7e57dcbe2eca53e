"""Learned sweep over the particle counts where its compiled slots change, against a
sweep made move by move from the public per-sample evaluation of the same network
(proposal, ln A) with the sampler's own Philox draws."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _philox(c, k0, k1):
    c = [x.astype(np.uint64) for x in c]
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        lo = np.uint64(0xFFFFFFFF)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & lo, (p0 >> np.uint64(32)) ^ c[3] ^ k1, p0 & lo]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & lo, (k1 + np.uint64(0xBB67AE85)) & lo
    return c


def _u01(x):
    return ((x >> np.uint64(9)).astype(np.float64) + 0.5) * 2.0 ** -23


@pytest.mark.parametrize("N", [2, 5, 17, 32, 33, 64, 65, 100, 129, 161, 193, 225, 256])
def test_sweep_matches_evaluation(lemc, cuda_ctx, N):
    W, seed = 5, 42
    prop = lemc.LearnedProposal(N, 3, init_sigma=1.5, seed=4)
    p = prop.params.copy()
    p[-260:-4] += 0.02 * np.random.default_rng(0).standard_normal(256).astype(np.float32)
    prop.params = p
    smp = lemc.Sampler(lemc.SamplerConfig(N, 3, W, seed=seed, step_sigma=1.2), [1])
    smp.init_walkers()
    smp.run(30, measure=False)
    xy = smp.positions()
    if N >= 129:  # a cluster on one lane's particles: more than four nearest in a lane
        xy[:, ::32] = xy[:, :1] + 0.5 * np.random.default_rng(1).standard_normal(xy[:, ::32].shape)
    smp.init_walkers(xy)
    smp.set_proposal(prop)
    smp.run(1, measure=False)
    got = smp.positions()
    w = np.arange(W, dtype=np.uint64)
    near = np.zeros(W, bool)  # a decision within the rounding of the two evaluations
    cur = xy.astype(np.float32).copy()
    for i in range(N):
        r = _philox([np.full(W, i), np.full(W, 30), w, np.full(W, 4)], np.uint64(seed), np.uint64(0))
        rad = np.sqrt(-2 * np.log(_u01(r[0])))
        eps = np.stack([rad * np.cos(2 * np.pi * _u01(r[1])), rad * np.sin(2 * np.pi * _u01(r[1]))], 1)
        out = prop.evaluate(cur, np.full(W, i, np.int32), eps.astype(np.float32))
        lu = np.log(_u01(r[2]))
        near |= np.abs(out[:, 6] - lu) < 2e-3
        acc = lu < out[:, 6]
        cur[acc, i] = out[acc, 4:6]
    ok = ~near
    assert ok.sum() >= 2
    # positions differ by the rounding of the draws (FP32 against FP64 Box-Muller)
    assert np.max(np.abs(got[ok] - cur[ok])) < 1e-3
    smp.close()
    prop.close()
