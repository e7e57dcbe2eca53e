"""Training samples, formed for several steps ahead or for a part of a step at a time: the
first step's objective against the public per-sample evaluation with the trainer's own
Philox draws, and a run of several steps against the same run step by step."""
import numpy as np
import pytest

from test_gpu_learned_slots import _philox, _u01

pytestmark = pytest.mark.gpu


def _setup(lemc, N, n_cfg):
    import torch
    smp = lemc.Sampler(lemc.SamplerConfig(N, 3, n_cfg, seed=3, step_sigma=1.2), [1])
    smp.init_walkers()
    smp.run(30, measure=False)
    xy = smp.positions().astype(np.float32)
    smp.close()
    prop = lemc.LearnedProposal(N, 3, init_sigma=1.5, seed=4)
    p = prop.params.copy()
    p[-260:-4] += 0.02 * np.random.default_rng(0).standard_normal(256).astype(np.float32)
    p = torch.from_numpy(p).bfloat16().float().numpy()  # evaluation reads BF16 weights
    prop.params = p
    return xy, torch.from_numpy(xy).cuda(), prop, p


# 32768 samples are formed at a time: less than a round of a block's warps, whole steps, one
# step in parts; N below the neighbour count and over the lanes' slots
@pytest.mark.parametrize("N, batch", [(5, 1), (17, 40), (64, 1000), (130, 32768), (256, 32769), (20, 70000)])
def test_objective_matches_evaluation(lemc, cuda_ctx, N, batch):
    n_cfg, seed = 37, 12
    xy, cfg, prop, p = _setup(lemc, N, n_cfg)
    # perturbations and a step too small to move the parameters
    trace = prop.train(cfg.data_ptr(), n_cfg, steps=1, batch=batch, pairs=1, lr=1e-20, es_sigma=1e-20,
                       seed=seed)
    prop.params = p
    r = _philox([np.arange(batch), np.zeros(batch), np.zeros(batch), np.full(batch, 5)],
                np.uint64(seed), np.uint64(0))
    rad, ang = np.sqrt(-2 * np.log(_u01(r[2]))), 2 * np.pi * _u01(r[3])
    eps = np.stack([rad * np.cos(ang), rad * np.sin(ang)], 1).astype(np.float32)
    out = prop.evaluate(xy[(r[0] % np.uint64(n_cfg)).astype(int)], (r[1] % np.uint64(N)).astype(np.int32), eps)
    val = np.exp(np.minimum(out[:, 6].astype(float), 0.0)) * out[:, 7]
    # FP32 against FP64 Box-Muller: 1e-5 of a step, times a log-ratio slope of order N
    assert abs(trace[0] - val.mean()) < 2e-3 * np.abs(val).mean()
    prop.close()


# 35 steps of 1000 and 3 of 16384: the last samples are formed in a second launch
@pytest.mark.parametrize("N, batch, steps", [(20, 7, 4), (65, 1000, 35), (129, 16384, 3), (40, 40000, 2)])
def test_steps_ahead(lemc, cuda_ctx, N, batch, steps):
    n_cfg = 64
    _, cfg, prop, p = _setup(lemc, N, n_cfg)
    prop.train(cfg.data_ptr(), n_cfg, steps=steps, batch=batch, pairs=2, lr=3e-3)
    once = prop.params
    prop.params = p
    for _ in range(steps):
        prop.train(cfg.data_ptr(), n_cfg, steps=1, batch=batch, pairs=2, lr=3e-3)
    # the same sums but for the order of the blocks' FP64 additions; a parameter moves 3e-3 a step
    assert np.max(np.abs(once - p)) > 1e-3
    assert np.max(np.abs(once - prop.params)) < 1e-5
    prop.close()
