"""Occupation walker with two of its lanes per thread (many walkers) against one lane per
thread (one walker less): the same chains, so the same averages of every row pair whose
walkers are the same in both runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# N at the ends of the ranges of 8, 16 and 32 lanes; W is the smallest that takes two a
# thread (15 warps on each of 148 SMs)
@pytest.mark.parametrize("N, W", [(33, 17760), (64, 17760), (65, 8880), (128, 8880), (129, 4440)])
def test_two_lanes_a_thread(lemc, cuda_ctx, N, W):
    dL, Lc = 6, 3 * (N - 1) + 15
    got, got_acc = lemc.occupation(N, 3, dL, Lc, W, 2, burn_in=1, step_sigma=0.5, seed=11)
    ref, ref_acc = lemc.occupation(N, 3, dL, Lc, W - 1, 2, burn_in=1, step_sigma=0.5, seed=11)
    D = got.shape[0]
    first = lambda p, w: -(-p * w // (D * D))  # noqa: E731  first walker of a pair
    same = [p for p in range(D * D)
            if first(p, W) == first(p, W - 1) and first(p + 1, W) == first(p + 1, W - 1)]
    assert len(same) > D  # pairs of several left rows
    got, ref = got.reshape(D * D, Lc)[same], ref.reshape(D * D, Lc)[same]
    scale = np.abs(ref).max(-1)
    # FP64 sums in another order: 1e-15 a term, more where a power sum all but cancels
    assert np.max(np.abs(got - ref).max(-1) / scale) < 1e-9
    assert abs(got_acc * W - ref_acc * (W - 1)) <= 1.0
