"""Occupation walker over the lane counts it is compiled for, with rows of one to
several distinct parts on either side, against the same walk in numpy (same Philox
draws): averages of every row pair none of whose walkers met a near-tie decision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M32 = np.uint64(0xFFFFFFFF)


def _philox(c, k0):
    c = [np.broadcast_to(np.asarray(x, np.uint64), np.broadcast(*c).shape).copy() for x in c]
    k0, k1 = np.uint64(k0), np.uint64(0)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & M32, (p0 >> np.uint64(32)) ^ c[3] ^ k1, p0 & M32]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & M32, (k1 + np.uint64(0xBB67AE85)) & M32
    return [((x >> np.uint64(9)).astype(float) + 0.5) * 2.0 ** -23 for x in c]


def _walk(N, m, rows, Lc, W, burn, meas, sigma, seed):
    D, w = len(rows), np.arange(W)
    pair = w * D * D // W
    R = np.sqrt(2.0 * m * N)
    u = _philox([np.arange(N + 1)[None], 0, w[:, None], 3], seed)
    z = (R * np.sqrt(u[0]) * np.exp(2j * np.pi * u[1])).astype(np.complex64).astype(complex)
    power = lambda zz, lo, hi, k: np.sum((zz[:, lo:hi] / R) ** k, 1)  # noqa: E731

    def poly(zz, side):  # ln|P| and arg P of each walker's row on one side
        out = np.zeros(W, complex)
        for p in range(D * D):
            sel = pair == p
            for k, r in rows[p // D if side == 0 else p % D][1]:
                if k:
                    out[sel] += r * np.log(power(zz[sel], side, N + side, k))
        return out

    near, est = np.zeros(W, bool), np.zeros((W, Lc), complex)
    l = np.arange(Lc)
    lnf = np.concatenate([[0.0], np.cumsum(np.log(np.arange(1, Lc)))])
    for s in range(burn + meas):
        for i in range(N + 1):
            u = _philox([i, s, w, 2], seed)
            zn = z.copy()
            zn[:, i] = (z[:, i] + sigma * np.sqrt(-2 * np.log(u[0])) * np.exp(2j * np.pi * u[1])).astype(
                np.complex64)
            oth = [j for j in range(1, N) if j != i]
            jas = np.sum(np.log(np.abs(zn[:, [i]] - z[:, oth])) - np.log(np.abs(z[:, [i]] - z[:, oth])), 1)
            gz = np.abs(z[:, i]) ** 2 - np.abs(zn[:, i]) ** 2
            d = np.zeros(W)
            if i < N:
                d += (poly(zn, 0) - poly(z, 0)).real + m * jas + 0.25 * gz
            if i > 0:
                d += (poly(zn, 1) - poly(z, 1)).real + m * jas + 0.25 * gz
            if 0 < i < N:
                for e in (0, N):
                    d += m * np.log(np.abs(zn[:, i] - z[:, e]) / np.abs(z[:, i] - z[:, e]))
            lu = np.log(u[2])
            near |= np.abs(d - lu) < 1e-3
            z = np.where((d >= lu)[:, None], zn, z)
        if s >= burn:
            q0 = 0.5 * z[:, 0] * z[:, N].conj()
            ph = (poly(z, 1) - poly(z, 0)).imag + m * np.sum(
                np.angle((z[:, 1:N] - z[:, [N]]) * (z[:, [0]] - z[:, 1:N]).conj()), 1)
            base = -0.25 * (np.abs(z[:, 0]) ** 2 + np.abs(z[:, N]) ** 2) - np.log(2 * np.pi)
            est += np.exp(base[:, None] + l * np.log(np.abs(q0))[:, None] - lnf +
                          1j * (l * np.angle(q0)[:, None] + ph[:, None]))
    occ, ok = np.zeros((D * D, Lc), complex), np.zeros(D * D, bool)
    for p in range(D * D):
        sel = pair == p
        occ[p], ok[p] = est[sel].sum(0) / (meas * sel.sum()), not near[sel].any()
    return occ.reshape(D, D, Lc), ok.reshape(D, D)


@pytest.mark.parametrize("N, dL, per", [(2, 1, 5), (4, 3, 3), (9, 6, 1), (33, 3, 3), (65, 2, 3), (130, 2, 2)])
def test_all_pairs_match_numpy(lemc, cuda_ctx, N, dL, per):
    rows, _, _ = lemc.partitions(N, [dL])
    D, Lc = len(rows), 3 * (N - 1) + 15
    W = D * D * per
    got, _ = lemc.occupation(N, 3, dL, Lc, W, 2, burn_in=2, step_sigma=0.5, seed=9)
    ref, ok = _walk(N, 3, rows, Lc, W, 2, 2, 0.5, 9)
    assert ok.sum() >= 1 and (N > 40 or ok.mean() > 0.5)
    # positions carry FP32 rounding (1e-7 of R a move), phases l times that
    scale = np.max(np.abs(ref[ok]), axis=-1)
    assert np.max(np.abs(got[ok] - ref[ok]).max(-1) / scale) < 5e-3
