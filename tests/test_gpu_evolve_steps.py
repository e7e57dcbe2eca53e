"""FP64 GPU evolution against the same Runge-Kutta steps in numpy: matrices held
in shared memory and not, one block and many, one save point and more than one
batch of them, with and without density components."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _herm(g, D):
    x = g.standard_normal((D, D)) + 1j * g.standard_normal((D, D))
    return 0.5 * (x + x.conj().T) / np.sqrt(D)


@pytest.mark.parametrize("D, ns, substeps, L", [
    (1, 3, 1, 1),
    (4, 1, 1, 1),        # the initial state only
    (5, 1030, 2, 2),     # two CTAs; a second batch of save points
    (33, 40, 1, 0),      # no density components
    (150, 33, 3, 3),     # 38 CTAs, a ragged last one; save points past a 32 tile
    (900, 5, 1, 2),      # 148 CTAs, rows read from global memory
])
def test_evolution_steps(lemc, cuda_ctx, D, ns, substeps, L):
    g = np.random.default_rng(11)
    M = np.eye(D) + 0.02 * _herm(g, D)
    H = np.diag(np.linspace(0.4, 0.6, D)) + 0.01 * _herm(g, D)
    U = _herm(g, D)
    rho = [_herm(g, D) for _ in range(L)]
    f = lambda t: 0.3 * np.exp(-(t - 1.0) ** 2)  # noqa: E731
    dt = 0.1
    _, got, norms, rank = lemc.evolve_device(M, H, U, rho, f, (ns - 0.5) * dt, dt, substeps=substeps)
    assert rank == D and norms.shape == (ns,) and got.shape == (ns, L)
    m, Q = np.linalg.eigh(M)
    X = Q / np.sqrt(m)
    Hp, Up = X.conj().T @ H @ X, X.conj().T @ U @ X
    Hp = Hp - np.trace(Hp).real / D * np.eye(D)
    R = [X.conj().T @ r @ X for r in rho]
    y, h = X.conj().T @ M[:, 0], dt / substeps
    k_of = lambda t, x: -1j * (Hp @ x + f(t) * (Up @ x))  # noqa: E731
    for s in range(ns):
        # rounding of s * substeps steps and of an r-term sum, in units of 2^-52
        tol = 2.3e-16 * 50 * (1 + s * substeps) * np.sqrt(D)
        assert abs(norms[s] - np.vdot(y, y).real) < tol
        for l in range(L):
            assert abs(got[s, l] - np.vdot(y, R[l] @ y)) < tol * max(1.0, np.linalg.norm(R[l], 2))
        for q in range(substeps):
            t = (s * substeps + q) * h
            k1 = k_of(t, y)
            k2 = k_of(t + 0.5 * h, y + 0.5 * h * k1)
            k3 = k_of(t + 0.5 * h, y + 0.5 * h * k2)
            k4 = k_of(t + h, y + h * k3)
            y = y + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
