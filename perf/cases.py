"""Performance cases: the work a user of the framework has it do.

Every case goes through the package's public entry points over the sizes of the
repository's own workloads: the spectrum of the small FP64 form (N=8), the
mixed-precision form (N=50, dL 0..12, 272 states), the batched form (N=100,
dL 1..20, 2713 states) and the learned-proposal form (N=200, same sectors); the
plain burn-in; a whole dynamic-structure-factor call; the matrices of the
edge-response pipeline (N=100, dL 0,2..16, 526 states); the reference
estimator's row averages; the occupations of the two-state walker; the
contraction on a program's own records; the FP64 time evolution; and the
training of the proposal.

Outputs are whole matrices, positions, series and traces.  Matrices of the FP64
accumulation and of the FP64 tail are returned as they come (double).  The
mixed-precision contraction works on FP32 basis values with split products and
single-precision sums, so a program that asks for it keeps its matrices in
single precision; those cases return complex64.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import laughlinedge_b200 as L
from laughlinedge_b200 import _lib
from laughlinedge_b200._lib import check
from laughlinedge_b200.dynamics import response_matrices

M_FILL = 3  # inverse filling nu = 1/m of every workload


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # The smallest sampling call: the N=8 form (29 states, FP64 sums), a few
        # measured sweeps and the six sectors read back; launches count here.
        dict(name="spectrum_fp64_N8", kind="spectrum", N=8, lo=1, hi=6, step=1, W=4096, mode="fp64",
             sweeps=4, learned=False),
        # The mixed-precision form: N=50, dL 0..12.
        dict(name="spectrum_mixed_N50", kind="spectrum", N=50, lo=0, hi=12, step=1, W=65536,
             mode="tf32x3", sweeps=16, learned=False),
        # The batched form: N=100, dL 1..20, the largest contraction.
        dict(name="spectrum_batched_N100", kind="spectrum", N=100, lo=1, hi=20, step=1, W=131072,
             mode="tf32x3", sweeps=8, learned=False),
        # The learned-proposal form (the bench's default workload).
        dict(name="spectrum_learned_N200", kind="spectrum", N=200, lo=1, hi=20, step=1, W=65536,
             mode="tf32x3", sweeps=4, learned=True),
        # Plain burn-in of the largest droplet; the walkers handed to a torch tensor.
        dict(name="burn_in_N200", kind="burn", N=200, W=65536, sweeps=10, sigma=0.3),
        # One whole call, context creation included, at a ragged walker count.
        dict(name="dsf_N20", kind="dsf", N=20, dL=4, W=8193, burn=40, sweeps=40),
        # The edge-response pipeline's matrix elements: S, H2, H4 of nine sectors
        # plus the USER/cos/sin cross sums of every sector pair.
        dict(name="response_N100", kind="response", N=100, hi=16, step=2, W=65536, k=2, sweeps=2),
        # The reference's own estimator: every row guided by |P_a Psi|^2.
        dict(name="rows_N8", kind="rows", N=8, lo=1, hi=6, W=16384, sweeps=10),
        # Occupations of the two-state walker, all 25 row pairs of dL = 4.
        dict(name="occupation_N50", kind="occupation", N=50, dL=4, W=65536, burn=10, sweeps=20),
        # A program with records of its own: basis build and contraction on its
        # device buffers (C-ABI), N=50 sectors.
        dict(name="contract_N50", kind="contract", N=50, lo=0, hi=12, W=65536, mode="tf32x3"),
        # The FP64 evolution of the edge-response pipeline: 526 states, nine
        # density components, steps of dt = 0.05 around the drive's peak.
        dict(name="evolve_D526", kind="evolve", D=526, rho=9, steps=500),
        # Training of the learned proposal on device configurations.
        dict(name="train_N200", kind="train", N=200, n_cfg=16384, steps=50, batch=1024, pairs=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["spectrum", "spectrum", "spectrum", "learned", "burn", "dsf", "response", "rows",
                       "occupation", "contract", "contract", "evolve", "train"])
    N = _log_int(rng, 6, 200)
    W = _log_int(rng, 256, 65536)
    if kind == "spectrum":
        lo = rng.choice([0, 1, 1, 2])
        mode = rng.choice(["fp64", "tf32x3", "tf32x3"])
        hi = rng.randint(max(lo, 2), 8 if mode == "fp64" else 20)
        if mode == "fp64":
            W = min(W, 16384)
        return dict(kind="spectrum", N=N, lo=lo, hi=hi, step=1, W=W, mode=mode,
                    sweeps=rng.randint(1, 12), learned=False)
    if kind == "learned":
        return dict(kind="spectrum", N=N, lo=1, hi=rng.randint(2, 16), step=1, W=W, mode="tf32x3",
                    sweeps=rng.randint(1, 4), learned=True)
    if kind == "burn":
        return dict(kind="burn", N=N, W=W, sweeps=rng.randint(1, 10), sigma=rng.choice([0.3, 1.243]))
    if kind == "dsf":
        return dict(kind="dsf", N=_log_int(rng, 6, 60), dL=rng.randint(1, 8), W=_log_int(rng, 512, 16384),
                    burn=rng.randint(5, 40), sweeps=rng.randint(5, 40))
    if kind == "response":
        return dict(kind="response", N=max(N, 16), hi=2 * rng.randint(1, 6), step=2, W=W, k=2,
                    sweeps=rng.randint(1, 3))
    if kind == "rows":
        return dict(kind="rows", N=_log_int(rng, 6, 30), lo=1, hi=rng.randint(2, 6), W=_log_int(rng, 512, 16384),
                    sweeps=rng.randint(1, 10))
    if kind == "occupation":
        return dict(kind="occupation", N=_log_int(rng, 6, 60), dL=rng.randint(1, 5), W=_log_int(rng, 512, 65536),
                    burn=rng.randint(1, 10), sweeps=rng.randint(1, 20))
    if kind == "contract":
        return dict(kind="contract", N=max(N, 20), lo=rng.choice([0, 1]), hi=rng.randint(2, 12), W=W,
                    mode=rng.choice(["fp64", "tf32x3", "tf32x3"]) if W <= 16384 else "tf32x3")
    if kind == "evolve":
        return dict(kind="evolve", D=_log_int(rng, 5, 500), rho=rng.randint(1, 9), steps=_log_int(rng, 20, 400))
    return dict(kind="train", N=max(N, 18), n_cfg=_log_int(rng, 64, 16384), steps=_log_int(rng, 2, 50),
                batch=_log_int(rng, 100, 2048), pairs=_log_int(rng, 2, 32))


# ---- what they need ----------------------------------------------------------

MODES = {"fp64": _lib.GRAM_FP64, "tf32x3": _lib.GRAM_TF32X3}


def _sectors(case):
    return list(range(case["lo"], case["hi"] + 1, case.get("step", 1)))


def _dims(N, sectors):
    """Basis size of each sector: partitions of dL into at most N parts (1 for dL = 0)."""
    top = max(sectors)
    p = [1] + [0] * top
    for part in range(1, min(N, top) + 1):  # parts <= N: the conjugate partitions
        for s in range(part, top + 1):
            p[s] += p[s - part]
    return [p[s] for s in sectors]


def work(case):
    kind = case["kind"]
    if kind in ("spectrum", "rows", "response"):
        N, W, ns = case["N"], case["W"], case["sweeps"]
        sec = list(range(0, case["hi"] + 1, case["step"])) if kind == "response" else _sectors(case)
        d = _dims(N, sec)
        K = max(4, max(sec))
        sd2 = sum(x * x for x in d)
        if kind == "rows":  # every row's walkers against every column
            flops = ns * W * (12.0 * N * (N - 1) + 2.0 * 30 * sum(d))
            return {"bytes": 16.0 * N * W + 8.0 * 3 * sum(d) ** 2, "flops": flops}
        contraction = 24.0 * sd2
        if kind == "response":  # three more planes over the sector pairs (C_ji = C_ij^H)
            contraction += 24.0 * (sum(d) ** 2 + sum(d)) / 2
        sweep = 12.0 * N * (N - 1) + N * (16 * K + 40)
        if case.get("learned"):
            net = 2 * (16 * 2 * 64 + 65 * 64 + 64 * 4) + 3 * N
            sweep = N * (1.4 * net + 12.0 * (N - 1)) + N * (16 * K + 40)
        out = (8 if case.get("mode", "tf32x3") == "tf32x3" else 16) * 3.0 * sd2
        return {"bytes": 16.0 * N * W + out, "flops": ns * W * (sweep + contraction)}
    if kind == "burn":
        N, W = case["N"], case["W"]
        return {"bytes": 16.0 * N * W, "flops": case["sweeps"] * W * (12.0 * N * (N - 1) + 40.0 * N)}
    if kind == "dsf":
        N, W, D = case["N"], case["W"], sum(_dims(case["N"], [0, case["dL"]]))
        return {"bytes": 8.0 * N * W, "flops": W * ((case["burn"] + case["sweeps"]) * 12.0 * N * (N - 1) +
                                                    case["sweeps"] * 48.0 * D * D)}
    if kind == "occupation":
        N, W, Lc = case["N"], case["W"], M_FILL * (case["N"] - 1) + 15
        D = _dims(N, [case["dL"]])[0]
        return {"bytes": 16.0 * D * D * Lc, "flops": W * ((case["burn"] + case["sweeps"]) * 12.0 * N * N +
                                                          case["sweeps"] * 12.0 * Lc)}
    if kind == "contract":
        d = _dims(case["N"], _sectors(case))
        K = max(4, case["hi"])
        sd2 = sum(x * x for x in d)
        return {"bytes": case["W"] * (8.0 * K + 12.0) + 24.0 * sd2,
                "flops": case["W"] * (24.0 * sd2 + 6.0 * sum(d))}
    if kind == "evolve":
        D, Lr, n = case["D"], case["rho"], case["steps"]
        return {"bytes": 16.0 * D * D * (3 + Lr), "flops": n * 8.0 * D * D * (4 * 2 + Lr)}
    N = case["N"]
    net = 2 * (16 * 2 * 64 + 65 * 64 + 64 * 4) + 3 * N
    return {"bytes": 8.0 * N * case["n_cfg"], "flops": case["steps"] * 2.0 * case["pairs"] * case["batch"] *
            (2.0 * net + 12.0 * N)}


def _seed(seed):
    return 1 + int(seed) % 1000003


def _context(case, seed, sectors, probes=None, **kw):
    """A context with burnt-in walkers, as a program holds one between its blocks of sweeps."""
    smp = L.Sampler(L.SamplerConfig(case["N"], M_FILL, case["W"], seed=_seed(seed), **kw), sectors, probes=probes)
    smp.init_walkers()
    smp.set_step(1.2)  # near 50 % acceptance: burnt in within some ten sweeps
    smp.run(80, measure=False)
    smp.set_step(kw.get("step_sigma", 0.3))
    return smp


def _proposal(N, seed):
    """Weights as training leaves them: step at the upper scale, neighbourhood-dependent mean."""
    prop = L.LearnedProposal(N, M_FILL, init_sigma=3.9, seed=_seed(seed))
    p = prop.params.copy()
    g = np.random.default_rng(seed)
    p[-260:-4] += 0.02 * g.standard_normal(256).astype(np.float32)
    prop.params = p
    return prop


def _hermitian(g, D):
    x = g.standard_normal((D, D)) + 1j * g.standard_normal((D, D))
    return 0.5 * (x + x.conj().T)


class _Profile:
    """The drive's Gaussian in time, eps = 1e-3, t0 = 50, tau = 10, entered at its flank."""

    def __call__(self, t):
        return 1e-3 * math.exp(-((t + 35.0 - 50.0) ** 2) / 200.0)


def _evolve_inputs(case, seed):
    g = np.random.default_rng(seed)
    D = case["D"]
    M = np.eye(D) + 0.02 * _hermitian(g, D) / math.sqrt(D)
    H = np.diag(0.4 + 0.1 * np.sort(g.random(D))) + 0.002 * _hermitian(g, D) / math.sqrt(D)
    U = 50.0 * _hermitian(g, D) / math.sqrt(D)
    rho = [_hermitian(g, D) / math.sqrt(D) for _ in range(case["rho"])]
    return M, H, U, rho


def _contract_inputs(case, seed):
    """Power sums and weight planes of a burnt-in droplet: p_k Gaussian with
    <|p_k|^2> = k/m in units of R, sum r^2 and sum r^4 with their spreads."""
    W, N, K = case["W"], case["N"], max(4, case["hi"])
    g = torch.Generator(device="cuda").manual_seed(_seed(seed))
    k = torch.arange(1, K + 1, device="cuda", dtype=torch.float32)
    p = torch.randn((K, W, 2), generator=g, device="cuda") * (k / (2 * M_FILL)).sqrt()[:, None, None]
    Wpad = (W + 63) // 64 * 64
    w = torch.zeros((_lib.N_WEIGHTS, Wpad), device="cuda")
    e = torch.randn((2, W), generator=g, device="cuda")
    w[0, :W] = 1.0
    w[1, :W] = M_FILL * N * N * (1 + 0.02 * e[0])
    w[2, :W] = 4 / 3 * M_FILL ** 2 * N ** 3 * (1 + 0.04 * e[0] + 0.01 * e[1])
    return p.contiguous(), w


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": _seed(seed)}
    if kind == "spectrum":
        smp = _context(case, seed, _sectors(case), gram_mode=MODES[case["mode"]])
        if case["learned"]:
            s["prop"] = _proposal(case["N"], seed)
            smp.set_proposal(s["prop"])
        smp.run(1, measure=True)  # the context fixes its range factors at the first measured sweep
        s["smp"] = smp
    elif kind == "burn":
        s["smp"] = _context(case, seed, [1], step_sigma=case["sigma"])
        s["xy"] = torch.empty((case["W"], case["N"], 2), dtype=torch.float32, device="cuda")
    elif kind == "response":
        sec = list(range(0, case["hi"] + 1, case["step"]))
        smp = _context(case, seed, sec, probes=[l for l in sec if l > 0], gram_mode=_lib.GRAM_TF32X3)
        check(smp.lib.lemc_set_multipole_potential(smp._h, case["k"], 1.0), "lemc_set_multipole_potential")
        smp.run(1, measure=True)
        s["smp"] = smp
    elif kind == "rows":
        smp = _context(case, seed, _sectors(case), guide=_lib.GUIDE_ROW)
        smp.run(1, measure=True)
        s["smp"] = smp
    elif kind == "contract":
        smp = L.Sampler(L.SamplerConfig(case["N"], M_FILL, case["W"]), _sectors(case))
        s["smp"] = smp
        s["p"], s["w"] = _contract_inputs(case, seed)
        s["V"] = torch.zeros((2 * smp.total_dim, s["w"].shape[1]), device="cuda")
    elif kind == "evolve":
        s["in"] = _evolve_inputs(case, seed)
    elif kind == "train":
        N, n = case["N"], case["n_cfg"]
        smp = L.Sampler(L.SamplerConfig(N, M_FILL, n, seed=_seed(seed), step_sigma=1.24), [1])
        smp.init_walkers()
        smp.run(60, measure=False)
        s["xy"] = torch.empty((n, N, 2), dtype=torch.float32, device="cuda")
        smp.copy_positions_device(s["xy"].data_ptr())
        smp.synchronize()
        smp.close()
        s["prop"] = L.LearnedProposal(N, M_FILL, init_sigma=1.24, seed=s["seed"])
        s["start"] = s["prop"].params
    return s


def _grams(smp, single):
    out = []
    for i in range(len(smp.sectors)):
        g = smp.gram(i)[:3]
        out.append([x.astype(np.complex64) for x in g] if single else list(g))
    return out


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "spectrum":
        smp = state["smp"]
        smp.reset()
        smp.run(case["sweeps"], measure=True)
        return _grams(smp, case["mode"] != "fp64")
    if kind == "burn":
        smp = state["smp"]
        smp.run(case["sweeps"], measure=False)
        smp.copy_positions_device(state["xy"].data_ptr())
        smp.synchronize()
        return state["xy"]
    if kind == "dsf":
        return L.dsf_compute(case["N"], M_FILL, case["dL"], case["W"], case["burn"], case["sweeps"], 1e-2,
                             1e-4, seed=state["seed"])
    if kind == "response":
        smp = state["smp"]
        smp.reset()
        smp.run(case["sweeps"], measure=True)
        M, H, U, rho = response_matrices(smp, smp.sectors, 2e-3, 2e-5)
        return [x.astype(np.complex64) for x in (M, H, U, *rho)]
    if kind == "rows":
        smp = state["smp"]
        smp.reset()
        smp.run(case["sweeps"], measure=True)
        return smp.rows(1e-2, 1e-4)
    if kind == "occupation":
        return L.occupation(case["N"], M_FILL, case["dL"], M_FILL * (case["N"] - 1) + 15, case["W"],
                            case["sweeps"], burn_in=case["burn"], seed=state["seed"])
    if kind == "contract":
        smp, p, w, V = state["smp"], state["p"], state["w"], state["V"]
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        W, ldv = case["W"], w.shape[1]
        smp.reset()
        check(smp.lib.lemc_basis_device(smp._h, C.c_void_p(p.data_ptr()), W, C.c_void_p(V.data_ptr()), ldv, st),
              "lemc_basis_device")
        check(smp.lib.lemc_gram_device(smp._h, C.c_void_p(V.data_ptr()), C.c_void_p(w.data_ptr()), W, ldv,
                                       MODES[case["mode"]], st), "lemc_gram_device")
        return _grams(smp, case["mode"] != "fp64")
    if kind == "evolve":
        M, H, U, rho = state["in"]
        _, out, norms, rank = L.evolve_device(M, H, U, rho, _Profile(), case["steps"] * 0.05, 0.05, substeps=1,
                                              eps=1e-10)
        return out, norms, rank
    prop = state["prop"]
    prop.params = state["start"]
    trace = prop.train(state["xy"].data_ptr(), case["n_cfg"], steps=case["steps"], batch=case["batch"],
                       pairs=case["pairs"], lr=3e-3, es_sigma=0.02, seed=state["seed"])
    return trace, prop.params


# ---- the same in 64 bits, where there is such a value ----------------------------

def _partitions(n, least=1):
    """Partitions of n as ascending parts, in lexicographic order (the basis order)."""
    if n == 0:
        yield []
    for part in range(least, n + 1):
        for rest in _partitions(n - part, part):
            yield [part] + rest


def _exact_contract(case, seed):
    """S, H2, H4 = sum_w w conj(v_a) v_b with v = prod p_k in FP64."""
    p32, w32 = _contract_inputs(case, seed)
    W, N = case["W"], case["N"]
    p = torch.view_as_complex(p32.double())
    w = w32[:3, :W].double()
    weights = [w[0], w[0] * w[1], w[0] * w[2]]
    out = []
    for sec in _sectors(case):
        rows = list(_partitions(sec))
        v = torch.ones((len(rows), W), dtype=torch.complex128, device="cuda")
        if sec == 0:
            v *= N  # the Laughlin row is p_0 = N
        for r, parts in enumerate(rows):
            for part in parts:
                v[r] *= p[part - 1]
        out.append([((v.conj() * x) @ v.T).cpu().numpy() for x in weights])
    return out


def _exact_evolve(case, seed):
    """The same Runge-Kutta steps in numpy's complex128."""
    M, H, U, rho = _evolve_inputs(case, seed)
    m, Q = np.linalg.eigh(M)
    keep = m > 1e-10 * m[-1]
    X = Q[:, keep] / np.sqrt(m[keep])
    Hp, Up = X.conj().T @ H @ X, X.conj().T @ U @ X
    Hp = Hp - np.trace(Hp).real / Hp.shape[0] * np.eye(Hp.shape[0])
    R = [X.conj().T @ r @ X for r in rho]
    y = X.conj().T @ M[:, 0]
    f, h, n = _Profile(), 0.05, int(math.ceil(case["steps"] * 0.05 / 0.05))
    out, norms = np.zeros((n, len(R)), complex), np.zeros(n)
    g = lambda t, x: -1j * (Hp @ x + f(t) * (Up @ x))  # noqa: E731
    for k in range(n):
        out[k] = [np.vdot(y, r @ y) for r in R]
        norms[k] = np.vdot(y, y).real
        t = k * h
        k1 = g(t, y)
        k2 = g(t + 0.5 * h, y + 0.5 * h * k1)
        k3 = g(t + 0.5 * h, y + 0.5 * h * k2)
        k4 = g(t + h, y + h * k3)
        y = y + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    return out, norms, None


def exact(case, seed):
    """Chains have no 64-bit value (their positions are FP32 by definition)."""
    if case["kind"] == "contract":
        return _exact_contract(case, seed)
    if case["kind"] == "evolve":
        return _exact_evolve(case, seed)
    return None
