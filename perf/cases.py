"""The measured cases of this framework: hierarchy propagations (RK4, RKF45),
steady states and batches as a user's program runs them through phi_b200.heom
(and one operator apply on the caller's device buffers through the C ABI).

A case is a dict of plain values:

  method     "rk4", "rkf45", "steady", "batch", "apply" or "job"
  bath       "independent" (a Drude bath per site), "diagonal" (correlated
             couplings) or "full" (matrix couplings)
  ham        "spin", "exciton", "ring" or "chain": the Hamiltonian's family
             (the distributions of phi_b200.configs)
  n, baths, k1, depth    states, baths, K + 1 terms per bath, depth L
  precision  "fp64" or "mixed"
  steps      RK4 steps;  t_end  the RKF45 span in ps
  state      True: the caller also reads the whole hierarchy back

A mixed run evaluates its stages in single precision, so what it returns is
kept in complex64; the hierarchies of the large runs stay on the device, as
they do in PHI, whose program prints rho_0.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from phi_b200 import capi, configs
from phi_b200.heom import HBAR, K_B, Batch, Hierarchy, PhiParameters

TEMPERATURE = 300.0
RKF45_TOL, RKF45_MIN_DT = 1e-6, 1e-6
STEADY_TOL = 1e-10
BATCH_DT = 0.0005
NU_1 = 2 * math.pi * K_B * TEMPERATURE / HBAR  # first Matsubara rate, 1/ps


def listed():
    return [
        # A qubit with one bath, the smallest model there is (11 nodes of
        # 2x2): 2 ps with a row every 10 fs, all of it latency.
        dict(name="spin_boson_rk4", method="rk4", bath="diagonal", ham="spin", n=2, baths=1, k1=1, depth=10,
             precision="fp64", steps=2000, state=True),
        # A trimer at a textbook depth (84 nodes): the size that parameter
        # scans and the golden tests run, thousands of tiny stages.
        dict(name="trimer_rk4", method="rk4", bath="independent", ham="exciton", n=3, baths=3, k1=2, depth=3,
             precision="fp64", steps=256, state=True),
        # The 7-site exciton at the benchmark's size (38,760 nodes), adaptive
        # steps in mixed precision: the framework's headline run.
        dict(name="frenkel7_rkf45_mixed", method="rkf45", bath="independent", ham="exciton", n=7, baths=7, k1=2,
             depth=6, precision="mixed", t_end=0.1, state=False),
        # The same exciton one tier lower in the default precision, fixed
        # steps with a row per 10 fs.
        dict(name="frenkel7_rk4", method="rk4", bath="independent", ham="exciton", n=7, baths=7, k1=2, depth=5,
             precision="fp64", steps=64, state=False),
        # A 24-site ring (20,475 nodes of 24x24), the largest state: mixed
        # precision, adaptive steps.
        dict(name="ring24_rkf45_mixed", method="rkf45", bath="independent", ham="ring", n=24, baths=24, k1=1,
             depth=4, precision="mixed", t_end=0.05, state=False),
        # A 16-site ring in the default precision: the middle of the range of
        # site counts, fixed steps.
        dict(name="ring16_rk4", method="rk4", bath="independent", ham="ring", n=16, baths=16, k1=1, depth=4,
             precision="fp64", steps=32, state=False),
        # A 9-site ring (no power of two, no size with a kernel of its own):
        # what a user with another molecule gets.
        dict(name="ring9_rk4", method="rk4", bath="independent", ham="ring", n=9, baths=9, k1=2, depth=4,
             precision="fp64", steps=32, state=False),
        # Correlated fluctuations: every bath shifts every site (diagonal
        # couplings), 5 sites with 3 shared baths.
        dict(name="correlated5_rk4", method="rk4", bath="diagonal", ham="exciton", n=5, baths=3, k1=2, depth=6,
             precision="fp64", steps=64, state=True),
        # General couplings (off-diagonal bath operators), as for a register
        # of qubits or a truncated basis, adaptive steps.
        dict(name="full6_rkf45", method="rkf45", bath="full", ham="exciton", n=6, baths=3, k1=2, depth=5,
             precision="fp64", t_end=0.05, state=True),
        # The steady state of the 4-site chain (125,970 nodes of 4x4).
        dict(name="chain4_steady", method="steady", bath="independent", ham="chain", n=4, baths=4, k1=3, depth=8,
             precision="fp64", state=False),
        # A parameter scan: 48 hierarchies of uneven size stepped together.
        dict(name="batch48_rk4_mixed", method="batch", bath="independent", count=48, mix=3, budget_mib=16,
             precision="mixed", steps=16),
        # One Liouvillian apply of the 7-site exciton on the caller's own
        # device buffers: the building block of a user's own integrator.
        dict(name="frenkel7_apply", method="apply", bath="independent", ham="exciton", n=7, baths=7, k1=2, depth=6,
             precision="fp64"),
    ]


# ---------------------------------------------------------------- the ranges

def _nodes(case) -> int:
    return configs.hierarchy_nodes(case["baths"] * case["k1"], case["depth"])


def _deepest(rng, case, lo, hi, elements) -> None:
    """A depth in lo..hi, lowered until the hierarchy has at most `elements`
    matrix elements; hierarchies of a few MB are read back whole."""
    case["depth"] = rng.randint(lo, hi)
    while case["depth"] > 1 and _nodes(case) * case["n"] ** 2 > elements:
        case["depth"] -= 1
    case["state"] = _nodes(case) * case["n"] ** 2 <= 2 ** 17


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spin", "small", "exciton", "exciton", "ring", "ring", "odd", "diagonal", "full", "steady",
                       "batch", "apply"])
    if kind == "spin":  # one or two baths on a qubit, shallow to deep
        case = dict(method="rk4", bath="diagonal", ham="spin", n=2, baths=1, k1=rng.randint(1, 2), precision="fp64",
                    steps=_log_int(rng, 128, 2000), state=True)
        case["depth"] = rng.randint(4, 14) if case["k1"] == 1 else rng.randint(3, 8)
    elif kind == "small":  # dimers to tetramers, tens to a few thousand nodes
        n = rng.randint(2, 4)
        case = dict(method="rk4", bath="independent", ham="exciton", n=n, baths=n, k1=rng.randint(1, 3),
                    precision=rng.choice(["fp64", "fp64", "mixed"]), steps=_log_int(rng, 32, 256))
        _deepest(rng, case, 2, 7, 2 ** 14)
    elif kind == "exciton":  # 5 to 8 sites, either precision, either integrator
        n = rng.randint(5, 8)
        case = dict(bath="independent", ham="exciton", n=n, baths=n, k1=rng.randint(1, 2),
                    precision=rng.choice(["fp64", "mixed"]))
        _deepest(rng, case, 3, 7, 2 ** 21)
        if rng.random() < 0.5:
            case.update(method="rkf45", t_end=round(rng.uniform(0.02, 0.08), 3))
        else:
            case.update(method="rk4", steps=_log_int(rng, 16, 64))
    elif kind == "ring":  # 10 to 24 sites, either precision, either integrator
        n = rng.choice([10, 12, 16, 24])
        case = dict(bath="independent", ham="ring", n=n, baths=n, k1=rng.choice([1, 1, 2]),
                    precision=rng.choice(["fp64", "mixed"]))
        _deepest(rng, case, 2, 5, 2 ** 23)
        if rng.random() < 0.5:
            case.update(method="rkf45", t_end=round(rng.uniform(0.02, 0.05), 3))
        else:
            case.update(method="rk4", steps=_log_int(rng, 8, 32))
    elif kind == "odd":  # site counts and term counts off the usual ones
        n = rng.choice([3, 4, 9, 9, 11, 13, 14, 15, 18, 20])
        case = dict(method="rk4", bath="independent", ham="ring" if n > 4 else "exciton", n=n, baths=n,
                    k1=4 if n <= 4 else rng.randint(1, 2), precision="fp64", steps=_log_int(rng, 8, 32))
        _deepest(rng, case, 2, 5, 2 ** 19)
    elif kind in ("diagonal", "full"):
        case = dict(bath=kind, ham="exciton", n=rng.randint(2, 10), baths=rng.randint(1, 4), k1=rng.randint(1, 3),
                    precision="fp64")
        _deepest(rng, case, 2, 8, 2 ** 17 if kind == "diagonal" else 2 ** 16)
        if kind == "full" and rng.random() < 0.6:
            case.update(method="rkf45", t_end=round(rng.uniform(0.01, 0.05), 3))
        else:
            case.update(method="rk4", steps=_log_int(rng, 16, 64))
    elif kind == "steady":
        n = rng.randint(2, 5)
        case = dict(method="steady", bath="independent", ham="chain", n=n, baths=n, k1=rng.randint(1, 3),
                    precision="fp64")
        _deepest(rng, case, 4, 8, 2 ** 20)
    elif kind == "batch":
        case = dict(method="batch", bath="independent", count=_log_int(rng, 8, 64), mix=rng.randint(0, 10 ** 6),
                    budget_mib=rng.choice([1, 4, 16]), precision=rng.choice(["fp64", "mixed"]), steps=16)
    else:
        n = rng.choice([4, 5, 6, 7, 8, 9, 12, 16, 24])
        case = dict(method="apply", bath="independent", ham="exciton" if n < 9 else "ring", n=n, baths=n,
                    k1=rng.randint(1, 2) if n > 5 else rng.randint(1, 3),
                    precision="fp64" if n == 9 else rng.choice(["fp64", "mixed"]))
        _deepest(rng, case, 3, 8, 2 ** 21)
    return case


# ------------------------------------------------------------- the problems

def _dt(case) -> float:
    """RK4 step in ps: 1 fs, halved until the deepest tier's damping is well
    inside RK4's stability region."""
    rate = case["depth"] * max(20.0, NU_1 * (case["k1"] - 1))
    dt = 0.001
    while dt * rate > 1.2:
        dt /= 2
    return dt


def _hamiltonian(ham: str, n: int, rng) -> np.ndarray:
    H = np.zeros((n, n))
    if ham == "spin":  # (eps / 2) sigma_z + Delta sigma_x
        H[0, 0] = rng.uniform(25.0, 75.0)
        H[1, 1] = -H[0, 0]
        H[0, 1] = H[1, 0] = rng.uniform(25.0, 75.0)
    elif ham == "exciton":  # all sites coupled
        H[np.diag_indices(n)] = rng.uniform(0.0, 600.0, size=n)
        iu = np.triu_indices(n, 1)
        H[iu] = rng.normal(0.0, 50.0, size=len(iu[0]))
        H = np.triu(H) + np.triu(H, 1).T
    elif ham == "ring":  # nearest and next-nearest neighbours, periodic
        H[np.diag_indices(n)] = rng.normal(0.0, 100.0, size=n)
        for i in range(n):
            for d, J in ((1, 300.0), (2, 30.0)):
                H[i, (i + d) % n] = H[(i + d) % n, i] = J
    else:  # chain
        H[np.diag_indices(n)] = rng.uniform(0.0, 300.0, size=n)
        for i, J in enumerate(rng.normal(0.0, 60.0, size=n - 1)):
            H[i, i + 1] = H[i + 1, i] = J
    return H


def _problem(case, seed: int) -> PhiParameters:
    rng = np.random.default_rng([20, int(seed)])
    n, nb = case["n"], case["baths"]
    p = PhiParameters(
        num_states=n, time_indepenent_hamiltonian=_hamiltonian(case["ham"], n, rng).astype(np.complex128),
        num_bath_couplings=nb, num_matsubara_terms=case["k1"], hierarchy_truncation_level=case["depth"] + 1,
        gamma=rng.uniform(10.0, 20.0, size=nb), lambda_=rng.uniform(20.0, 50.0, size=nb), temperature=TEMPERATURE)
    rho = np.zeros((n, n), np.complex128)
    site = int(rng.integers(n))
    rho[site, site] = 1.0
    p.initial_density_matrix = rho
    if case["bath"] == "diagonal":
        p.is_diagonal_bath_coupling = True
        p.bath_coupling_op = (np.array([[1.0, -1.0]]) if case["ham"] == "spin" else rng.normal(size=(nb, n)))
    elif case["bath"] == "full":
        V = rng.normal(size=(nb, n, n)) / 2
        p.is_full_bath_coupling = True
        p.bath_coupling_op = (V + V.transpose(0, 2, 1)) / 2
    p.fix_incompatible_combinations(case["method"])
    return p


def _batch_problems(case, seed: int) -> list:
    """The sizes of one configs.batched draw (by the case), the energies,
    couplings and baths of another (by the seed)."""
    out = configs.batched(seed=case["mix"], count=case["count"], budget_bytes=case["budget_mib"] * 2 ** 20)
    rng = np.random.default_rng([21, int(seed)])
    for p in out:
        n = p.num_states
        H = np.diag(rng.uniform(0.0, 400.0, size=n))
        for s, J in enumerate(rng.normal(0.0, 80.0, size=n - 1)):
            H[s, s + 1] = H[s + 1, s] = J
        p.time_indepenent_hamiltonian = H.astype(np.complex128)
        p.lambda_ = rng.uniform(10.0, 100.0, size=n)
        p.gamma = rng.uniform(5.0, 20.0, size=n)
        # Away from the resonance of the first Matsubara rate with a bath, and
        # with its tiers' damping inside RK4's stability region.
        p.temperature = TEMPERATURE
    return out


def _apply_input(case, seed: int) -> np.ndarray:
    """(M, N, N) Hermitian ADOs, smaller towards the deep tiers."""
    rng = np.random.default_rng([22, int(seed)])
    n, M = case["n"], _nodes(case)
    A = rng.normal(size=(M, n, n)) + 1j * rng.normal(size=(M, n, n))
    A = (A + np.conj(np.transpose(A, (0, 2, 1)))) / 2
    return A / (1.0 + np.arange(M))[:, None, None] ** 0.25


# ---------------------------------------------------------------- one pass

def _precision(case) -> int:
    return capi.PHI_PREC_MIXED if case["precision"] == "mixed" else capi.PHI_PREC_FP64


def prepare(case, seed):
    st = {"case": case}
    if case["method"] == "batch":
        st["batch"] = Batch(_batch_problems(case, seed), precision=_precision(case))
        return st
    st["h"] = h = Hierarchy(_problem(case, seed), precision=_precision(case))
    if case["method"] == "apply":
        # Node-major storage, each ADO column-major; the complex64 buffers of
        # mixed precision hold an even number of elements per node.
        n = case["n"]
        x = np.transpose(_apply_input(case, seed), (0, 2, 1)).reshape(h.num_nodes, n * n)
        if case["precision"] == "mixed":
            pad = np.zeros((h.num_nodes, n * n + n % 2), np.complex64)
            pad[:, :n * n] = x
            x = pad
        st["x"] = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        st["y"] = torch.zeros_like(st["x"])
    return st


def _result(case, **out):
    """What a program keeps: single precision from a mixed run."""
    if case["precision"] == "mixed":
        out = {k: v.astype(np.complex64) if isinstance(v, np.ndarray) else v for k, v in out.items()}
    return out


def run(state):
    case = state["case"]
    if case["method"] == "batch":
        b = state["batch"]
        for h in b.instances:
            h.reset(0.0)
        torch.cuda.synchronize()  # the instances' own streams, before the batch's
        b.rk4(BATCH_DT, case["steps"])
        return _result(case, rho0=np.concatenate([h.rho0().reshape(-1) for h in b.instances]))
    h = state["h"]
    if case["method"] == "apply":
        h._check(h.lib.phi_gpu_apply_device(h.ctx, state["x"].data_ptr(), state["y"].data_ptr(),
                                            torch.cuda.current_stream().cuda_stream))
        return state["y"]
    if case["method"] == "steady":
        h.steady_state(tol=STEADY_TOL, ell=2)
        out = _result(case, rho0=h.rho0())
    elif case["method"] == "rkf45":
        h.reset(0.0)
        st = h.rkf45(0.001, case["t_end"], RKF45_TOL, RKF45_MIN_DT)
        out = _result(case, rho0=h.rho0(), time=st["final_time"])
    else:
        h.reset(0.0)
        dt, steps = _dt(case), case["steps"]
        every = 10 * dt
        _, times, rows = h.rk4(dt, (steps - 0.5) * dt, output_min_step=every, capacity=steps // 10 + 2)
        out = _result(case, rows=rows, rho0=h.rho0(), times=times)
    if case["state"]:
        out.update(_result(case, state=h.get_state().view(np.complex128)))
    return out


# ------------------------------------------------------------ what it takes

def _apply_flops(n, baths, k1, nodes, bath) -> float:
    """Real operations of one Liouvillian apply: the commutator's product with
    a real H, the decay, the neighbour terms."""
    T = baths * k1
    per_node = 4.0 * n ** 3 + 8.0 * n ** 2
    if bath == "independent":
        per_node += 16.0 * T * n
    elif bath == "diagonal":
        per_node += 12.0 * T * n ** 2
    else:
        per_node += baths * 8.0 * n ** 3 + 16.0 * T * n ** 2
    return nodes * per_node


def work(case):
    """Per apply: the stage input read and the next one written, in the
    storage type; RK4 and RKF45 also read and write the complex128 state once
    a step.  RKF45 steps and BiCG steps are estimates (stiffest damping times
    step about 3.5, 1.5 fs at most; 150 steps of two applies and 12 vector passes)."""
    if case["method"] == "batch":
        rate, total, flops, state = 0.0, 0.0, 0.0, 0.0
        for p in _batch_problems(case, 0):
            e = p.nodes * p.num_states ** 2
            total += 2.0 * e * (8 if case["precision"] == "mixed" else 16)
            state += 32.0 * e
            flops += _apply_flops(p.num_states, p.num_states, p.num_matsubara_terms, p.nodes, "independent")
        return {"bytes": case["steps"] * (4 * total + state), "flops": 4.0 * case["steps"] * flops}
    M, n = _nodes(case), case["n"]
    e = float(M * n * n)
    xb = 8 if case["precision"] == "mixed" else 16
    flops = _apply_flops(n, case["baths"], case["k1"], M, case["bath"])
    if case["method"] == "apply":
        return {"bytes": 2 * e * xb, "flops": flops}
    if case["method"] == "steady":
        return {"bytes": 150 * (2 * 2 + 12) * e * 16, "flops": 300 * flops}
    if case["method"] == "rk4":
        s, stages = case["steps"], 4
    else:
        rate = case["depth"] * max(20.0, NU_1 * (case["k1"] - 1))
        s, stages = max(4.0, case["t_end"] / min(0.0015, 3.5 / rate)), 6
    return {"bytes": s * (stages * 2 * e * xb + 2 * e * 16), "flops": s * stages * flops}


# ------------------------------------------------- the same in plain 64 bits

def _multi_indices(T: int, depth: int) -> np.ndarray:
    """Multi-indices in PHI's node order: tier by tier, candidate q = k C + m
    raises term (m + k) mod T of node m of the tier above (C nodes), the
    first occurrence counts."""
    tiers = [np.zeros((1, T), np.int64)]
    for _ in range(depth):
        up = tiers[-1]
        C = len(up)
        cand = np.concatenate([up] * T)
        q = np.arange(T * C)
        cand[q, (q % C + q // C) % T] += 1
        _, first = np.unique(cand, axis=0, return_index=True)
        tiers.append(cand[np.sort(first)])
    return np.concatenate(tiers)


class _Exact:
    """The hierarchy's Liouvillian on (M, N, N) complex128 tensors."""

    def __init__(self, p: PhiParameters):
        self.dev = dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        n, nb, k1 = p.num_states, p.num_bath_couplings, p.num_matsubara_terms
        T, L = nb * k1, p.hierarchy_truncation_level - 1
        mi = _multi_indices(T, L)
        self.M, self.n, self.T, self.k1 = len(mi), n, T, k1
        key = (L + 1) ** np.arange(T, dtype=object) if (L + 1.0) ** T > 2.0 ** 62 else (L + 1) ** np.arange(T)
        code = mi.astype(key.dtype) @ key
        order = np.argsort(code, kind="stable")
        sorted_code = code[order]

        def find(c, ok):
            at = np.clip(np.searchsorted(sorted_code, c), 0, self.M - 1)
            ok = ok & (sorted_code[at] == c)
            return np.where(ok, order[at], 0), ok
        kT = p.boltzmann_constant * p.temperature
        nu = 2 * math.pi * kT / p.hbar
        diagonal = p.is_diagonal_bath_coupling
        c, rate, delta = np.zeros(T, np.complex128), np.zeros(T), np.zeros(nb)
        for b in range(nb):
            g, lam = float(p.gamma[b]), float(p.lambda_[b])
            a = g * lam / p.hbar
            c[b * k1] = a / math.tan(g * p.hbar / (2 * kT)) - 1j * a
            rate[b * k1] = g
            delta[b] = 2 * lam * kT / p.hbar ** 2 / g - lam / p.hbar / math.tan(p.hbar * g / (2 * kT))
            for k in range(1, k1):
                c[b * k1 + k] = 4 * lam * g * kT / p.hbar ** 2 * nu * k / ((nu * k) ** 2 - g ** 2)
                rate[b * k1 + k] = nu * k
                delta[b] -= 4 * lam * kT / p.hbar ** 2 * g / ((nu * k) ** 2 - g ** 2)
        self.terms = []
        tier = mi.sum(axis=1)
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        for t in range(T):
            nx, nx_on = find(code + key[t], tier < L)
            pv, pv_on = find(code - key[t], mi[:, t] > 0)
            if p.is_rho_normalized and not diagonal:
                s, sp = np.sqrt((mi[:, t] + 1) * abs(c[t])), np.sqrt(mi[:, t] / abs(c[t]))
            else:
                s, sp = np.ones(self.M), mi[:, t].astype(np.float64)
            self.terms.append((up(nx), up(pv), up(s * nx_on), up(sp * pv_on), complex(c[t])))
        self.damp = up((mi @ rate).astype(np.float64))[:, None, None]
        self.H = up(np.asarray(p.time_indepenent_hamiltonian, np.complex128)) / p.hbar
        self.kind = "full" if p.is_full_bath_coupling else "diagonal" if diagonal else "independent"
        self.V, self.delta = None, delta
        mats = np.zeros((n, n))
        if self.kind == "independent":
            mats = (delta[:, None] + delta[None, :]) * (1 - np.eye(n))
        else:
            self.V = up(np.asarray(p.bath_coupling_op, np.float64)).to(torch.complex128)
            if diagonal:
                for b in range(nb):
                    v = np.asarray(p.bath_coupling_op[b], np.float64)
                    mats += delta[b] * (v[:, None] - v[None, :]) ** 2
        self.mats = up(mats)
        self.vacuum = L == 0
        self.y0 = torch.zeros((self.M, n, n), dtype=torch.complex128, device=dev)
        self.y0[0] = up(np.asarray(p.initial_density_matrix, np.complex128))

    def apply(self, X):
        A = -1j * (self.H @ X)
        out = A + A.mH
        if self.vacuum:
            return out
        out -= (self.damp + self.mats) * X
        for b in range(self.T // self.k1):
            if self.kind == "independent":  # V = |b><b|: column b, and its conjugate in row b
                Xb, col = X[:, :, b], 0
                for nx, pv, s, sp, c in self.terms[b * self.k1:(b + 1) * self.k1]:
                    col = col + 1j * s[:, None] * Xb[nx] + (1j * c.conjugate()) * sp[:, None] * Xb[pv]
                out[:, :, b] += col
                out[:, b, :] += col.conj()
                continue
            left = 0
            for nx, pv, s, sp, c in self.terms[b * self.k1:(b + 1) * self.k1]:
                left = left - 1j * s[:, None, None] * X[nx] - (1j * c) * sp[:, None, None] * X[pv]
            if self.kind == "diagonal":
                left = self.V[b][:, None] * left
            else:
                V = self.V[b]
                left = V @ left - float(self.delta[b]) * (V @ (V @ X - X @ V))
            out += left + left.mH
        return out

    def rk4(self, dt, steps, every):
        y, rows = self.y0.clone(), []
        for k in range(steps):
            k0 = self.apply(y)
            k1 = self.apply(y + (dt / 2) * k0)
            k2 = self.apply(y + (dt / 2) * k1)
            k3 = self.apply(y + dt * k2)
            y = y + (dt / 6) * (k0 + 2 * k1 + 2 * k2 + k3)
            if k % every == 0:
                rows.append(y[0].clone())
        return y, rows

    def rkf45(self, dt, t_end, tol, min_dt):
        """Fehlberg's pair with PHI's step control."""
        B = [[2 / 9], [1 / 12, 1 / 4], [69 / 128, -243 / 128, 135 / 64], [-17 / 12, 27 / 4, -27 / 5, 16 / 15],
             [65 / 432, -5 / 16, 13 / 16, 4 / 27, 5 / 144]]
        c4, c5 = [1 / 9, 0, 9 / 20, 16 / 45, 1 / 12], [47 / 450, 0, 12 / 25, 32 / 225, 1 / 30, 6 / 25]
        y, t, up = self.y0.clone(), 0.0, 1.1
        while t < t_end:
            k = [self.apply(y)]
            for row in B:
                k.append(self.apply(y + sum((dt * b) * v for b, v in zip(row, k))))
            y4 = y + sum((dt * b) * v for b, v in zip(c4, k) if b)
            y5 = y + sum((dt * b) * v for b, v in zip(c5, k) if b)
            err = float((y4 - y5).abs().max())
            if not math.isfinite(err):
                return None
            if err < tol or dt * 0.5 < min_dt:
                y, t, grow = y5, t + dt, err < tol / 10
                if t + dt > t_end:
                    grow, up = True, (t_end - t) / dt
                dt *= up if grow else 1.0
            else:
                dt *= 0.5
        return y, t

    def steady(self):
        """L x = 0 with tr rho_0 = 1: x[0, 0, 0] = 1 eliminated, solved
        by BiCGSTAB(2) on the real space of Hermitian hierarchies."""
        def dot(a, b):
            return float((torch.view_as_real(a) * torch.view_as_real(b)).sum())

        def A(v):
            w = self.apply(v)
            w[0, 0, 0] = 0
            return w
        one = torch.zeros_like(self.y0)
        one[0, 0, 0] = 1
        b = -A(one)
        x = torch.zeros_like(b)
        x[0, range(1, self.n), range(1, self.n)] = 1
        r0 = b - A(x)
        hat, u0, goal = r0.clone(), torch.zeros_like(b), 1e-28 * dot(b, b)
        rho0, alpha, omega = 1.0, 0.0, 1.0
        for _ in range(600):
            r, u, rho0 = [r0], [u0], -omega * rho0
            for j in range(2):
                rho1 = dot(hat, r[j])
                beta, rho0 = alpha * rho1 / rho0, rho1
                u = [a - beta * d for a, d in zip(r, u)]
                u.append(A(u[j]))
                alpha = rho0 / dot(hat, u[j + 1])
                r = [a - alpha * d for a, d in zip(r, u[1:])]
                r.append(A(r[j]))
                x = x + alpha * u[0]
            G = np.array([[dot(r[1], r[1]), dot(r[1], r[2])], [dot(r[1], r[2]), dot(r[2], r[2])]])
            try:
                g1, g2 = np.linalg.solve(G, np.array([dot(r[0], r[1]), dot(r[0], r[2])]))
            except np.linalg.LinAlgError:
                return None
            x = x + g1 * r[0] + g2 * r[1]
            r0, u0, omega = r[0] - g1 * r[1] - g2 * r[2], u[0] - g1 * u[1] - g2 * u[2], g2
            rr = dot(r0, r0)
            if not math.isfinite(rr):
                return None
            if rr <= goal:
                x[0, 0, 0] = 1
                return x / float(x[0].diagonal().real.sum())
        return None


def _as_stored(y) -> np.ndarray:
    """Node-major, each ADO column-major."""
    return np.ascontiguousarray(y.transpose(1, 2).cpu().numpy()).reshape(-1)


def exact(case, seed):
    if case["method"] == "batch":
        rho = [_Exact(p).rk4(BATCH_DT, case["steps"], 1)[0][0].cpu().numpy().reshape(-1)
               for p in _batch_problems(case, seed)]
        return {"rho0": np.concatenate(rho)}
    ex = _Exact(_problem(case, seed))
    if case["method"] == "apply":
        x = torch.from_numpy(_apply_input(case, seed)).to(ex.dev)
        if case["precision"] == "mixed":  # the operator on the input as it is stored
            x = x.to(torch.complex64).to(torch.complex128)
        y = ex.apply(x).transpose(1, 2).reshape(ex.M, -1)
        if case["precision"] == "mixed" and case["n"] % 2:
            y = torch.cat([y, torch.zeros_like(y[:, :1])], dim=1)
        return y
    if case["method"] == "steady":
        y = ex.steady()
        if y is None:
            return None
        out = {"rho0": y[0].cpu().numpy()}
    elif case["method"] == "rkf45":
        got = ex.rkf45(0.001, case["t_end"], RKF45_TOL, RKF45_MIN_DT)
        if got is None:
            return None
        y, t = got
        out = {"rho0": y[0].cpu().numpy(), "time": t}
    else:
        y, rows = ex.rk4(_dt(case), case["steps"], 10)
        out = {"rows": np.stack([r.cpu().numpy() for r in rows]), "rho0": y[0].cpu().numpy(), "times": None}
    if case["state"]:
        out["state"] = _as_stored(y)
    return out
