"""Workloads of the framework, through its public entry points.

Each case is one call (or one small group of calls) that a program built on
``mcpi_b200`` makes over and over: H.psi, densities, the gradient's adjoint
and transition densities, ground states, a batched sweep, H.psi on host
buffers. ``prepare`` makes the space, the integrals and the states such a
program holds; ``run`` is one pass; ``exact`` computes the same results in 64
bits with plain torch and numpy, from the definitions of the operators.

Interactions ("kind"):
  lieb     contact interaction on a ring, plane-wave orbitals (mcpi_b200.lieb_integrals)
  gauss    finite-range (Gaussian) interaction on a ring, plane-wave orbitals: conserves
           momentum, every momentum transfer with a strength of its own
  general  random Hermitian Ho and random complex Hint with the bosonic 8-fold symmetry
"""
import math

import numpy as np
import torch

import mcpi_b200 as mc

DEVICE = 0
M_BATCH = (7, 9, 11)


def listed():
    return [
        # An ordinary mid-size space with a finite-range interaction: momentum is conserved, but
        # no momentum block has a simpler form than a dense one.
        {"name": "hpsi_gauss_n12_m11", "op": "hpsi", "kind": "gauss", "N": 12, "M": 11, "g": 2.0},
        # The headline: H.psi of the Lieb-Liniger gas, 16 bosons in 10 orbitals.
        {"name": "hpsi_lieb_n16_m10", "op": "hpsi", "kind": "lieb", "N": 16, "M": 10, "g": 1.0},
        # The largest single space that the benchmark uses (ten million configurations).
        {"name": "hpsi_lieb_n20_m10", "op": "hpsi", "kind": "lieb", "N": 20, "M": 10, "g": 10.0},
        # More orbitals than bosons: an accurate orbital basis for few particles.
        {"name": "hpsi_lieb_n9_m13", "op": "hpsi", "kind": "lieb", "N": 9, "M": 13, "g": 1.0},
        # General orbitals (a time-dependent orbital basis): the reference's own test size.
        {"name": "hpsi_general_n10_m10", "op": "hpsi", "kind": "general", "N": 10, "M": 10, "g": 1.0},
        # General orbitals at the benchmark's size.
        {"name": "hpsi_general_n16_m10", "op": "hpsi", "kind": "general", "N": 16, "M": 10, "g": 1.0},
        # A host program's own arrays (page-locked), streamed through the device: the
        # drop-in way to call H.psi. Four states per call.
        {"name": "hpsi_host_n14_m9", "op": "host", "kind": "lieb", "N": 14, "M": 9, "g": 1.0, "states": 4},
        # rho1 and rho2 of one state: what every step of the orbital equations asks for.
        {"name": "densities_n16_m10", "op": "densities", "kind": "lieb", "N": 16, "M": 10, "g": 1.0},
        # Forward and backward of out = H psi in psi, Ho and Hint at the adjoint
        # configuration: H.psi, H^dagger phi and both transition densities. The smallest calls.
        {"name": "adjoint_n8_m8", "op": "adjoint", "kind": "general", "N": 8, "M": 8, "g": 1.0},
        # Ground state as the reference's driver computes its published table: five bosons,
        # eleven orbitals, nc / 8 Lanczos steps. Tiny vectors, thousands of launches.
        {"name": "ground_n5_m11", "op": "ground", "kind": "lieb", "N": 5, "M": 11, "g": 10.0, "steps": 375},
        # Ground state at the headline size: 150 Lanczos steps with full reorthogonalisation.
        {"name": "ground_n16_m10", "op": "ground", "kind": "lieb", "N": 16, "M": 10, "g": 1.0, "steps": 150},
        # A sweep over interaction strengths and uneven sizes, advanced together.
        {"name": "batch_24", "op": "batch", "kind": "lieb", "members": 24, "n_lo": 6, "n_hi": 12, "steps": 80, "pick": 2024},
    ]


def nc_of(n, m):
    return math.comb(n + m - 1, n) if n >= 0 else 0


def _fit(M, target, most):
    """The particle number whose space over M orbitals is nearest to `target`, at most `most` and 40 particles."""
    N = 2
    while N < 40 and nc_of(N + 1, M) <= most and abs(nc_of(N + 1, M) - target) <= abs(nc_of(N, M) - target):
        N += 1
    return N


def draw(rng):
    op = rng.choice(["hpsi"] * 6 + ["densities"] * 3 + ["adjoint"] * 2 + ["ground"] * 2 + ["host", "batch"])
    if op == "batch":
        return {"op": op, "kind": "lieb", "members": rng.randrange(6, 25), "n_lo": rng.randrange(3, 7), "n_hi": rng.randrange(8, 13),
                "steps": rng.randrange(30, 81), "pick": rng.randrange(1 << 20)}
    kind = {"hpsi": rng.choice(["lieb", "lieb", "gauss", "general"]), "densities": "lieb", "adjoint": "general",
            "ground": rng.choice(["lieb", "lieb", "gauss"]), "host": "lieb"}[op]
    lo, hi = {"hpsi": (1e3, 2.1e6 if kind == "general" else 1.01e7), "densities": (1e3, 2.1e6), "adjoint": (1e3, 1e5),
              "ground": (1e3, 2.1e6), "host": (1e5, 1e6)}[op]
    M = rng.randrange(5, 11 if op in ("adjoint", "host") else 13 if op == "densities" or kind == "general" else 15)
    if M >= 12:
        hi = min(hi, 1e6)
    target = 10.0 ** rng.uniform(math.log10(lo), math.log10(hi))
    N = _fit(M, target, hi)
    case = {"op": op, "kind": kind, "N": N, "M": M, "g": round(10.0 ** rng.uniform(-1, 1.5), 4)}
    if op == "host":
        case["states"] = rng.randrange(2, 7)
    if op == "ground":
        case["steps"] = max(2, min(rng.randrange(30, 151), nc_of(N, M) // 8))
    return case


# ---- inputs -------------------------------------------------------------------------------------


def _integrals(case, seed):
    """(Ho, flat Hint[k + s M + q M^2 + l M^3]) of a case, in plain numpy."""
    M, kind = case["M"], case["kind"]
    if kind == "general":
        rng = np.random.default_rng(seed)
        A = rng.standard_normal((M, M)) + 1j * rng.standard_normal((M, M))
        t = (rng.standard_normal(M ** 4) + 1j * rng.standard_normal(M ** 4)).reshape(M, M, M, M)  # axes (l, q, s, k)
        t = case["g"] * (t + t.transpose(0, 1, 3, 2) + t.transpose(1, 0, 2, 3) + t.transpose(1, 0, 3, 2)) / 4.0
        return (A + A.conj().T) / 2.0, ((t + np.conj(t.transpose(2, 3, 0, 1))) / 2.0).reshape(-1)
    k = 2 * np.pi * (np.arange(M) - M // 2)
    Ho = np.diag(0.5 * k * k).astype(np.complex128)
    i = np.arange(M)
    l, q, s, kk = np.meshgrid(i, i, i, i, indexing="ij")
    v = (lambda p: np.exp(-0.5 * (0.35 * p) ** 2)) if kind == "gauss" else (lambda p: np.ones(p.shape))
    t = np.where(kk + s == q + l, case["g"] * 0.5 * (v(kk - l) + v(kk - q)), 0.0)
    return Ho, t.reshape(-1).astype(np.complex128)


def _state(n, seed, device="cuda"):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = torch.randn(n, dtype=torch.complex128, device="cuda", generator=gen)
    x /= torch.linalg.vector_norm(x)
    return x if device == "cuda" else x.cpu()


def _members(case):
    """(N, M, g) of a sweep's members: the sizes from the case alone."""
    rng = np.random.default_rng(case["pick"])
    n = rng.integers(case["n_lo"], case["n_hi"] + 1, case["members"])
    m = rng.choice(M_BATCH, case["members"])
    g = 10.0 ** rng.uniform(-2.0, 2.0, case["members"])
    return [(int(a), int(b), float(c)) for a, b, c in zip(n, m, g)]


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        members = _members(case)
        b = mc.Batch([(n, m) for n, m, _ in members], case["steps"], device=DEVICE)
        for k, (n, m, g) in enumerate(members):
            b.set_integrals(k, *mc.lieb_integrals(m, g))
            b.set_start(k, _state(b.nc[k], seed * 1000 + k, "cpu").numpy())
        return {"op": op, "batch": b}
    sp = mc.FockSpace(case["N"], case["M"], device=DEVICE)
    if case["kind"] == "lieb":
        sp.set_integrals(*mc.lieb_integrals(case["M"], case["g"]))
    else:
        sp.set_integrals(*_integrals(case, seed))
    s = {"op": op, "space": sp}
    if op == "host":
        s["x"] = [_state(sp.nc, seed * 1000 + k, "cpu").pin_memory() for k in range(case["states"])]
        s["out"] = [torch.empty(sp.nc, dtype=torch.complex128).pin_memory() for _ in range(case["states"])]
        return s
    s["x"] = _state(sp.nc, seed * 1000)
    if op == "hpsi":
        s["out"] = torch.empty_like(s["x"])
    elif op == "adjoint":
        s["y"] = _state(sp.nc, seed * 1000 + 1)
    elif op == "ground":
        s["steps"] = case["steps"]
    return s


def run(state):
    op = state["op"]
    if op == "batch":
        return state["batch"].run()                                   # energies, steps done
    sp = state["space"]
    if op == "hpsi":
        return sp.apply_h(state["x"], state["out"])
    if op == "host":
        return sp.apply_h_host(state["x"], state["out"])
    if op == "densities":
        return sp.rho1(state["x"]), sp.rho2(state["x"])
    if op == "adjoint":
        x, y = state["x"], state["y"]
        return sp.apply_h(x), sp.apply_h_adjoint(y), sp.trans_rho1(y, x), sp.trans_rho2(y, x)
    return sp.ground(state["x"], state["steps"])                      # energy, ground state, steps done


# ---- what a pass cannot do without --------------------------------------------------------------


def _hpsi_flops(kind, N, M):
    """Multiply-adds of the pair-space product (4 real operations each with real values, 8 with complex ones):
    contact interactions have one pair sum per total momentum, finite-range ones a block, general ones P x P."""
    P, n2 = M * (M + 1) // 2, nc_of(N - 2, M)
    if kind == "lieb":
        return 4.0 * 2 * P * n2
    if kind == "gauss":
        return 4.0 * n2 * (P + sum((K // 2 - max(0, K - M + 1) + 1) ** 2 for K in range(2 * M - 1)))
    return 8.0 * P * P * n2


def work(case):
    op = case["op"]
    if op == "batch":
        b = f = 0.0
        for n, m, _ in _members(case):
            c = nc_of(n, m)
            b += sum(2.0 * 16 * c * (i + 2) for i in range(case["steps"] - 1)) + 16.0 * c
            f += sum(2.0 * 8 * c * (i + 2) for i in range(case["steps"] - 1)) + case["steps"] * _hpsi_flops("lieb", n, m)
        return {"bytes": b, "flops": f}
    N, M, c = case["N"], case["M"], nc_of(case["N"], case["M"])
    P, n1, n2 = M * (M + 1) // 2, nc_of(N - 1, M), nc_of(N - 2, M)
    if op == "hpsi":
        return {"bytes": 32.0 * c, "flops": _hpsi_flops(case["kind"], N, M)}
    if op == "host":
        return {"bytes": 32.0 * c * case["states"], "flops": case["states"] * _hpsi_flops(case["kind"], N, M)}
    if op == "densities":
        return {"bytes": 2 * 16.0 * c + 16.0 * (M ** 2 + M ** 4), "flops": 4.0 * (M * (M + 1) * n1 + P * (P + 1) * n2)}
    if op == "adjoint":
        return {"bytes": 2 * 32.0 * c + 2 * 32.0 * c + 16.0 * (M ** 2 + M ** 4),
                "flops": 2 * _hpsi_flops("general", N, M) + 8.0 * (M * M * n1 + P * P * n2)}
    steps = case["steps"]
    return {"bytes": sum(2.0 * 16 * c * (i + 2) for i in range(steps - 1)) + 32.0 * c,
            "flops": sum(2.0 * 8 * c * (i + 2) for i in range(steps - 1)) + steps * _hpsi_flops(case["kind"], N, M)}


# ---- the same results in 64 bits, from the definitions ------------------------------------------


def _prefix(N, M):
    """Prefix counts P_i = v_0 + .. + v_i (int64, (M, nc)) of every N-particle configuration, in index order."""
    nc = nc_of(N, M)
    R = nc - 1 - torch.arange(nc, device="cuda")
    P = torch.empty((M, nc), dtype=torch.int64, device="cuda")
    P[M - 1] = N
    for i in range(M - 2, -1, -1):
        t = torch.tensor([math.comb(p + i, i + 1) for p in range(N + 1)], device="cuda")
        P[i] = torch.searchsorted(t, R, right=True) - 1
        R = R - t[P[i]]
    return P


def _holes(N, M, order):
    """For every hole configuration m of N - order particles and every orbital (order 1) or pair q <= l
    (order 2): index of m plus those particles, and <m|a_q a_l|that>."""
    P = _prefix(N - order, M)
    v = torch.diff(P, dim=0, prepend=torch.zeros_like(P[:1])).to(torch.float64)
    tabs = [torch.tensor([math.comb(p + i, i + 1) for p in range(N + 1)], device="cuda") for i in range(M - 1)]
    cols = [(q, l) for q in range(M) for l in range(q, M)] if order == 2 else [(q, None) for q in range(M)]
    idx = torch.empty((len(cols), P.shape[1]), dtype=torch.int64, device="cuda")
    c = torch.empty((len(cols), P.shape[1]), dtype=torch.float64, device="cuda")
    for x, (q, l) in enumerate(cols):
        s = torch.zeros_like(P[0])
        for i in range(M - 1):
            s += tabs[i][P[i] + (i >= q) + (l is not None and i >= l)]
        idx[x] = nc_of(N, M) - 1 - s
        c[x] = torch.sqrt(v[q] + 1) if l is None else torch.sqrt((v[q] + 1) * (v[l] + (2 if q == l else 1)))
    return idx, c


class _Exact:
    """The operators of one space as gathers to the hole spaces and products there."""

    def __init__(self, N, M, Ho, Hint):
        self.N, self.M, self.nc = N, M, nc_of(N, M)
        self.h2 = _holes(N, M, 2) if N >= 2 else None
        self.pairs = [(q, l) for q in range(M) for l in range(q, M)]
        T = Hint.reshape(M, M, M, M)      # axes (l, q, s, k)
        A = np.zeros((len(self.pairs), len(self.pairs)), np.complex128)
        for x, (k, s) in enumerate(self.pairs):
            for y, (q, l) in enumerate(self.pairs):
                A[x, y] = 0.5 * sum(T[b, a, d, c] for c, d in {(k, s), (s, k)} for a, b in {(q, l), (l, q)})
        self.A = torch.from_numpy(A).cuda()
        self.Ho = torch.from_numpy(np.asarray(Ho)).cuda()
        if np.count_nonzero(Ho - np.diag(np.diag(Ho))):
            self.h1 = _holes(N, M, 1)
        else:
            P = _prefix(N, M).to(torch.float64)
            v = torch.diff(P, dim=0, prepend=torch.zeros_like(P[:1]))
            self.h1, self.diag = None, torch.einsum("k,kn->n", self.Ho.diagonal().real, v)

    @staticmethod
    def _back(holes, E, out):
        idx, c = holes
        for x in range(idx.shape[0]):
            out[idx[x]] += c[x] * E[x]

    def apply(self, psi):
        if self.h1 is None:
            out = self.diag * psi
        else:
            out = torch.zeros_like(psi)
            self._back(self.h1, self.Ho @ (self.h1[1] * psi[self.h1[0]]), out)
        if self.h2 is not None:
            self._back(self.h2, self.A @ (self.h2[1] * psi[self.h2[0]]), out)
        return out

    def rho1(self, phi, psi):
        idx, c = _holes(self.N, self.M, 1)
        return (c * phi[idx]).conj() @ (c * psi[idx]).T

    def rho2(self, phi, psi):
        idx, c = self.h2
        G = (c * phi[idx]).conj() @ (c * psi[idx]).T
        M, at = self.M, {}
        for x, (q, l) in enumerate(self.pairs):
            at[q, l] = at[l, q] = x
        to = torch.tensor([at[k, s] * len(self.pairs) + at[q, l] for l in range(M) for q in range(M) for s in range(M) for k in range(M)], device="cuda")
        return G.reshape(-1)[to]

    def energy(self, x, steps):
        """Lowest eigenvalue after `steps` Lanczos steps from x, fully reorthogonalised (twice)."""
        V = torch.empty((steps, self.nc), dtype=torch.complex128, device="cuda")
        V[0] = x
        d, e = [], []
        for i in range(steps):
            r = self.apply(V[i])
            d.append(torch.vdot(V[i], r).real)
            for _ in range(2):
                r = r - V[: i + 1].T @ (V[: i + 1].conj() @ r)
            if i + 1 < steps:
                e.append(torch.linalg.vector_norm(r))
                V[i + 1] = r / e[-1]
        T = torch.diag(torch.stack(d))
        if e:
            T += torch.diag(torch.stack(e), 1) + torch.diag(torch.stack(e), -1)
        return float(torch.linalg.eigvalsh(T)[0])


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        out = []
        for k, (n, m, g) in enumerate(_members(case)):
            one = {"kind": "lieb", "M": m, "g": g}
            out.append(_Exact(n, m, *_integrals(one, seed)).energy(_state(nc_of(n, m), seed * 1000 + k), case["steps"]))
        return np.array(out), None
    N, M = case["N"], case["M"]
    x = _Exact(N, M, *_integrals(case, seed))
    psi = _state(x.nc, seed * 1000)
    if op == "hpsi":
        return x.apply(psi)
    if op == "host":
        return [x.apply(_state(x.nc, seed * 1000 + k)) for k in range(case["states"])]
    if op == "densities":
        return x.rho1(psi, psi), x.rho2(psi, psi)
    if op == "adjoint":
        phi = _state(x.nc, seed * 1000 + 1)
        return x.apply(psi), x.apply(phi), x.rho1(phi, psi), x.rho2(phi, psi)
    return x.energy(psi, case["steps"]), None, None   # the vector's sign is the solver's own
