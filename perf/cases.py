"""Workloads of the engine, each one pass through its public entry points.

A case names an entry point (`kind`), a basis (a pyrochlore lattice of the package, sublattice up-counts or the whole
ice manifold, spinon pairs) and the options of the call.  The Hamiltonian is the ring-exchange and Zeeman model of
`build_ring_zeeman` with couplings and field drawn from the seed, as a point of a phase diagram; bases with a spinon
pair also carry the bond hopping, whose images mostly leave the basis.

  apply     y (+)= H x, one FP64 vector: what an outer solver calls, matrix-free or on the materialised operator
  batched   Y (+)= H X for R vectors stored [row][R], FP64 or FP32
  solve     the lowest eigenvalues by thick-restart Lanczos (the mfsparse algorithm), FP64 or mixed precision
  eigval0   the ground-state energy by the plain three-term Lanczos (the mfeig0 algorithm)
  ftlm      finite-temperature Lanczos recurrences of R random vectors in one or several sectors
  expect    ring expectation values and ring-ring correlations of a few eigenvector-like vectors
"""
from __future__ import annotations

import json
import math

import numpy as np
import torch

import qsi_subspace_ed_gb300 as q
from qsi_subspace_ed_gb300 import workloads

DEVICE = "cuda"
KAPPA = 0.5

# Bases by name: lattice, sublattice up-counts (None: the whole two-in-two-out manifold), spinon pairs.  Beside each
# its number of states.
BASES = {
    "32s4.4.4.4": ("pyro_1x2x1", (4, 4, 4, 4), 0),          # 388
    "32q0": ("pyro_1x2x1", None, 0),                        # 3,618
    "32q0p1": ("pyro_1x2x1", None, 1),                      # 7,236
    "32q0p2": ("pyro_1x2x1", None, 2),                      # 234,044
    "64s4.4.12.12": ("pyro_1x2x2", (4, 4, 12, 12), 0),      # 15,528
    "64s4.8.8.12": ("pyro_1x2x2", (4, 8, 8, 12), 0),        # 36,056
    "64s6.6.10.10": ("pyro_1x2x2", (6, 6, 10, 10), 0),      # 113,952
    "64s8.8.8.8": ("pyro_1x2x2", (8, 8, 8, 8), 0),          # 221,628
    "64s8.8.8.8p1": ("pyro_1x2x2", (8, 8, 8, 8), 1),        # 443,256
    "64q0": ("pyro_1x2x2", None, 0),                        # 2,891,562
    "64q0p1": ("pyro_1x2x2", None, 1),                      # 5,783,124
    "96s4.4.20.20": ("pyro_1x2x3", (4, 4, 20, 20), 0),      # 113,244
    "96s4.12.12.20": ("pyro_1x2x3", (4, 12, 12, 20), 0),    # 797,256
    "96s6.6.18.18": ("pyro_1x2x3", (6, 6, 18, 18), 0),      # 3,160,224
    "96s8.8.16.16": ("pyro_1x2x3", (8, 8, 16, 16), 0),      # 30,812,529
    "96s12.12.12.12": ("pyro_1x2x3", (12, 12, 12, 12), 0),  # 196,465,480
}
STATES = {"32s4.4.4.4": 388, "32q0": 3618, "32q0p1": 7236, "32q0p2": 234044, "64s4.4.12.12": 15528,
          "64s4.8.8.12": 36056, "64s6.6.10.10": 113952, "64s8.8.8.8": 221628, "64s8.8.8.8p1": 443256,
          "64q0": 2891562, "64q0p1": 5783124, "96s4.4.20.20": 113244, "96s4.12.12.20": 797256,
          "96s6.6.18.18": 3160224, "96s8.8.16.16": 30812529, "96s12.12.12.12": 196465480}


def listed():
    return [
        # The smallest call: one apply inside a user's own Krylov loop on the 32-spin cell.
        {"name": "apply_f64_32spin", "kind": "apply", "basis": "32q0", "materialised": False, "accumulate": False},
        # The ordinary apply, on the whole manifold of the 64-spin cell.
        {"name": "apply_f64_64spin", "kind": "apply", "basis": "64q0", "materialised": False, "accumulate": False},
        # The largest: the zero-winding sector of the 96-spin cell, the benchmark's headline.
        {"name": "apply_f64_96spin", "kind": "apply", "basis": "96s12.12.12.12", "materialised": False,
         "accumulate": False},
        # diag_DOQSI_ham --algorithm sparse: the operator materialised once, then applied; the y += H x form.
        {"name": "apply_sparse_96spin", "kind": "apply", "basis": "96s8.8.16.16", "materialised": True,
         "accumulate": True},
        # FTLM's block of random vectors in mixed precision on a large sector.
        {"name": "batched_mixed_r64_96spin", "kind": "batched", "basis": "96s8.8.16.16", "R": 64, "dtype": "float32",
         "materialised": False, "accumulate": False},
        # A handful of FP64 vectors at an odd count (a user's block method), projected hopping, y += H x.
        {"name": "batched_f64_r5_64spin", "kind": "batched", "basis": "64s8.8.8.8p1", "R": 5, "dtype": "float64",
         "materialised": False, "accumulate": True},
        # The default solve of diag_DOQSI_ham on a small cell: one eigenpair, launch and latency bound.
        {"name": "solve_f64_32spin", "kind": "solve", "basis": "32q0", "precision": "f64", "nev": 1, "ncv": 15,
         "tol": 1e-10, "vectors": True, "materialised": False},
        # A phase-diagram point: ground state and gap on the 64-spin cell, in plain FP64 ...
        {"name": "solve_f64_64spin", "kind": "solve", "basis": "64q0", "precision": "f64", "nev": 2, "ncv": 24,
         "tol": 1e-9, "vectors": False, "materialised": False},
        # ... and in mixed precision with the FP64 polish.
        {"name": "solve_mixed_64spin", "kind": "solve", "basis": "64q0", "precision": "mixed", "nev": 2, "ncv": 24,
         "tol": 1e-9, "vectors": False, "materialised": False},
        # The mfeig0 algorithm with its default 5,000 iterations on a mid-sized sector.
        {"name": "eigval0_64spin", "kind": "eigval0", "basis": "64s8.8.8.8", "iterations": 5000},
        # Finite temperature: three sectors of uneven size (none, one and two spinon pairs) advanced together.
        {"name": "ftlm_mixed_sectors", "kind": "ftlm", "basis": "64q0,64q0p1,32q0p2", "R": 16, "M": 24,
         "precision": "mixed"},
        # eval_observables on two eigenvectors: rings and ring-ring correlations.
        {"name": "expect_64spin", "kind": "expect", "basis": "64s8.8.8.8", "nvec": 2, "cross": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pick(rng, most, least=0):
    """A basis of between `least` and `most` states, spread over the logarithm of its size."""
    names = [k for k in BASES if least <= STATES[k] <= most]
    want = rng.uniform(math.log(STATES[min(names, key=STATES.get)]), math.log(STATES[max(names, key=STATES.get)]))
    near = sorted(names, key=lambda k: abs(math.log(STATES[k]) - want))
    return near[min(len(near) - 1, rng.randrange(2))]


def draw(rng):
    kind = rng.choice(["apply", "apply", "batched", "batched", "batched", "solve", "solve", "eigval0", "ftlm", "ftlm",
                       "expect"])
    if kind == "apply":
        return {"kind": kind, "basis": _pick(rng, 40_000_000), "materialised": rng.random() < 0.4,
                "accumulate": rng.random() < 0.4}
    if kind == "batched":
        dtype = rng.choice(["float32", "float32", "float64"])
        R = rng.choice([16, 32, 64, 128]) if dtype == "float32" and rng.random() < 0.4 else _log_int(rng, 2, 130)
        return {"kind": kind, "basis": _pick(rng, min(6_000_000, 400_000_000 // R)), "R": R, "dtype": dtype,
                "materialised": rng.random() < 0.3, "accumulate": rng.random() < 0.3}
    if kind == "solve":  # the second level only where the sector is known to be one connected piece
        basis = rng.choice(["32q0", "64s4.8.8.12", "64s6.6.10.10", "64s8.8.8.8", "64q0", "96s4.4.20.20"])
        return {"kind": kind, "basis": basis, "precision": rng.choice(["f64", "mixed"]),
                "nev": rng.choice([1, 2]) if basis in ("32q0", "64s8.8.8.8", "64q0") else 1,
                "ncv": rng.randint(12, 30), "tol": rng.choice([1e-9, 1e-10]), "vectors": False,
                "materialised": rng.random() < 0.4}
    if kind == "eigval0":
        return {"kind": kind, "basis": _pick(rng, 900_000, 3000), "iterations": _log_int(rng, 400, 3000)}
    if kind == "ftlm":
        return {"kind": kind, "basis": ",".join(_pick(rng, 3_500_000, 10_000) for _ in range(rng.choice([1, 1, 2]))),
                "R": rng.choice([1, 4, 8, 16, 32, 64]), "M": rng.randint(10, 24),
                "precision": rng.choice(["mixed", "mixed", "f64"])}
    return {"kind": kind, "basis": _pick(rng, 800_000, 300), "nvec": rng.randint(1, 4), "cross": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs
_bases: dict = {}  # the host arrays of the bases met so far: what a user's program has read from its basis files


def _basis(name):
    if name not in _bases:
        lat, sector, pairs = BASES[name]
        _bases[name] = q.enumerate_basis_gpu(workloads.lattice(lat), sector=sector, n_spinon_pairs=pairs)
    return _bases[name]


def _params(name, seed):
    """Ring couplings by hexagon type, field, and the hopping of bases with spinon pairs."""
    rng = np.random.default_rng([seed, 11])
    g = [float(v) for v in rng.uniform(0.2, 1.0, 4)]
    B = [float(v) for v in rng.uniform(-0.5, 0.5, 3)]
    return g, B, 0.05 if BASES[name][2] else 0.0


def _randn(shape, dtype, seed):
    gen = torch.Generator(DEVICE).manual_seed(int(seed))
    return torch.randn(shape, dtype=dtype, device=DEVICE, generator=gen)


def _operator(name, seed, materialised=False):
    g, B, jpm = _params(name, seed)
    op = q.LazyOpSum(q.ZBasis(_basis(name)), q.build_ring_zeeman(workloads.lattice(BASES[name][0]), g, B, Jpm=jpm))
    if materialised:
        op.materialise(True)
    return op


def _vectors(case, seed):
    """x and the y that is accumulated into: N(0, 1) entries over sqrt(states)."""
    n = len(_basis(case["basis"]))
    shape = (n, case["R"]) if case["kind"] == "batched" else (n,)
    dtype = getattr(torch, case.get("dtype", "float64"))
    x = _randn(shape, dtype, 2 * seed).mul_(n ** -0.5)
    y = _randn(shape, dtype, 2 * seed + 1).mul_(n ** -0.5) if case["accumulate"] else torch.zeros_like(x)
    return x, y


def _psi(case, seed):
    """Orthonormal columns, as eigenvectors are."""
    n = len(_basis(case["basis"]))
    return np.ascontiguousarray(torch.linalg.qr(_randn((n, case["nvec"]), torch.float64, seed))[0].cpu().numpy())


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ftlm":
        names = case["basis"].split(",")
        return {"case": case, "seed": seed, "ops": [_operator(b, seed) for b in names]}
    if kind == "expect":
        lat = workloads.lattice(BASES[case["basis"]][0])
        return {"case": case, "basis": q.ZBasis(_basis(case["basis"])), "rings": q.get_ring_ops(lat)[0],
                "psi": _psi(case, seed)}
    state = {"case": case, "seed": seed, "op": _operator(case["basis"], seed, case.get("materialised", False))}
    if kind in ("apply", "batched"):
        state["x"], state["y"] = _vectors(case, seed)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        if case["accumulate"]:
            state["op"].evaluate_add(state["x"], state["y"])
        else:
            state["op"].evaluate(state["x"], state["y"])
        return state["y"]
    if kind == "batched":
        state["op"].apply_batched(state["x"], state["y"], accumulate=case["accumulate"])
        return state["y"]
    if kind == "solve":
        evals, evecs, _ = q.diagonalise(state["op"], nev=case["nev"], ncv=case["ncv"], tol=case["tol"],
                                        seed=state["seed"], precision=case["precision"],
                                        want_vectors=case["vectors"])
        return [evals, evecs] if case["vectors"] else [evals]
    if kind == "eigval0":
        return np.array([q.eigval0(state["op"], seed=state["seed"], max_iterations=case["iterations"],
                                   calc_eigenvector=False)[0]])
    if kind == "ftlm":
        return q.ftlm(state["ops"], [case["R"]] * len(state["ops"]), M=case["M"], seed=state["seed"],
                      precision=case["precision"])
    expect, cross = q.expectations(state["basis"], state["rings"], state["psi"], cross=case["cross"])
    return [expect, cross] if case["cross"] else [expect]


def work(case):
    """States and vectors read once and results written once, per apply; a row has about one admitted off-diagonal
    term for every six spins.  Solves count their usual number of Lanczos steps, each with one read of half the
    Krylov basis on average."""
    def one(name, R, size):
        n, spins = STATES[name], int(name[:2])
        return n * (16 + 2 * R * size), 2 * n * R * (spins / 6 + 1), n

    kind = case["kind"]
    if kind == "ftlm":
        size = 4 if case["precision"] == "mixed" else 8
        got = [one(b, case["R"], size) for b in case["basis"].split(",")]
        return {"bytes": case["M"] * sum(b + 3 * n * case["R"] * size for b, _, n in got),
                "flops": case["M"] * sum(f + 8 * n * case["R"] for _, f, n in got)}
    size = 4 if case.get("dtype") == "float32" else 8
    b, f, n = one(case["basis"], case.get("R", 1), size)
    if kind == "solve":
        steps = 80
        return {"bytes": steps * (b + n * 4 * case["ncv"]), "flops": steps * (f + 2 * n * case["ncv"])}
    if kind == "eigval0":
        return {"bytes": case["iterations"] * b, "flops": case["iterations"] * (f + 6 * n)}
    if kind == "expect":
        rings, nv = int(case["basis"][:2]), case["nvec"]
        k = rings * nv
        return {"bytes": 16 * n + 8 * n * nv + (8 * n * k if case["cross"] else 0),
                "flops": 2 * n * k * nv + (n * k * k if case["cross"] else 0)}
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ the same results in 64 bits, by plain torch
_TOP = -(1 << 63)  # flipping the top bit maps unsigned order onto signed order


class _Plain:
    """H of a case by masks, gathers and binary searches over the sorted states."""

    def __init__(self, name, g, B, jpm):
        lohi = _basis(name)
        self.n = n = len(lohi)
        words = torch.from_numpy(lohi.view(np.int64)).to(DEVICE)
        self.lo, self.hi = words[:, 0].contiguous(), words[:, 1].contiguous()
        del words
        path = workloads.LATTICE_DIR / (BASES[name][0] + ".json")
        lat = json.loads(path.read_text())
        self.rings = [r for r in lat["rings"] if len(r["member_spin_idx"]) == 6]
        # a state's key: its position among the distinct high words, then among the distinct low words
        self.ulo = torch.unique(self.lo ^ _TOP)
        self.uhi = torch.unique(self.hi)
        self.keys = self._key(self.lo, self.hi)
        self.patterns = []  # (coefficient, spins up before, spins down before)
        for r in self.rings:
            plus = [s for s, v in zip(r["member_spin_idx"], r["signs"]) if v == 1]
            minus = [s for s, v in zip(r["member_spin_idx"], r["signs"]) if v != 1]
            self.patterns += [(-g[int(r["sl"])], minus, plus), (-g[int(r["sl"])], plus, minus)]
        if jpm:
            for b in lat["bonds"]:
                i, j = int(b["from_idx"]), int(b["to_idx"])
                self.patterns += [(-jpm, [i], [j]), (-jpm, [j], [i])]
        axes = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]], dtype=np.float64) / math.sqrt(3.0)
        self.diag = torch.zeros(n, dtype=torch.float64, device=DEVICE)
        for i, a in enumerate(lat["atoms"]):
            up = ((self.lo if i < 64 else self.hi) >> (i % 64)) & 1
            self.diag += -KAPPA * float(axes[int(a["sl"])] @ np.asarray(B)) * (2 * up - 1).double()

    def _key(self, lo, hi):
        return torch.searchsorted(self.uhi, hi) * len(self.ulo) + torch.searchsorted(self.ulo, lo ^ _TOP)

    def entries(self, up, down):
        """(rows, columns) of one pattern: rows whose spins `up` are up and `down` are down, and whose flipped state
        is in the basis."""
        def masks(spins):
            m = [0, 0]
            for s in spins:
                m[s // 64] |= 1 << (s % 64)
            return [v - (1 << 64) if v >> 63 else v for v in m]
        u, x = masks(up), masks(list(up) + list(down))
        rows = (((self.lo & x[0]) == u[0]) & ((self.hi & x[1]) == u[1])).nonzero().squeeze(1)
        lo, hi = self.lo[rows] ^ x[0], self.hi[rows] ^ x[1]
        at = torch.searchsorted(self.keys, self._key(lo, hi)).clamp_(max=self.n - 1)
        found = (self.lo[at] == lo) & (self.hi[at] == hi)
        return rows[found], at[found]

    def apply(self, x):
        x = x.double()
        y = (self.diag * x if x.ndim == 1 else self.diag[:, None] * x)
        for c, up, down in self.patterns:
            rows, cols = self.entries(up, down)
            for a in range(0, len(rows), 1 << 22):
                y.index_add_(0, rows[a:a + (1 << 22)], x[cols[a:a + (1 << 22)]], alpha=c)
        return y

    def matrix(self):
        r, c, v = [torch.arange(self.n, device=DEVICE)], [torch.arange(self.n, device=DEVICE)], [self.diag]
        for k, up, down in self.patterns:
            rows, cols = self.entries(up, down)
            r.append(rows), c.append(cols), v.append(torch.full((len(rows),), k, dtype=torch.float64, device=DEVICE))
        coo = torch.sparse_coo_tensor(torch.stack([torch.cat(r), torch.cat(c)]), torch.cat(v), (self.n, self.n))
        return coo.coalesce().to_sparse_csr()


def _lowest(H, k):
    """The k lowest distinct eigenvalues: dense, or Lanczos with full reorthogonalisation."""
    n = H.shape[0]
    if n <= 4000:
        return torch.linalg.eigvalsh(H.to_dense())[:k].cpu().numpy()
    m = min(n, 260)
    V = torch.zeros(m + 1, n, dtype=torch.float64, device=DEVICE)
    v = _randn((n,), torch.float64, 1)
    V[0] = v / v.norm()
    a, b, last = np.zeros(m), np.zeros(m), None
    for j in range(m):
        w = H @ V[j]
        a[j] = float(V[j] @ w)
        for _ in range(2):
            w -= V[:j + 1].T @ (V[:j + 1] @ w)
        b[j] = float(w.norm())
        V[j + 1] = w / b[j]
        if j >= 60 and j % 20 == 0 or j == m - 1:
            T = np.diag(a[:j + 1]) + np.diag(b[:j], 1) + np.diag(b[:j], -1)
            ev = np.linalg.eigvalsh(T)[:k]
            if last is not None and np.abs(ev - last).max() < 1e-13 * np.abs(ev).max():
                return ev
            last = ev
    return last


def _shr(z, k):
    return (z >> k) & ((1 << (64 - k)) - 1)


def _signed(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _splitmix(z):
    z = z + _signed(0x9E3779B97F4A7C15)
    z = (z ^ _shr(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _recurrence(H, R, M, seed):
    """Three-term Lanczos of R random sign vectors (the signs are the top bits of a hash of seed, column and row)."""
    n = H.shape[0]
    i = torch.arange(n, device=DEVICE)[:, None]
    r = torch.arange(R, device=DEVICE)[None, :]
    up = _splitmix(_splitmix((r << 40) ^ i) ^ _signed(seed)) < 0
    cur = torch.where(up, n ** -0.5, -n ** -0.5).to(torch.float64)
    prev = torch.zeros_like(cur)
    al, be = np.zeros((R, M)), np.zeros((R, M))
    beta = torch.zeros(R, dtype=torch.float64, device=DEVICE)
    for j in range(M):
        w = H @ cur
        alpha = (cur * w).sum(0)
        w -= alpha * cur
        w -= beta * prev
        beta = w.square().sum(0).sqrt()
        al[:, j], be[:, j] = alpha.cpu().numpy(), beta.cpu().numpy()
        prev, cur = cur, w / beta
    return al, be


def exact(case, seed):
    kind = case["kind"]
    names = case["basis"].split(",")
    if max(STATES[b] for b in names) > 50_000_000:
        return None  # the searches alone take over twenty seconds
    if kind == "ftlm":
        return [_recurrence(_Plain(b, *_params(b, seed)).matrix(), case["R"], case["M"], seed + s)
                for s, b in enumerate(names)]
    P = _Plain(names[0], *_params(names[0], seed))
    if kind in ("apply", "batched"):
        x, y = _vectors(case, seed)
        out = P.apply(x)
        return out.add_(y) if case["accumulate"] else out
    if kind == "solve":
        evals = _lowest(P.matrix(), case["nev"])
        return [evals, None] if case["vectors"] else [evals]  # an eigenvector's sign is free
    if kind == "eigval0":
        return _lowest(P.matrix(), 1)
    psi = torch.from_numpy(_psi(case, seed)).to(DEVICE)
    nv, L = psi.shape[1], len(P.rings)
    W = torch.zeros(L, nv, P.n, dtype=torch.float64, device=DEVICE)
    for k in range(L):
        r = P.rings[k]
        plus = [s for s, v in zip(r["member_spin_idx"], r["signs"]) if v == 1]
        minus = [s for s, v in zip(r["member_spin_idx"], r["signs"]) if v != 1]
        rows, cols = P.entries(minus, plus)  # O raises `plus` and lowers `minus`: row's image is the column
        W[k][:, cols] = psi[rows].T
    W = W.reshape(L * nv, P.n)
    expect = (W @ psi).reshape(L, nv, nv).cpu().numpy()
    if not case["cross"]:
        return [expect]
    gram = (W @ W.T).reshape(L, nv, L, nv).permute(0, 2, 1, 3)
    return [expect, gram.contiguous().cpu().numpy()]
