"""The solver's work as its users have it done, in cases that can be timed.

Each case is one call (or the few calls that belong together) of the public
Python API on inputs made from a seed:

  maps     the constraint maps A u and A^T w on device vectors, instance-interleaved
  project  the PSD-cone projection Update_xz, from host state (``host``) or on
           device vectors without allocation (``device``)
  gemm     the projection's dense block product, FP64 or on the tensor cores
  warm     the learned warm start's network: forward pass, or loss and gradient
  solve    whole boundary-point solves, to their stopping test

``n`` is the number of active orbitals everywhere; the active spaces are the
seeded synthetic ones of ``v2rdm_casscf_b200.hamiltonian`` (C1, singlet).
"""
import math

import numpy as np
import torch

import v2rdm_casscf_b200 as V
from v2rdm_casscf_b200.hamiltonian import ActiveSpace, synthetic

DEVICE = "cuda:0"
HIDDEN = 224  # width of the warm start's hidden layers (the network's default)
FEATURES, OUTPUTS = 16, 3

# The product mode of the solver, as bench.py runs it, and the plain mode (the reference's loop).
PRODUCT = dict(projection="adaptive", start="feasible", cg_extrapolate=True, anderson_memory=10, mixed_precision=True)
PLAIN = dict(projection="exact", start="feasible")
# A solve fixes the energies only to its tolerances, the primal and dual vectors to less (the dual is not
# unique), so the solves return the energies; the product mode, whose path to them moves with rounding, runs
# to tight tolerances.
PRODUCT_OPTIONS = dict(MU_UPDATE_FREQUENCY=250, R_CONVERGENCE=1e-8, E_CONVERGENCE=1e-9)
PLAIN_OPTIONS = dict(R_CONVERGENCE=1e-6, E_CONVERGENCE=1e-7)


def listed():
    return [
        # one CG map pair of a single (10e,10o) instance, the H10 layout: latency and launches
        dict(name="maps_n10", kind="maps", n=10, nvec=1, positivity="DQG"),
        # the batched workload's largest layout group: 19 instances of n = 20, an odd interleave
        dict(name="maps_n20x19", kind="maps", n=20, nvec=19, positivity="DQG"),
        # three-particle conditions: many more rows, a small odd group
        dict(name="maps_t2_n8x3", kind="maps", n=8, nvec=3, positivity="DQGT2"),
        # one large instance, tables and vectors beyond L2
        dict(name="maps_n28", kind="maps", n=28, nvec=1, positivity="DQG"),
        # projection of a small active space inside a program that owns all device memory
        dict(name="project_device_n5", kind="project", entry="device", n=5, positivity="DQG", mu=1.0),
        # one projection step of the (10e,10o) layout from host state (blocks up to 200)
        dict(name="project_host_n10", kind="project", entry="host", n=10, positivity="DQG", mu=1.0),
        # the same with blocks up to 450, odd sizes
        dict(name="project_host_n15", kind="project", entry="host", n=15, positivity="DQG", mu=1.0),
        # FP64 eigenvector update V^T W of every block above 64 of five n = 13 instances (ragged sizes)
        dict(name="gemm_fp64_n13x5", kind="gemm", n=13, count=5, blocks="all", tensor=False, ta=True, tb=False,
             scaled=False),
        # mixed-precision rebuild V D V^T of the largest blocks of the n = 20 group (19 of 800)
        dict(name="gemm_tensor_n20x19", kind="gemm", n=20, count=19, blocks="largest", tensor=True, ta=False, tb=True,
             scaled=True),
        # one training gradient of the warm start on a minibatch of 4,096 pairs
        dict(name="warm_gradient_4096", kind="warm", op="gradient", rows=4096),
        # two small spaces of unlike size in the plain mode: one lock-step group each, launches and barriers count
        dict(name="solve_plain_n4_5", kind="solve", mode="plain", nmin=4, nmax=5, count=2, space=0),
        # one (10e,10o) space in the product mode, the layout and options of the benchmark
        dict(name="solve_product_n10", kind="solve", mode="product", nmin=10, nmax=10, count=1, space=1),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["maps", "maps", "maps", "project", "project", "gemm", "gemm", "warm", "solve"])
    if kind == "maps":
        if rng.random() < 0.25:
            pos = rng.choice(["DQGT1", "DQGT2"])
            return dict(kind=kind, n=rng.randint(4, 8), nvec=_log_int(rng, 1, 6), positivity=pos)
        n = _log_int(rng, 4, 28)
        return dict(kind=kind, n=n, nvec=_log_int(rng, 1, max(1, min(32, 19 * 20**4 // n**4))), positivity="DQG")
    if kind == "project":
        mu = round(math.exp(rng.uniform(math.log(0.2), math.log(5.0))), 3)
        if rng.random() < 0.4:
            return dict(kind=kind, entry="device", n=rng.randint(2, 5), positivity=rng.choice(["DQG", "DQ"]), mu=mu)
        return dict(kind=kind, entry="host", n=rng.randint(4, 15), positivity=rng.choice(["DQG", "DQG", "DQ", "DG"]),
                    mu=mu)
    if kind == "gemm":
        tensor = rng.random() < 0.5
        n = rng.randint(15, 20) if tensor else rng.randint(6, 16)
        return dict(kind=kind, n=n, count=_log_int(rng, 1, 19 if tensor else 8),
                    blocks="largest" if tensor else rng.choice(["all", "largest"]), tensor=tensor,
                    ta=rng.random() < 0.5, tb=rng.random() < 0.5, scaled=rng.random() < 0.5)
    if kind == "warm":
        return dict(kind=kind, op=rng.choice(["forward", "gradient"]), rows=_log_int(rng, 36, 8192))
    if rng.random() < 0.5:
        return dict(kind=kind, mode="plain", nmin=5, nmax=5, count=rng.randint(1, 4), space=rng.randint(0, 11))
    n = rng.randint(5, 8)
    return dict(kind=kind, mode="product", nmin=n, nmax=n, count=rng.randint(1, 3), space=rng.randint(0, 11))


# ---- inputs ----------------------------------------------------------------

_layouts = {}  # one solver handle per layout: its index tables serve every instance of that layout


def _layout(n, positivity):
    key = (n, positivity)
    if key not in _layouts:
        _layouts[key] = V.V2RDMSolver([n], n // 2, n // 2, options=dict(POSITIVITY=positivity))
    return _layouts[key]


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _host_rng(seed):
    return np.random.Generator(np.random.Philox(key=[seed, 11]))


def _block_sizes(case):
    n = case["n"]
    gab, gaa = n * n, n * (n - 1) // 2
    one = [2 * gab] if case["blocks"] == "largest" else [gab, gaa, gaa, gab, gab, gaa, gaa, gab, gab, 2 * gab]
    return [d for d in one if d > 64] * case["count"]


def _padded(d):
    return (d + 63) // 64 * 64


def _start_vectors(case, seed, sizes):
    """x, y, z as the plugin's random start draws them: uniform in (-2, 0)."""
    g = _host_rng(seed)
    return [g.uniform(-2.0, 0.0, k) for k in sizes]


def _weights(seed):
    g = _host_rng(seed)
    dims = [FEATURES, HIDDEN, HIDDEN, HIDDEN, OUTPUTS]
    layers = []
    for i, o in zip(dims, dims[1:]):
        layers.append((g.normal(0.0, math.sqrt(2.0 / i), (o, i)).astype(np.float32),
                       g.normal(0.0, 0.05, o).astype(np.float32)))
    return layers


def _pairs(case, seed):
    """Features of orbital pairs (order one, the last a constant) and targets."""
    g = _host_rng(seed + 1)
    f = g.uniform(-1.0, 1.0, (case["rows"], FEATURES)).astype(np.float32)
    f[:, -1] = 1.0
    return f, g.normal(0.0, 0.3, (case["rows"], OUTPUTS)).astype(np.float32)


def _near(n, space, seed):
    """A neighbour of a fixed active space, as in a geometry scan: its integrals plus 2 % of another's."""
    a, b = synthetic(n, space), synthetic(n, seed)
    return ActiveSpace(a.h + 0.02 * b.h, a.L + 0.02 * b.L, a.na, a.nb)


def _solve_sizes(case):
    return [case["nmax"] - i % (case["nmax"] - case["nmin"] + 1) for i in range(case["count"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "maps":
        s = _layout(case["n"], case["positivity"])
        g = _generator(seed)
        nv = case["nvec"]
        u = torch.randn(s.dimx * nv, dtype=torch.float64, device=DEVICE, generator=g)
        w = torch.randn(s.nconstraints * nv, dtype=torch.float64, device=DEVICE, generator=g)
        au, atw = torch.empty_like(w), torch.empty_like(u)
        # a first application puts the layout's tables on the device
        s.map_batched_device(nv, u.data_ptr(), au.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return dict(case=case, solver=s, u=u, w=w, au=au, atw=atw)
    if kind == "project":
        s = V.V2RDMSolver.from_active_space(synthetic(case["n"], seed), options=dict(POSITIVITY=case["positivity"]))
        x, y, z = _start_vectors(case, seed, (s.dimx, s.nconstraints, s.dimx))
        state = dict(case=case, solver=s, keep=_layout(case["n"], case["positivity"]), x=x, y=y, z=z, mu=case["mu"])
        s.ATu(y)  # puts the layout's tables on the device
        if case["entry"] == "device":
            to = lambda a: torch.from_numpy(a).to(DEVICE)  # noqa: E731
            state |= dict(dc=to(s.c), dy=to(y), dx0=to(x), dx=to(x), dz=to(z))
        return state
    if kind == "gemm":
        dims = _block_sizes(case)
        total = sum(_padded(d) ** 2 for d in dims)
        g = _generator(seed)
        a, b = (torch.zeros(total, dtype=torch.float64, device=DEVICE) for _ in range(2))
        d = torch.zeros(sum(_padded(k) for k in dims), dtype=torch.float64, device=DEVICE)
        o = od = 0
        for k in dims:
            p = _padded(k)
            for m in (a, b):
                m[o:o + p * p].view(p, p)[:k, :k] = torch.randn(k, k, dtype=torch.float64, device=DEVICE,
                                                                generator=g) / math.sqrt(k)
            # half of the eigenvalue weights are zero, as in V max(L, 0) V^T
            d[od:od + k] = torch.randn(k, dtype=torch.float64, device=DEVICE, generator=g).clamp_min(0.0)
            o, od = o + p * p, od + p
        return dict(case=case, dims=dims, a=a, b=b, d=d if case["scaled"] else None, c=torch.empty_like(a))
    if kind == "warm":
        net = V.WarmStart(hidden=HIDDEN)
        net.params = np.concatenate([v.reshape(-1) for layer in _weights(seed) for v in layer])
        f, t = _pairs(case, seed)
        return dict(case=case, net=net, f=f, t=t)
    sizes = _solve_sizes(case)
    kw, options = (PRODUCT, PRODUCT_OPTIONS) if case["mode"] == "product" else (PLAIN, PLAIN_OPTIONS)
    solvers = [V.V2RDMSolver.from_active_space(_near(n, case["space"] + i, seed + 17 * i), options=options, **kw)
               for i, n in enumerate(sizes)]
    return dict(case=case, solvers=solvers, keep=[_layout(n, "DQG") for n in sorted(set(sizes))])


# ---- one pass --------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "maps":
        s, nv = state["solver"], case["nvec"]
        stream = torch.cuda.current_stream().cuda_stream
        s.map_batched_device(nv, state["u"].data_ptr(), state["au"].data_ptr(), stream)
        s.map_batched_device(nv, state["w"].data_ptr(), state["atw"].data_ptr(), stream, transpose=True)
        return state["au"], state["atw"]
    if kind == "project":
        s, mu = state["solver"], state["mu"]
        if case["entry"] == "device":
            state["dx"].copy_(state["dx0"])  # x is replaced by the projection
            s.update_xz_noalloc(mu, state["dc"].data_ptr(), state["dy"].data_ptr(), state["dx"].data_ptr(),
                                state["dz"].data_ptr(), torch.cuda.current_stream().cuda_stream)
            return state["dx"], state["dz"]
        s.set_state(state["x"], state["y"], state["z"], mu)
        s.update_xz(mu)
        x, _, z, _ = s.get_state()
        return x, z
    if kind == "gemm":
        d = state["d"]
        V.block_gemm_device(state["dims"], state["a"].data_ptr(), state["b"].data_ptr(), state["c"].data_ptr(),
                            trans_a=case["ta"], trans_b=case["tb"], d_d=None if d is None else d.data_ptr(),
                            tensor_cores=case["tensor"])
        return state["c"]
    if kind == "warm":
        if case["op"] == "forward":
            return state["net"].forward(state["f"])
        loss, grad = state["net"].gradient(state["f"], state["t"])
        return loss, grad
    solvers = state["solvers"]
    results = V.solve_batch(solvers)
    return np.array([r["e_primal"] for r in results]), np.array([r["e_dual"] for r in results])


# ---- what a pass cannot do without -----------------------------------------


def _shape(n, positivity):
    """(dimx, constraints, block sizes) of a layout."""
    s = _layout(n, positivity)
    return s.dimx, s.nconstraints, [int(d) for d in s.dimensions]


def work(case):
    kind = case["kind"]
    if kind == "maps":
        nx, nc, _ = _shape(case["n"], case["positivity"])
        return dict(bytes=16.0 * (nx + nc) * case["nvec"], flops=4.0 * nx * case["nvec"])
    if kind == "project":
        nx, nc, dims = _shape(case["n"], case["positivity"])
        # c, x and y in, x and z out; a symmetric eigendecomposition with vectors (9 n^3) and the two products
        return dict(bytes=8.0 * (4 * nx + nc), flops=float(sum(13 * d**3 for d in dims)))
    if kind == "gemm":
        dims = _block_sizes(case)
        return dict(bytes=24.0 * sum(d * d for d in dims), flops=2.0 * sum(d**3 for d in dims))
    if kind == "warm":
        weights = FEATURES * HIDDEN + 2 * HIDDEN * HIDDEN + HIDDEN * OUTPUTS
        times = 2 if case["op"] == "forward" else 6
        return dict(bytes=4.0 * (case["rows"] * (FEATURES + OUTPUTS) + 2 * weights),
                    flops=float(times * case["rows"] * weights))
    # a solve: about 500 outer iterations of 20 CG iterations (two maps each) and one projection
    total = dict(bytes=0.0, flops=0.0)
    for n in _solve_sizes(case):
        nx, nc, dims = _shape(n, "DQG")
        total["bytes"] += 500.0 * (20 * 16.0 * (nx + nc) + 8.0 * (4 * nx + nc))
        total["flops"] += 500.0 * (20 * 4.0 * nx + sum(13.0 * d**3 for d in dims))
    return total


# ---- the same in 64 bits, without the solver -------------------------------


class _DQG:
    """The D, Q and G constraint rows of a C1 singlet as a sparse matrix, from their definitions.

    Geminal (p, q) of opposite spin has index q n + p; same-spin geminals are those with p > q in that order."""

    def __init__(self, n, electrons, q2=True, g2=True):
        self.n, na = n, electrons // 2
        gab, gaa = n * n, n * (n - 1) // 2
        names = [("d2ab", gab), ("d2aa", gaa), ("d2bb", gaa), ("d200", gab), ("d1a", n), ("d1b", n), ("q1a", n),
                 ("q1b", n)]
        names += [("q2ab", gab), ("q2aa", gaa), ("q2bb", gaa)] if q2 else []
        names += [("g2ab", gab), ("g2ba", gab), ("g2aa", 2 * gab)] if g2 else []
        self.dim = dict(names)
        self.dims = [d for _, d in names]
        self.off = dict(zip(self.dim, np.concatenate([[0], np.cumsum(np.square(self.dims))[:-1]]).tolist()))
        self.dimx = int(np.sum(np.square(self.dims)))
        self.rows, self.parts = 0, []
        r = np.arange(n)
        pq = [(p, q) for q in range(n) for p in range(n) if p > q]
        ai, aj = (np.array([v[k] for v in pq], dtype=np.int64) for k in (0, 1))
        aa = np.zeros((n, n), dtype=np.int64)
        sign = np.zeros((n, n))
        aa[ai, aj] = aa[aj, ai] = np.arange(gaa)
        sign[ai, aj], sign[aj, ai] = -1.0, 1.0  # +1 where the first index is the smaller
        self.aa, self.sign = aa, sign
        ab = lambda p, q: q * n + p  # noqa: E731
        el = self.el
        i, j = (v.reshape(-1) for v in np.meshgrid(r, r, indexing="ij"))
        off_diagonal = i != j
        # traces of D2
        self.emit(1, 0, el("d2ab", ab(i, j), ab(i, j)), 1.0)
        for f in ("d2aa", "d2bb"):
            k = aa[i[off_diagonal], j[off_diagonal]]
            self.emit(1, 0, el(f, k, k), 1.0)
        # D1 + Q1 = 1
        for d, q in (("d1a", "q1a"), ("d1b", "q1b")):
            k = np.arange(n * n)
            self.emit(n * n, np.tile(k, 2), np.concatenate([el(d, j, i), el(q, i, j)]), 1.0)
        # contractions of D2 to D1
        a, b, c = (v.reshape(-1) for v in np.meshgrid(r, r, r, indexing="ij"))
        row = a * n + b
        for d, first in (("d1a", True), ("d1b", False)):
            x, y = (ab(a, c), ab(b, c)) if first else (ab(c, a), ab(c, b))
            self.emit(n * n, np.concatenate([i * n + j, row]), np.concatenate([el(d, i, j), el("d2ab", x, y)]),
                      np.concatenate([np.full(n * n, float(na)), np.full(row.size, -1.0)]))
        keep = (c != a) & (c != b)
        for d, f in (("d1a", "d2aa"), ("d1b", "d2bb")):
            ak, bk, ck = a[keep], b[keep], c[keep]
            self.emit(n * n, np.concatenate([i * n + j, row[keep]]),
                      np.concatenate([el(d, i, j), el(f, aa[ak, ck], aa[bk, ck])]),
                      np.concatenate([np.full(n * n, na - 1.0), -sign[ak, ck] * sign[bk, ck]]))
        # S^2 and the singlet relations
        self.emit(1, 0, el("d2ab", ab(i, j), ab(j, i)), 1.0)
        for d, f, m in (("d1a", "d1b", n), ("d2aa", "d2bb", gaa)):
            k = np.arange(m * m)
            self.emit(m * m, np.tile(k, 2), np.concatenate([self.off[d] + k, self.off[f] + k]),
                      np.repeat([1.0, -1.0], m * m))
        s, t = (v.reshape(-1) for v in np.meshgrid(np.arange(gaa), np.arange(gaa), indexing="ij"))
        si, sj, ti, tj = ai[s], aj[s], ai[t], aj[t]
        for f in ("d2aa", "d2bb"):
            self.emit(gaa * gaa, np.tile(np.arange(gaa * gaa), 5), np.concatenate([
                el(f, s, t), el("d2ab", ab(si, sj), ab(ti, tj)), el("d2ab", ab(sj, si), ab(ti, tj)),
                el("d2ab", ab(si, sj), ab(tj, ti)), el("d2ab", ab(sj, si), ab(tj, ti))]),
                np.repeat([1.0, -0.5, 0.5, 0.5, -0.5], gaa * gaa))
        g, h = (v.reshape(-1) for v in np.meshgrid(np.arange(gab), np.arange(gab), indexing="ij"))
        gi, gj, hi, hj = g % n, g // n, h % n, h // n
        k = np.arange(gab * gab)
        w = -0.5 / (np.where(gi == gj, math.sqrt(2.0), 1.0) * np.where(hi == hj, math.sqrt(2.0), 1.0))
        self.emit(k.size, np.tile(k, 5), np.concatenate([
            el("d200", g, h), el("d2ab", g, h), el("d2ab", ab(gj, gi), h), el("d2ab", g, ab(hj, hi)),
            el("d2ab", ab(gj, gi), ab(hj, hi))]), np.concatenate([np.ones(k.size), w, w, w, w]))
        if g2:
            x, y = (v.reshape(-1) for v in np.meshgrid(np.arange(gab), r, indexing="ij"))
            self.emit(gab, x, el("g2ba", x, ab(y, y)), 1.0)
            self.emit(gab, x, el("g2ba", ab(y, y), x), 1.0)
        if q2:
            self.emit_if(k.size, [(None, "d2ab", g, h, 1.0), (None, "q2ab", g, h, -1.0),
                                  (gj == hj, "d1a", hi, gi, -1.0), (gi == hi, "d1b", hj, gj, -1.0)])
            for d, q, o in (("d2aa", "q2aa", "d1a"), ("d2bb", "q2bb", "d1b")):
                self.emit_if(s.size, [(None, d, s, t, 1.0), (None, q, s, t, -1.0), (sj == tj, o, ti, si, -1.0),
                                      (sj == ti, o, tj, si, 1.0), (si == tj, o, ti, sj, 1.0),
                                      (si == ti, o, tj, sj, -1.0)])
        if g2:
            self.emit_if(k.size, [(None, "g2ab", g, h, -1.0), (gj == hj, "d1a", gi, hi, 1.0),
                                  (None, "d2ab", ab(gi, hj), ab(hi, gj), -1.0)])
            self.emit_if(k.size, [(None, "g2ba", g, h, -1.0), (gj == hj, "d1b", gi, hi, 1.0),
                                  (None, "d2ab", ab(hj, gi), ab(gj, hi), -1.0)])
            x, y = (v.reshape(-1) for v in np.meshgrid(np.arange(2 * gab), np.arange(2 * gab), indexing="ij"))
            xi, xj, yi, yj = x % gab % n, x % gab // n, y % gab % n, y % gab // n
            low, left = x < gab, y < gab
            entries = [(None, "g2aa", x, y, -1.0)]
            for same, d, f in ((low & left, "d1a", "d2aa"), (~low & ~left, "d1b", "d2bb")):
                entries.append((same & (xj == yj), d, xi, yi, 1.0))
                entries.append((same & (xi != yj) & (yi != xj), f, aa[xi, yj], aa[yi, xj],
                                -sign[xi, yj] * sign[yi, xj]))
            entries.append((low & ~left, "d2ab", ab(xi, yj), ab(xj, yi), 1.0))
            entries.append((~low & left, "d2ab", ab(yj, xi), ab(yi, xj), 1.0))
            self.emit_if(x.size, entries)

    def el(self, f, r, c):
        return self.off[f] + r * self.dim[f] + c

    def emit(self, count, rows, cols, vals):
        rows = np.broadcast_to(rows, cols.shape) + self.rows
        self.parts.append((rows, cols, np.broadcast_to(vals, cols.shape)))
        self.rows += count

    def emit_if(self, count, entries):
        rows, cols, vals = [], [], []
        for where, f, r, c, v in entries:
            k = np.arange(count) if where is None else np.nonzero(where)[0]
            rows.append(k)
            cols.append(self.el(f, r, c)[k])
            vals.append(np.broadcast_to(v, (count,))[k])
        self.emit(count, np.concatenate(rows), np.concatenate(cols), np.concatenate(vals))

    def matrix(self):
        r, c, v = (torch.from_numpy(np.concatenate([p[k] for p in self.parts])) for k in range(3))
        return r, c, v.to(torch.float64)

    def times(self, u, transpose):
        """A u (or A^T u) for the columns of u."""
        r, c, v = self.matrix()
        if transpose:
            r, c = c, r
        out = torch.zeros(self.dimx if transpose else self.rows, u.shape[1], dtype=torch.float64)
        for b in range(u.shape[1]):
            out[:, b].index_add_(0, r, v * u[c, b])
        return out

    def cost(self, space):
        """The cost vector: (ik|jl) on D2ab, its antisymmetrised form on D2aa and D2bb, h on D1."""
        n = self.n
        eri = space.eri()
        c = np.zeros(self.dimx)
        ab = np.einsum("ikjl->jilk", eri).reshape(n * n, n * n)  # row q n + p, column s n + r
        c[:self.dim["d2ab"] ** 2] = ab.reshape(-1)
        pq = np.array([q * n + p for q in range(n) for p in range(n) if p > q], dtype=np.int64)
        swapped = (pq % n) * n + pq // n
        same = ab[np.ix_(pq, pq)] - ab[np.ix_(pq, swapped)]
        for f in ("d2aa", "d2bb"):
            c[self.off[f]:self.off[f] + same.size] = same.reshape(-1)
        for f in ("d1a", "d1b"):
            c[self.off[f]:self.off[f] + n * n] = space.h.reshape(-1)
        return c


def exact(case, seed):
    kind = case["kind"]
    if kind == "maps":
        if case["positivity"] != "DQG":
            return None  # no definition of the three-particle rows outside the solver and its reference
        L = _DQG(case["n"], 2 * (case["n"] // 2))
        g = _generator(seed)
        nv = case["nvec"]
        u = torch.randn(L.dimx * nv, dtype=torch.float64, device=DEVICE, generator=g).cpu().view(-1, nv)
        w = torch.randn(L.rows * nv, dtype=torch.float64, device=DEVICE, generator=g).cpu().view(-1, nv)
        return L.times(u, False).reshape(-1), L.times(w, True).reshape(-1)
    if kind == "project":
        space = synthetic(case["n"], seed)
        L = _DQG(case["n"], 2 * (case["n"] // 2), "Q" in case["positivity"], "G" in case["positivity"])
        x, y, _ = _start_vectors(case, seed, (L.dimx, L.rows, L.dimx))
        U = L.times(torch.from_numpy(y)[:, None], True)[:, 0].numpy() - L.cost(space) + case["mu"] * x
        xs, zs = [], []
        o = 0
        for d in L.dims:
            m = U[o:o + d * d].reshape(d, d)
            lam, v = np.linalg.eigh(0.5 * (m + m.T))
            xs.append(((v * np.maximum(lam, 0.0) / case["mu"]) @ v.T).reshape(-1))
            zs.append(((v * np.maximum(-lam, 0.0)) @ v.T).reshape(-1))
            o += d * d
        return np.concatenate(xs), np.concatenate(zs)
    if kind == "gemm":
        s = prepare(case, seed)
        out, o, od = [], 0, 0
        for k in s["dims"]:
            p = _padded(k)
            a, b = (s[m][o:o + p * p].view(p, p) for m in ("a", "b"))
            a, b = a.T if case["ta"] else a, b.T if case["tb"] else b
            if s["d"] is not None:
                a = a * s["d"][od:od + p]
            out.append((a @ b).reshape(-1))
            o, od = o + p * p, od + p
        return torch.cat(out)
    if kind == "warm":
        f, t = _pairs(case, seed)
        acts = [torch.from_numpy(f).double()]
        # weights in bfloat16, biases in 32 bits, everything else in 64
        layers = [(torch.from_numpy(w).bfloat16().double().requires_grad_(),
                   torch.from_numpy(b).double().requires_grad_()) for w, b in _weights(seed)]
        for k, (w, b) in enumerate(layers):
            y = acts[-1] @ w.T + b
            acts.append(y if k == len(layers) - 1 else y.clamp_min(0.0))
        if case["op"] == "forward":
            return acts[-1].detach()
        loss = (acts[-1] - torch.from_numpy(t).double()).square().mean()
        loss.backward()
        return float(loss), torch.cat([v.grad.reshape(-1) for layer in layers for v in layer])
    return None  # a solve has no closed form
