"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is a deck (a box of C3D4 or C3D20 elements as decks.py generates them: jittered
nodes, one face clamped, a load on the opposite face; material, jitter and load from the
seed) and what the user does with it:

  text     deck bytes in memory -> displacements on the host: parse, upload, solve, read back
  arrays   the same from binary mesh arrays
  solve    a *STATIC step of a model in hand: reset the state, solve, read the displacements
  nlgeom   an NLGEOM step of a model in hand: temperature-dependent material, thermal load,
           amplitude, increments, Newton iterations
  batch    many small decks in hand through batch_solve
  serve    mixed decks through the request loop
  forces   internal and thermal forces of a displacement field
  matrix   the assembled stiffness as CSR on the host
  stress   nodal stress and strain of a displacement field

exact() gives the same outputs from plain 64-bit torch.
"""
import math

import numpy as np
import torch

import ferrix_b200 as fx
from ferrix_b200 import decks

# ------------------------------------------------------------------ the cases


def listed():
    return [
        # the smallest decks a user has: the size of the reference's own test decks, from text
        dict(name="text_c3d20_1k", kind="text", npe=20, nx=3, ny=2, nz=9),
        # the C3D4 cantilever of the tests (24,000 tets, 14,883 DOF), as its deck arrives
        dict(name="text_c3d4_15k", kind="text", npe=4, nx=10, ny=10, nz=40),
        # an ordinary solid part that arrives as arrays, odd cell counts
        dict(name="arrays_c3d20_93k", kind="arrays", npe=20, nx=13, ny=11, nz=49),
        # a large linear-tet model in hand, solved again (another load, a parameter study)
        dict(name="solve_c3d4_205k", kind="solve", npe=4, nx=33, ny=41, nz=47, precision="mixed"),
        # the benchmark's C3D20 box: the largest deck
        dict(name="solve_c3d20_417k", kind="solve", npe=20, nx=20, ny=20, nz=80, precision="mixed"),
        # FP64 throughout, as a user who wants the last digits asks for
        dict(name="solve_fp64_c3d20_45k", kind="solve", npe=20, nx=9, ny=10, nz=36, precision="fp64"),
        # the NLGEOM beam of the tests at an ordinary size: ten increments of Newton iterations
        dict(name="nlgeom_c3d4_16k", kind="nlgeom", npe=4, nx=48, ny=9, nz=10, increments=10),
        # a parameter sweep: small decks (2k to 60k DOF) solved as one batch
        dict(name="batch_c3d4_24", kind="batch", npe=4, decks=24, dof_lo=2000, dof_hi=60000, sizes=7),
        # a service: mixed decks submitted at once to the request loop's four slots
        dict(name="serve_mixed_12", kind="serve", npe=0, decks=12, dof_lo=5000, dof_hi=150000, sizes=2027),
        # what an outer nonlinear driver evaluates again and again
        dict(name="forces_c3d20_121k", kind="forces", npe=20, nx=15, ny=14, nz=44),
        # a caller that brings its own linear solver
        dict(name="matrix_c3d4_48k", kind="matrix", npe=4, nx=19, ny=23, nz=33),
        # result fields after a solve
        dict(name="stress_c3d20_205k", kind="stress", npe=20, nx=17, ny=19, nz=48),
    ]


# DOF range of a kind's decks: the smallest decks up to what its largest listed case costs
_RANGES = {"text": (600, 60e3), "arrays": (600, 200e3), "solve": (600, 400e3), "nlgeom": (1500, 16e3),
           "forces": (3e3, 200e3), "matrix": (3e3, 50e3), "stress": (3e3, 250e3)}


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["text", "arrays", "solve", "solve", "solve", "nlgeom", "batch", "serve", "forces", "matrix",
                       "stress"])
    if kind in ("batch", "serve"):
        return dict(kind=kind, npe=4 if kind == "batch" else 0, decks=rng.randint(3, 16), dof_lo=2000,
                    dof_hi=int(_log_uniform(rng, 15e3, 60e3)), sizes=rng.randint(1, 10 ** 6))
    npe = 4 if kind == "nlgeom" else rng.choice([4, 20])
    dof = _log_uniform(rng, *_RANGES[kind])
    side = [rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6), rng.uniform(1.0, 4.0)]  # slender along the load path
    s = (dof / 3.0 / (1.0 if npe == 4 else 4.0) / (side[0] * side[1] * side[2])) ** (1.0 / 3.0)
    nx, ny, nz = (max(2, round(a * s)) for a in side)
    case = dict(kind=kind, npe=npe, nx=nx, ny=ny, nz=nz)
    if kind == "solve":
        case["precision"] = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "nlgeom":
        case.update(nx=max(nx, ny, nz), ny=min(nx, ny, nz), nz=sorted((nx, ny, nz))[1], increments=rng.randint(2, 10))
    return case


# The reference solves with a sparse Cholesky factorisation, so its users have a direct solver's digits:
# a relative residual of 1e-10 leaves displacements good to about ten (the default 1e-8 leaves an error
# of up to 1e-9 on slender parts).
RTOL = 1e-10

# ------------------------------------------------------------------ inputs


def _mesh(npe, nx, ny, nz, lengths, rng):
    if npe == 20:
        return decks.hex20_box(nx, ny, nz, *lengths, jitter=0.1, seed=int(rng.integers(1 << 30)))
    m = decks.tet_box(nx, ny, nz, *lengths)
    inner = np.all((m.lattice > 0) & (m.lattice < np.array([nx, ny, nz])), axis=1)
    m.xyz[inner] += rng.uniform(-0.1, 0.1, size=(int(inner.sum()), 3)) * np.array(lengths) / np.array([nx, ny, nz])
    return m


def _spec(case, seed):
    """The deck of a single-deck case: unit cells (the NLGEOM beam: 50 x 10 x 10), material and load from the seed."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["kind"] in ("nlgeom", "forces", "stress"):
        beam = (50.0, 10.0, 10.0) if case["kind"] == "nlgeom" else (float(nx), float(ny), float(nz))
        m = _mesh(case["npe"], nx, ny, nz, beam, rng)
        long = int(np.argmax(beam))
        e, nu = float(rng.uniform(1.9e5, 2.2e5)), float(rng.uniform(0.28, 0.32))
        inc = case.get("increments", 1)
        dt = 1.0 / inc
        return decks.DeckSpec(m, [(e, nu, 20.0), (0.94 * e, nu, 220.0)], expansion=(1.2e-5, 20.0), clamp_axis=long,
                              load_total=(0.0, 0.0, -6.0e4 * float(rng.uniform(0.5, 1.0))),
                              nlgeom=case["kind"] == "nlgeom", static_line=f"{dt!r}, 1.0, 1e-05, {dt!r}",
                              amplitude=[(0.0, 0.0), (1.0, 1.0)],
                              init_temp=20.0 + 200.0 * m.xyz[:, long] / beam[long])
    return _box(_mesh(case["npe"], nx, ny, nz, (float(nx), float(ny), float(nz)), rng), 2, rng)


def _box(mesh, axis, rng):
    e = float(np.exp(rng.uniform(math.log(7.0e4), math.log(2.1e5))))
    d = rng.normal(size=3)
    load = d / np.linalg.norm(d) * float(rng.uniform(100.0, 5000.0))
    return decks.DeckSpec(mesh, [(e, float(rng.uniform(0.25, 0.35)), None)], clamp_axis=axis,
                          load_total=tuple(float(v) for v in load))


def _population(case, seed):
    """The decks of a batch or serving case: sizes from the case, material, jitter and load from the seed."""
    sizes, rng = np.random.default_rng(case["sizes"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["decks"]):
        npe = case["npe"] or (20 if sizes.uniform() < 0.4 else 4)
        dof = math.exp(sizes.uniform(math.log(case["dof_lo"]), math.log(case["dof_hi"])))
        L = sizes.uniform(10.0, 40.0, size=3)
        s = (dof / 3.0 / (1.0 if npe == 4 else 4.0) / float(np.prod(L))) ** (1.0 / 3.0)
        cells = [max(2, int(round(v * s))) for v in L]
        out.append(_box(_mesh(npe, *cells, tuple(float(v) for v in L), rng), int(sizes.integers(0, 3)), rng))
    return out


def _field(mesh, seed):
    """A smooth displacement field with noise, as a driver's iterate is."""
    rng = np.random.default_rng(seed + 1)
    c = mesh.xyz / mesh.xyz.max(axis=0)
    u = np.stack([np.sin(c @ rng.uniform(-3, 3, 3) + rng.uniform(0, 6)) for _ in range(3)], axis=1)
    return (1e-2 * (u + 1e-3 * rng.normal(size=u.shape))).ravel()


# ------------------------------------------------------------------ the passes

_KEPT = {}  # one context (and one server) per process, as a program on one GPU has


def _context():
    if "ctx" not in _KEPT:
        _KEPT["ctx"] = fx.Context(0)
    return _KEPT["ctx"]


def _server():
    if "srv" not in _KEPT:
        _KEPT["srv"] = fx.Server(0, slots=4, hbm_budget_bytes=16e9, opts=fx.solve_opts(rtol=RTOL))
    return _KEPT["srv"]


def _in_hand(spec, ctx):
    """A parsed model bound to the context with its state initialised (mesh on the device)."""
    p = fx.Project.from_arrays(**decks.deck_arrays(spec), ctx=ctx)
    st = fx.SolutionState(p.num_dofs, p.num_nodes)
    st.initialize(p)
    return p, st


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    s = dict(kind=kind, ctx=ctx, opts=fx.solve_opts(
        precision=fx.PREC_FP64 if case.get("precision") == "fp64" else fx.PREC_MIXED, rtol=RTOL))
    if kind == "batch":
        s["models"] = [_in_hand(spec, ctx) for spec in _population(case, seed)]
        return s
    if kind == "serve":
        s["server"] = _server()
        s["models"] = [fx.Project.from_arrays(**decks.deck_arrays(spec)) for spec in _population(case, seed)]
        return s
    spec = _spec(case, seed)
    if kind == "text":
        s["deck"] = decks.write_deck(spec).encode()
    elif kind == "arrays":
        s["arrays"] = decks.deck_arrays(spec)
    else:
        s["project"], s["state"] = _in_hand(spec, ctx)
        if kind in ("forces", "matrix", "stress"):
            s["u"] = _field(spec.mesh, seed)
        if kind in ("forces", "stress"):
            temp = spec.init_temp + 30.0
            s["state"].set_temperatures(t_cur=temp)
        if kind == "stress":
            s["state"].displacements = s["u"]
    return s


def _solve_deck(project, opts):
    state = fx.SolutionState(project.num_dofs, project.num_nodes)
    state.initialize(project)
    project.steps[0].solve(1, project, state, None, fx.SolverTime(), opts)
    u = state.displacements
    project.close()
    return u


def run(s):
    kind = s["kind"]
    if kind == "text":
        return _solve_deck(fx.Project.from_inp_text(s["deck"], s["ctx"]), s["opts"])
    if kind == "arrays":
        return _solve_deck(fx.Project.from_arrays(**s["arrays"], ctx=s["ctx"]), s["opts"])
    if kind in ("solve", "nlgeom"):
        s["state"].initialize(s["project"])
        s["project"].steps[0].solve(1, s["project"], s["state"], None, fx.SolverTime(), s["opts"])
        return s["state"].displacements
    if kind == "batch":
        for p, st in s["models"]:
            st.initialize(p)
        fx.batch_solve(s["ctx"], [p for p, _ in s["models"]], s["opts"])
        return [st.displacements for _, st in s["models"]]
    if kind == "serve":
        tickets = [s["server"].submit(p) for p in s["models"]]
        return [s["server"].wait(t)[0] for t in tickets]
    if kind == "forces":
        return s["project"].internal_force(s["u"]), s["project"].thermal_force()
    if kind == "matrix":
        return s["project"].assemble_csr(s["u"])
    return s["project"].nodal_stress_strain()


def _counts(case):
    """(nodes, elements, 3x3 blocks of K) of a case's decks, together."""
    if "decks" in case:
        cells = [m.mesh.dims + (m.mesh.npe,) for m in _population(case, 0)]
    else:
        cells = [(case["nx"], case["ny"], case["nz"], case["npe"])]
    n = e = b = 0
    for x, y, z, npe in cells:
        if npe == 4:
            nodes, elems, blocks = (x + 1) * (y + 1) * (z + 1), 6 * x * y * z, 15
        else:
            mids = x * (y + 1) * (z + 1) + (x + 1) * y * (z + 1) + (x + 1) * (y + 1) * z
            nodes, elems, blocks = (x + 1) * (y + 1) * (z + 1) + mids, x * y * z, 42
        n, e, b = n + nodes, e + elems, b + blocks * nodes
    return n, e, b


def work(case):
    """Mesh and field in, result out; a solve reads and writes its matrix once and computes it once."""
    n, e, b = _counts(case)
    npe = case["npe"] or 4
    mesh = 24.0 * n + 4.0 * npe * e
    stiff = 354780.0 if npe == 20 else 900.0
    kind = case["kind"]
    if kind == "forces":
        return {"bytes": mesh + 4 * 24.0 * n, "flops": 2 * e * stiff / 60.0}
    if kind == "stress":
        return {"bytes": mesh + 24.0 * n + 96.0 * n, "flops": 300.0 * npe * e}
    if kind == "matrix":
        return {"bytes": mesh + 9 * 16.0 * b, "flops": e * stiff}
    steps = case.get("increments", 1)
    return {"bytes": mesh + 24.0 * n + steps * 2 * 72.0 * b, "flops": steps * (e * stiff + 18.0 * b)}


# ------------------------------------------------------------------ 64-bit values in plain torch

_LOCAL20 = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1),
            (0, -1, -1), (1, 0, -1), (0, 1, -1), (-1, 0, -1), (0, -1, 1), (1, 0, 1), (0, 1, 1), (-1, 0, 1),
            (-1, -1, 0), (1, -1, 0), (1, 1, 0), (-1, 1, 0)]


def _shape(npe, pt):
    """(N, dN/dxi) of the linear tet or the 20-node serendipity brick at a local point."""
    if npe == 4:
        x, y, z = pt
        return np.array([1 - x - y - z, x, y, z]), np.array([[-1.0, 1, 0, 0], [-1.0, 0, 1, 0], [-1.0, 0, 0, 1]])
    N, dN = np.zeros(20), np.zeros((3, 20))
    for a, c in enumerate(_LOCAL20):
        f = [1 + pt[k] * c[k] if c[k] else 1 - pt[k] ** 2 for k in range(3)]
        g = [float(c[k]) if c[k] else -2 * pt[k] for k in range(3)]
        prod = f[0] * f[1] * f[2]
        d = [g[0] * f[1] * f[2], f[0] * g[1] * f[2], f[0] * f[1] * g[2]]
        if all(c):
            s = sum(pt[k] * c[k] for k in range(3)) - 2
            N[a] = prod * s / 8
            dN[:, a] = [(d[k] * s + prod * c[k]) / 8 for k in range(3)]
        else:
            N[a], dN[:, a] = prod / 4, [v / 4 for v in d]
    return N, dN


def _rule(npe):
    if npe == 4:
        return [((0.25, 0.25, 0.25), 1.0 / 6.0)]
    p, w = [-0.774596669241483, 0.0, 0.774596669241483], [0.5555555555555556, 0.8888888888888888, 0.5555555555555556]
    return [((p[i], p[j], p[k]), w[i] * w[j] * w[k]) for i in range(3) for j in range(3) for k in range(3)]


class _Plain:
    """A deck's finite element operators in 64-bit torch."""

    def __init__(self, spec):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        m = spec.mesh
        self.spec, self.npe, self.dev = spec, m.npe, dev
        self.x = torch.tensor(m.xyz, dtype=torch.float64, device=dev)
        self.conn = torch.tensor(m.conn, device=dev)
        n = self.x.shape[0]
        self.dofs = (3 * self.conn[:, :, None] + torch.arange(3, device=dev)).reshape(len(self.conn), -1)
        t0 = torch.zeros(n) if spec.init_temp is None else torch.tensor(spec.init_temp)
        self.t_init = t0.to(dev, torch.float64)
        self.t_cur = self.t_init.clone()
        rows = spec.materials
        self.tab = [[(0.0 if t is None else t) for _, _, t in rows], [e for e, _, _ in rows], [v for _, v, _ in rows]]
        fixed = decks.face_nodes(m, spec.clamp_axis, spec.clamp_side)
        self.fixed = torch.tensor((3 * fixed[:, None] + np.arange(3)).ravel(), device=dev)
        loaded = decks.face_nodes(m, spec.clamp_axis, 1 - spec.clamp_side)
        self.load = torch.zeros(n, 3, dtype=torch.float64, device=dev)
        self.load[torch.tensor(loaded, device=dev)] = torch.tensor(spec.load_total, dtype=torch.float64,
                                                                   device=dev) / len(loaded)
        self.load = self.load.reshape(-1)

    def lut(self, col, t):
        ts, vs = self.tab[0], self.tab[col]
        if len(ts) == 1:
            return torch.full_like(t, vs[0])
        f = ((t - ts[0]) / (ts[1] - ts[0])).clamp(0.0, 1.0)
        return vs[0] + (vs[1] - vs[0]) * f

    def elastic(self, t):
        """(lambda, mu) at temperature t."""
        e, nu = self.lut(1, t), self.lut(2, t)
        return e * nu / ((1 + nu) * (1 - 2 * nu)), e / (2 * (1 + nu))

    def thermal_strain(self, t_from, t_to):
        if self.spec.expansion is None:
            return torch.zeros_like(t_to)
        a, ref = self.spec.expansion
        return a * (t_to - ref) - a * (t_from - ref)

    def points(self, x, pts):
        """(N, gradients (E, 3, npe), |det J| w) at every point of a rule."""
        xe = x[self.conn]
        for pt, w in pts:
            N, dN = _shape(self.npe, pt)
            dN = torch.tensor(dN, device=self.dev)
            J = dN @ xe
            yield torch.tensor(N, device=self.dev), torch.linalg.solve(J, dN.expand(len(xe), -1, -1)), \
                torch.linalg.det(J).abs() * w

    def stiffness(self, x):
        n = self.npe
        te = self.t_cur[self.conn]
        K = torch.zeros(len(self.conn), 3 * n, 3 * n, dtype=torch.float64, device=self.dev)
        for N, g, w in self.points(x, _rule(n)):
            lam, mu = self.elastic(te @ N)
            gg = torch.einsum("eia,ejb->eaibj", g, g)
            k = gg * (lam * w)[:, None, None, None, None]
            k += gg.transpose(2, 4) * (mu * w)[:, None, None, None, None]
            tr = torch.einsum("eia,eib->eab", g, g) * (mu * w)[:, None, None]
            for i in range(3):
                k[:, :, i, :, i] += tr
            K += k.reshape(len(self.conn), 3 * n, 3 * n)
        return K

    def csr(self, x, penalty=True):
        K = self.stiffness(x)
        big = K.diagonal(dim1=1, dim2=2).max()
        n, k = self.x.numel(), 3 * self.npe
        i = self.dofs[:, :, None].expand(-1, -1, k).reshape(-1)
        j = self.dofs[:, None, :].expand(-1, k, -1).reshape(-1)
        v = K.reshape(-1)
        del K
        if penalty:
            i, j = torch.cat([i, self.fixed]), torch.cat([j, self.fixed])
            v = torch.cat([v, (1e6 * big).expand(len(self.fixed))])
        return torch.sparse_coo_tensor(torch.stack([i, j]), v, (n, n)).coalesce().to_sparse_csr(), big

    def force(self, x, u, sign):
        """sum B^T D (B u - eps_th) with B on x (u None: -eps_th alone), times sign."""
        te0, te1 = self.t_init[self.conn], self.t_cur[self.conn]
        f = torch.zeros(self.x.shape, dtype=torch.float64, device=self.dev)
        for N, g, w in self.points(x, _rule(self.npe)):
            t0, t1 = te0 @ N, te1 @ N
            lam, mu = self.elastic(t1)
            eye = torch.eye(3, dtype=torch.float64, device=self.dev)
            eps = -self.thermal_strain(t0, t1)[:, None, None] * eye
            if u is not None:
                grad = torch.einsum("eia,eaj->eij", g, u.reshape(-1, 3)[self.conn])
                eps = eps + (grad + grad.transpose(1, 2)) / 2
            tr = eps.diagonal(dim1=1, dim2=2).sum(1)
            sig = lam[:, None, None] * tr[:, None, None] * eye + 2 * mu[:, None, None] * eps
            fe = (sign * w)[:, None, None] * torch.einsum("eij,eib->ebj", sig, g)
            f.index_add_(0, self.conn.reshape(-1), fe.reshape(-1, 3))
        return f.reshape(-1)


def _pcg(A, b, rtol):
    """Jacobi-preconditioned CG, scalars kept on the device between checks."""
    d = _diagonal(A)
    x, r = torch.zeros_like(b), b.clone()
    z = r / d
    p, rz = z.clone(), r @ z
    stop = rtol * rtol * rz
    for it in range(1, 60000):
        q = A @ p
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        z = r / d
        new = r @ z
        p = z + (new / rz) * p
        rz = new
        if it % 50 == 0 and bool(rz <= stop):
            break
    return x


def _diagonal(A):
    rows = torch.repeat_interleave(torch.arange(A.shape[0], device=A.device), A.crow_indices().diff())
    on = rows == A.col_indices()
    return A.values()[on]


def _direct(A, b):
    """A x = b to 64-bit accuracy: dense Cholesky while it fits, else CG; one refinement."""
    if A.shape[0] <= 24000:
        L = torch.linalg.cholesky(A.to_dense())
        one = lambda v: torch.cholesky_solve(v[:, None], L)[:, 0]  # noqa: E731
        x = one(b)
        return x + one(b - A @ x)
    x = _pcg(A, b, 1e-12)
    return x + _pcg(A, b - A @ x, 1e-5)


def _linear(spec):
    m = _Plain(spec)
    A, _ = m.csr(m.x)
    return _direct(A, m.load).cpu().numpy()


def _newton(spec, increments):
    """The NLGEOM step: equal increments, the load along the amplitude, Newton to |R| / |F| < 1e-3."""
    m = _Plain(spec)
    u = torch.zeros_like(m.load)
    free = torch.ones_like(u)
    free[m.fixed] = 0.0
    cur, dt = 0.0, 1.0 / increments
    while cur < 1.0:
        if cur + dt > 1.0:
            dt = 1.0 - cur
        now = cur + dt
        for _ in range(15):
            f = m.load * now + m.force(m.x, None, -1.0)
            x = m.x + u.reshape(-1, 3)
            r = f - m.force(x, u, 1.0)
            if float((r * free).norm() / (f * free).norm()) < 1e-3:
                break
            A, big = m.csr(x)
            r[m.fixed] -= 1e6 * big * u[m.fixed]
            u = u + _direct(A, r)
        else:
            return None  # cut back: not a case of these ranges
        cur += dt
    return u.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if "decks" in case:
        return [_linear(spec) for spec in _population(case, seed)]
    spec = _spec(case, seed)
    if kind in ("text", "arrays", "solve"):
        return _linear(spec)
    if kind == "nlgeom":
        return _newton(spec, case["increments"])
    m = _Plain(spec)
    u = torch.tensor(_field(spec.mesh, seed), device=m.dev)
    if kind == "matrix":
        A, big = m.csr(m.x + u.reshape(-1, 3), penalty=False)
        return None, None, A.values().cpu().numpy(), float(big)
    m.t_cur = m.t_init + 30.0
    if kind == "forces":
        return (m.force(m.x, u, 1.0).cpu().numpy(), m.force(m.x, None, -1.0).cpu().numpy())
    S = torch.zeros(m.x.shape[0], 6, dtype=torch.float64, device=m.dev)
    E, count = torch.zeros_like(S), torch.zeros(m.x.shape[0], dtype=torch.float64, device=m.dev)
    for a, (_, g, _) in enumerate(m.points(m.x, [(p, 1.0) for p in _LOCAL20])):
        node = m.conn[:, a]
        grad = torch.einsum("eia,eaj->eij", g, u.reshape(-1, 3)[m.conn])
        th = m.thermal_strain(m.t_init[node], m.t_cur[node])
        lam, mu = m.elastic(m.t_cur[node])
        d = [grad[:, k, k] - th for k in range(3)]
        shear = [grad[:, i, j] + grad[:, j, i] for i, j in ((0, 1), (1, 2), (0, 2))]
        e = torch.stack(d + shear, dim=1)
        tr = (d[0] + d[1] + d[2]) * lam
        s = torch.stack([tr + 2 * mu * v for v in d] + [mu * v for v in shear], dim=1)
        S.index_add_(0, node, s)
        E.index_add_(0, node, e)
        count.index_add_(0, node, torch.ones_like(th))
    return (S / count[:, None]).cpu().numpy(), (E / count[:, None]).cpu().numpy()
