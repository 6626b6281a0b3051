"""Performance cases of the injective-deformation step: what a program asks of
this package through its public entry points, from the smallest call to the
headline solve.

Kinds of case (``case["kind"]``):

* ``energy``: the allocation-free elastic energy over device arrays;
* ``step``: one implicit Euler step of a tet body (``advance``), driven by a
  velocity (a bar) or by the normal-flow predictor (the bumpy blob);
* ``batch``: one step of many uneven pairs of bars pushed into contact, all
  in one arena;
* ``flow``: one flow-mode step of a closed triangle shell;
* ``shell``: one frame of a character sequence on an elastic shell with
  moving Dirichlet rows;
* ``direction`` / ``gradient`` / ``hessian``: the Newton direction, the energy
  with its gradient, and a Hessian product at a program's own positions;
* ``contacts`` / ``ccd``: the constraint set, and the intersection-free step
  size, of a stack of plates a fraction of d-hat apart.

Meshes depend on a case's sizes only and are made once; everything a call
takes (positions, velocities, directions) is made from the seed. A step's
result is read back as the program reads it, positions into its own array,
with the energy and kappa of the call's result record (the velocity a context
holds after a step is (x - x^n) / h, nothing that these do not say).
"""
import ctypes
import functools
import math

import numpy as np
import torch

import idp_gb300 as idp
from idp_gb300 import meshgen
from idp_gb300.api import initialize_oipc

DENSITY, YOUNG, NU = 1000.0, 1e4, 0.3  # the tet workloads' material
H = 0.1                                # and time step
FLOW = 0.05                            # normal-flow distance of one step
SHELL = dict(h=0.04, density=1000.0, E=100.0, nu=0.4, thickness=0.01, dhat=0.01)
FLOWSHELL = dict(h=0.5, density=1000.0, thickness=0.01, step=0.005)
BATCH_GAP, BATCH_DHAT = 2e-3, 5e-3    # pairs of bars: gap before the step and d-hat
PLATE_CELL, PLATE_DHAT = 0.05, 0.01    # plate stacks: cube edge and d-hat


def listed():
    return [
        # a frame loop's energy probe on device buffers: the smallest call, two launches
        dict(name="energy on device arrays", kind="energy", shape="bar", nx=9, ny=7, nz=31),
        # one body of an interactive scene: a step that is nothing but latency
        dict(name="small bar step", kind="step", shape="bar", nx=3, ny=3, nz=9, fp64=False),
        # the headline workload: one normal-flow step of the 220k-tet blob
        dict(name="large blob step", kind="step", shape="blob", n=64, fp64=False),
        # the plain FP64 path on a mid-size body (reference results)
        dict(name="FP64 blob step", kind="step", shape="blob", n=30, fp64=True),
        # many independent bodies with self-contact in one arena
        dict(name="contact batch step", kind="batch", count=20, tmin=200, tmax=6000, fp64=False),
        # the reference's normal-flow script on a shell about the size of its cat.obj
        dict(name="shell flow step", kind="flow", n=48, fp64=False),
        # the character-sequence script under gravity: next frame as rest shape, velocity and DBC targets
        dict(name="elastic shell frame", kind="shell", n=41, fp64=False),
        # a program with its own outer loop: the linear solve alone, to FP64 accuracy
        dict(name="Newton direction", kind="direction", shape="blob", n=45, fp64=False),
        # an optimiser's objective and gradient at an odd small size
        dict(name="energy and gradient", kind="gradient", shape="bar", nx=7, ny=5, nz=13, fp64=False),
        # operator product in FP64 (eigenvalue or sensitivity codes)
        dict(name="FP64 Hessian product", kind="hessian", shape="bar", nx=11, ny=13, nz=45, fp64=True),
        # contact queries of a packed scene
        dict(name="plate stack contacts", kind="contacts", nx=33, ny=29, plates=7),
        dict(name="plate stack CCD", kind="ccd", nx=33, ny=29, plates=7),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["energy", "step", "step", "batch", "flow", "shell", "direction", "gradient", "hessian",
                       "contacts", "ccd"])
    c = dict(kind=kind)
    if kind in ("energy", "step", "direction", "gradient", "hessian"):
        c["shape"] = rng.choice(["bar", "blob"])
        if c["shape"] == "bar":
            c.update(nx=_log(rng, 2, 13), ny=_log(rng, 2, 13), nz=_log(rng, 5, 47))
        else:
            c.update(n=_log(rng, 12, 60))
        if kind != "energy":
            c["fp64"] = rng.random() < 0.3
        if c.get("fp64") and "n" in c:
            c["n"] = min(c["n"], 41)
    elif kind == "batch":
        c.update(count=rng.randint(3, 20), tmin=_log(rng, 100, 400), tmax=_log(rng, 1000, 6000), fp64=False)
    elif kind == "flow":
        c.update(n=_log(rng, 14, 60), fp64=rng.random() < 0.3)
    elif kind == "shell":
        c.update(n=_log(rng, 13, 41), fp64=False)
    else:
        c.update(nx=_log(rng, 5, 37), ny=_log(rng, 5, 37), plates=rng.randint(2, 8))
    return c


# ---------------------------------------------------------------- meshes and problems
@functools.lru_cache(maxsize=32)
def _bar(nx, ny, nz):
    cell = 1.0 / 6.0
    return meshgen.bar(nx, ny, nz, size=(cell * nx, cell * ny, cell * nz), jitter=0.05, seed=0)


@functools.lru_cache(maxsize=32)
def _blob(n):
    X, tets, _ = meshgen.blob(n=n, lmax=8, amp=0.3, seed=0)
    return X, tets


@functools.lru_cache(maxsize=32)
def _blob_shell(n):
    return meshgen.shell_from_tets(*_blob(n))


def _body(c):
    return _bar(c["nx"], c["ny"], c["nz"]) if c["shape"] == "bar" else _blob(c["n"])


@functools.lru_cache(maxsize=32)
def _plates(nx, ny, plates):
    """A stack of one-cube-thick jittered plates, each turned a little against
    the one below so that edges cross; gaps are set per seed."""
    X, tets = meshgen.bar(nx, ny, 1, size=(PLATE_CELL * nx, PLATE_CELL * ny, PLATE_CELL), jitter=0.0, seed=0)
    V = X.shape[0]
    mid = X.mean(0)
    Xs = []
    for p in range(plates):
        a = 0.11 * p
        R = np.array([[math.cos(a), -math.sin(a), 0.0], [math.sin(a), math.cos(a), 0.0], [0.0, 0.0, 1.0]])
        Xs.append((X - mid) @ R.T + [0.0, 0.0, 1.5 * PLATE_CELL * p])
    return np.concatenate(Xs), np.concatenate([tets + p * V for p in range(plates)]).astype(np.int32), V


def _tet_problem(X, tets, dHat=None):
    mass = meshgen.lumped_mass(X, tets, DENSITY)
    lam, mu = meshgen.lame(YOUNG, NU)
    dHat2 = (1e-3 * float(np.linalg.norm(X.max(0) - X.min(0))) if dHat is None else dHat) ** 2
    k, km = initialize_oipc(float(mass.mean()), dHat2)
    return dict(mass=mass, lam=lam, mu=mu, dHat2=dHat2, kappa=k, kappa_max=km)


@functools.lru_cache(maxsize=32)
def _body_problem(shape, a, b, c):
    X, tets = _bar(a, b, c) if shape == "bar" else _blob(a)
    return _tet_problem(X, tets)


def _problem_of(c):
    return _body_problem(c["shape"], *((c["nx"], c["ny"], c["nz"]) if c["shape"] == "bar" else (c["n"], 0, 0)))


def _smooth(rng, X, amp):
    """A smooth displacement field: three random plane waves, and a random affine part."""
    L = float(np.linalg.norm(X.max(0) - X.min(0)))
    U = (X - X.mean(0)) @ rng.normal(0.0, 0.3 * amp / L, (3, 3))
    for _ in range(3):
        k, d = rng.normal(0.0, 4.0 / L, 3), rng.normal(0.0, 0.3 * amp, 3)
        U = U + np.sin(X @ k + rng.uniform(0.0, 2 * math.pi))[:, None] * d
    return U


def _tet_inputs(c, seed):
    """Rest shape, current positions and velocity of a tet body."""
    X0, tets = _body(c)
    rng = np.random.default_rng(seed)
    X = X0 + _smooth(rng, X0, 0.02)
    return X0, tets, X, _smooth(rng, X0, 0.3)


def _tet_context(c, X0, tets, **params):
    p = _problem_of(c)
    ctx = idp.Context(h=H, mode=idp.MODE_FP64 if c["fp64"] else idp.MODE_MIXED, **params)
    ctx.add_instance(X0, tets, p["mass"], p["lam"], p["mu"], p["dHat2"], p["kappa"], p["kappa_max"])
    ctx.commit()
    return ctx, [p["kappa"], p["kappa_max"], 0.0]


@functools.lru_cache(maxsize=8)
def _batch_bodies(count, tmin, tmax):
    """Pairs of bars side by side BATCH_GAP apart, tet counts log-uniform."""
    rng = np.random.default_rng(count)
    out = []
    for i in range(count):
        t = math.exp(rng.uniform(math.log(tmin), math.log(tmax)))
        n = max(1, int(round((t / 20.0) ** (1.0 / 3.0))))
        X, tets = meshgen.bar(n, n, 2 * n, size=(1.0, 1.0, 2.0), jitter=0.05, seed=i)
        Y = X + [1.0 + BATCH_GAP, rng.uniform(-0.3, 0.3), rng.uniform(-0.3, 0.3)]
        X0 = np.concatenate([X, Y])
        T = np.concatenate([tets, tets + X.shape[0]]).astype(np.int32)
        out.append((X0, T, _tet_problem(X0, T, dHat=BATCH_DHAT)))
    return out


def _shell_rows(X):
    """DBC rows of the character-sequence script: the top of the bounding box."""
    lo, hi = X.min(0), X.max(0)
    return np.nonzero((X[:, 1] - lo[1]) >= 0.867 * (hi[1] - lo[1]))[0].astype(np.int32)


def _shell_mass(X, F, density, thickness):
    n = np.cross(X[F[:, 1]] - X[F[:, 0]], X[F[:, 2]] - X[F[:, 0]])
    m = np.zeros(X.shape[0])
    np.add.at(m, F.reshape(-1), np.repeat(np.linalg.norm(n, axis=1) / 2 * thickness * density / 3, 3))
    return m


def _turned(rng, X, degrees):
    """The next frame: turned about y, leant about z, stretched a little."""
    a, b = np.deg2rad(degrees * rng.uniform(0.5, 1.0)), np.deg2rad(0.5 * degrees * rng.uniform(0.5, 1.0))
    Ry = np.array([[np.cos(a), 0, np.sin(a)], [0, 1, 0], [-np.sin(a), 0, np.cos(a)]])
    Rz = np.array([[np.cos(b), -np.sin(b), 0], [np.sin(b), np.cos(b), 0], [0, 0, 1]])
    return (X * [1.0, 1.0 + 0.003 * rng.uniform(0.5, 1.0), 1.0]) @ (Rz @ Ry).T


def _dev(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=dtype)).cuda()


def _rest(X0, tets):
    """Row-major inverse rest basis (columns x1-x0, x2-x0, x3-x0) and volume."""
    Dm = np.stack([X0[tets[:, k]] - X0[tets[:, 0]] for k in (1, 2, 3)], axis=-1)
    return np.linalg.inv(Dm), np.linalg.det(Dm) / 6.0


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "energy":
        X0, tets = _body(c)
        IB, vol = _rest(X0, tets)
        lam, mu = meshgen.lame(YOUNG, NU)
        T = tets.shape[0]
        X = X0 + _smooth(np.random.default_rng(seed), X0, 0.02)
        s = dict(T=T, tets=_dev(tets, np.int32), X=_dev(X, np.float64), IB=_dev(IB.reshape(-1, 9), np.float64),
                 vol=_dev(vol, np.float64), lam=_dev(np.full(T, lam), np.float64), mu=_dev(np.full(T, mu), np.float64),
                 energy=torch.zeros(1, dtype=torch.float64, device="cuda"),
                 inverted=torch.zeros(1, dtype=torch.int32, device="cuda"))
    elif kind in ("step", "direction", "gradient", "hessian"):
        X0, tets, X, v = _tet_inputs(c, seed)
        params = dict(pcg_rel_tol=1e-12) if kind == "direction" else {}
        ctx, kappa = _tet_context(c, X0, tets, **params)
        s = dict(ctx=ctx, X=X, v=v, kappa=kappa, blob=c["shape"] == "blob", Xout=np.empty_like(X))
        if kind != "step":  # the sub-steps take the predictor from the context's own state
            ctx.set_velocity(0, v)
        if kind == "hessian":
            s["x"] = np.random.default_rng(seed + 1).normal(0.0, 1.0, X.shape)
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        # resting contact is stiff: a tighter stop than the default settles the positions to FP64 accuracy
        ctx = idp.Context(h=H, newton_tol=1e-5, mode=idp.MODE_FP64 if c["fp64"] else idp.MODE_MIXED)
        X, v, kappa = [], [], []
        for X0, tets, p in _batch_bodies(c["count"], c["tmin"], c["tmax"]):
            ctx.add_instance(X0, tets, p["mass"], p["lam"], p["mu"], p["dHat2"], p["kappa"], p["kappa_max"])
            half = X0.shape[0] // 2
            vi = _smooth(rng, X0, 0.02)
            vi[half:, 0] -= rng.uniform(0.2, 0.3)  # the second bar moves into the first
            X.append(X0)
            v.append(vi)
            kappa.append([p["kappa"], p["kappa_max"], 0.0])
        ctx.commit()
        s = dict(ctx=ctx, X=X, v=v, kappa=kappa, Xout=[np.empty_like(x) for x in X])
    elif kind == "flow":
        X0, F = _blob_shell(c["n"])
        rng = np.random.default_rng(seed)
        X0 = X0 + _smooth(rng, X0, 0.02)  # the element data follow the shape the program loads
        f = FLOWSHELL
        dHat2 = (1e-3 * float(np.linalg.norm(X0.max(0) - X0.min(0)))) ** 2
        k, km = initialize_oipc(float(_shell_mass(X0, F, f["density"], f["thickness"]).mean()), dHat2)
        # the step is one linear solve when no contact forms: solved to FP64 accuracy
        ctx = idp.Context(h=f["h"], pcg_rel_tol=1e-12, mode=idp.MODE_FP64 if c["fp64"] else idp.MODE_MIXED)
        ctx.add_shell_instance(X0, F, f["density"], f["thickness"], dHat2, k, km)
        ctx.commit()
        s = dict(ctx=ctx, X=X0, kappa=[k, km, 0.0], Xout=np.empty_like(X0))
    elif kind == "shell":
        X0, F = _blob_shell(c["n"])
        rng = np.random.default_rng(seed)
        X = X0 + _smooth(rng, X0, 0.01)
        frame = _turned(rng, X0, 1.0)
        rows = _shell_rows(X0)
        q = SHELL
        mass = _shell_mass(frame, F, q["density"], q["thickness"])
        k, km = initialize_oipc(float(mass.mean()), q["dhat"] ** 2)
        ctx = idp.Context(h=q["h"], mode=idp.MODE_FP64 if c["fp64"] else idp.MODE_MIXED)
        ctx.add_elastic_shell_instance(X, F, q["density"], q["E"], q["nu"], q["thickness"], q["dhat"] ** 2, k, km,
                                       X0=frame, dbc_idx=rows)
        ctx.set_body_force(0, mass[:, None] * np.array([0.0, -9.8, 0.0]))
        ctx.commit()
        s = dict(ctx=ctx, X=X, v=(frame - X) / q["h"], kappa=[k, km, 0.0], targets=frame[rows],
                 Xout=np.empty_like(X))
    else:
        X0, tets, V = _plates(c["nx"], c["ny"], c["plates"])
        rng = np.random.default_rng(seed)
        ctx = idp.Context(h=H)
        p = _tet_problem(X0, tets, dHat=PLATE_DHAT)
        ctx.add_instance(X0, tets, p["mass"], p["lam"], p["mu"], p["dHat2"], p["kappa"], p["kappa_max"])
        ctx.commit()
        X, d = X0.copy(), np.zeros_like(X0)
        for k in range(c["plates"]):
            b = slice(k * V, (k + 1) * V)
            X[b, 2] = X0[b, 2] - X0[b, 2].min() + k * (PLATE_CELL + 0.6 * PLATE_DHAT)  # gaps of 0.6 d-hat
            X[b] += [rng.uniform(-0.4, 0.4) * PLATE_CELL, rng.uniform(-0.4, 0.4) * PLATE_CELL, 0.0]
            d[b] = _smooth(rng, X0[b], 0.3 * PLATE_DHAT) - [0.0, 0.0, 0.8 * PLATE_DHAT * k * rng.uniform(0.5, 1.0)]
        X += _smooth(rng, X0, 0.3 * PLATE_DHAT) + rng.uniform(-0.05, 0.05, X.shape) * PLATE_DHAT
        s = dict(ctx=ctx, X=X, d=d, records=np.zeros((24 * X.shape[0], 4), np.int32))
    s["kind"] = kind
    return s


# ---------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "energy":
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc = idp.load().idp_tet_energy_noalloc(s["T"], s["tets"].data_ptr(), s["X"].data_ptr(), s["IB"].data_ptr(),
                                               s["vol"].data_ptr(), s["lam"].data_ptr(), s["mu"].data_ptr(), H * H,
                                               s["energy"].data_ptr(), s["inverted"].data_ptr(), stream)
        if rc:
            raise idp.IDPError(rc, "idp_tet_energy_noalloc")
        return dict(energy=s["energy"], inverted=s["inverted"])
    ctx = s["ctx"]
    if kind == "batch":
        for i, (X, v, k) in enumerate(zip(s["X"], s["v"], s["kappa"])):
            ctx.set_positions(i, X)
            ctx.set_velocity(i, v)
            ctx.set_kappa(i, k)
        _, res = ctx.advance()
        for i, X in enumerate(s["Xout"]):
            ctx.state_ptr(i, X.ctypes.data)
        return dict(X=s["Xout"], kappa=np.array([r["kappa"] for r in res]), energy=np.array([r["energy"] for r in res]))
    if kind in ("step", "flow", "shell"):
        ctx.set_positions(0, s["X"])
        ctx.set_kappa(0, s["kappa"])
        if kind == "shell":
            ctx.set_velocity(0, s["v"])
            ctx.set_dbc_targets(0, s["targets"])
        elif kind == "flow":
            ctx.set_normal_flow(0, FLOWSHELL["step"])
        elif s["blob"]:
            ctx.set_normal_flow(0, FLOW)
        else:
            ctx.set_velocity(0, s["v"])
        _, res = ctx.advance()
        ctx.state_ptr(0, s["Xout"].ctypes.data)
        return dict(X=s["Xout"], kappa=res[0]["kappa"], energy=res[0]["energy"])
    if kind == "direction":
        return ctx.newton_direction(0, s["X"])[0]
    if kind == "gradient":
        return dict(energy=list(ctx.energy(0, s["X"])), gradient=ctx.gradient(0, s["X"]))
    if kind == "hessian":
        return ctx.hessian_apply(0, s["X"], s["x"])
    if kind == "contacts":
        found = ctx.constraint_set(0, s["X"])  # kept in the program's own array, one row per record
        n = min(len(found), len(s["records"]))
        s["records"][:n] = found[:n]
        s["records"][n:] = 0
        return dict(count=len(found), records=s["records"])
    return ctx.ccd_stepsize(0, s["X"], s["d"])[0]


# ---------------------------------------------------------------- work
def _counts(c):
    """Vertices, elements and surface triangles (or faces)."""
    kind = c["kind"]
    if kind in ("flow", "shell"):
        X, F = _blob_shell(c["n"])
        return X.shape[0], F.shape[0], F.shape[0]
    if kind in ("contacts", "ccd"):
        X, tets, _ = _plates(c["nx"], c["ny"], c["plates"])
        return X.shape[0], tets.shape[0], c["plates"] * 4 * (c["nx"] * c["ny"] + c["nx"] + c["ny"])
    if kind == "batch":
        b = _batch_bodies(c["count"], c["tmin"], c["tmax"])
        return sum(x[0].shape[0] for x in b), sum(x[1].shape[0] for x in b), 0
    X, tets = _body(c)
    return X.shape[0], tets.shape[0], 0


def work(case):
    c, kind = case, case["kind"]
    V, T, S = _counts(c)
    tet = 16 + 72 + 8 + 16           # ids, inverse rest basis, volume, Lame parameters
    el = 8 if c.get("fp64") else 4   # a matrix value
    B = V + 2 * 7 * V                # 3x3 blocks of the tet graph, about
    if kind == "energy":
        return dict(bytes=24 * V + tet * T, flops=90 * T)
    if kind == "gradient":
        return dict(bytes=2 * (24 * V + tet * T) + 24 * V + 8 * V, flops=(90 + 200) * T)
    if kind == "hessian":            # positions and x in, y out; the matrix is not needed in memory
        return dict(bytes=72 * V + tet * T + 8 * V, flops=2000 * T)
    if kind == "direction":          # one pass over the matrix at the least
        return dict(bytes=48 * V + tet * T + B * 9 * el, flops=(2000 + 200) * T + 18 * B)
    if kind in ("step", "batch"):    # three Newton iterations: energy, gradient, Hessian, one product
        return dict(bytes=96 * V + 3 * (2 * tet * T + B * 9 * el), flops=3 * ((2000 + 300) * T + 18 * B))
    if kind == "flow":
        return dict(bytes=96 * V + 20 * T + 7 * V * 9 * el, flops=60 * T + 18 * 7 * V)
    if kind == "shell":              # faces, and 3/2 as many hinges, of 12 and 4 vertices' worth of data
        return dict(bytes=120 * V + 3 * (76 + 48) * T + 3 * 13 * V * 9 * el, flops=3 * 9000 * T)
    return dict(bytes=(24 if kind == "contacts" else 48) * V + 12 * S + 8 * 3 * S // 2, flops=400 * S)


# ---------------------------------------------------------------- exact
class _Tet:
    """The contact-free incremental potential of a tet body in 64 bits:
    h^2 sum vol Psi(F) + |x - x_tilde|^2_M / 2, its gradient, and products
    with its element-wise PSD-projected Hessian."""

    def __init__(self, X0, tets, mass):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)  # noqa: E731
        IB, vol = _rest(X0, tets)
        self.tets, self.m = t(tets).long(), t(mass)
        IB = t(IB)
        self.Bm = torch.cat([-IB.sum(1, keepdim=True), IB], 1)  # F = sum_a x_a (x) Bm_a
        self.wv = H * H * t(vol)
        self.lam, self.mu = meshgen.lame(YOUNG, NU)

    def tensor(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def F(self, X):
        return torch.einsum("tai,taj->tij", X[self.tets], self.Bm)

    def elastic(self, X):
        F = self.F(X)
        J = torch.linalg.det(F)
        if bool((J <= 0).any()):
            return None
        lJ = J.log()
        return (self.wv * (self.mu / 2 * (F.square().sum((1, 2)) - 3) - self.mu * lJ + self.lam / 2 * lJ * lJ)).sum()

    def scatter(self, P):
        f = torch.einsum("tij,taj->tai", P, self.Bm) * self.wv[:, None, None]
        return torch.zeros(self.m.numel(), 3, dtype=torch.float64, device=self.dev).index_add_(
            0, self.tets.reshape(-1), f.reshape(-1, 3))

    def gradient(self, X, Xt):
        F = self.F(X)
        G = torch.linalg.inv(F).transpose(1, 2)
        lJ = torch.linalg.det(F).log()[:, None, None]
        return self.scatter(self.mu * (F - G) + self.lam * lJ * G) + self.m[:, None] * (X - Xt)

    def linearise(self, X):
        F = self.F(X)
        G = torch.linalg.inv(F).transpose(1, 2)
        lJ = torch.linalg.det(F).log()
        T = F.shape[0]
        A = torch.einsum("til,tkj->tijkl", G, G).reshape(T, 9, 9) * (self.mu - self.lam * lJ)[:, None, None]
        g = G.reshape(T, 9)
        A = A + self.lam * g[:, :, None] * g[:, None, :] + self.mu * torch.eye(9, dtype=A.dtype, device=self.dev)
        A = (A + A.transpose(1, 2)) / 2
        for b in range(0, T, 8192):  # batched eigen-solvers take so many at a time
            w, Q = torch.linalg.eigh(A[b:b + 8192])
            A[b:b + 8192] = torch.einsum("tpk,tk,tqk->tpq", Q, w.clamp(min=0), Q)
        self.A = A
        # diagonal of the matrix, for a Jacobi preconditioner
        d = torch.einsum("tijij->tij", self.A.reshape(T, 3, 3, 3, 3))
        D = torch.einsum("tij,taj->tai", d, self.Bm.square()) * self.wv[:, None, None]
        self.D = self.m[:, None] + torch.zeros_like(X).index_add_(0, self.tets.reshape(-1), D.reshape(-1, 3))

    def product(self, x):
        dF = self.F(x)
        return self.scatter(torch.einsum("tpq,tq->tp", self.A, dF.reshape(-1, 9)).reshape(-1, 3, 3)) + self.m[:, None] * x

    def solve(self, b, tol, most=4000):
        return _cg(self.product, b, 1.0 / self.D, tol, most)


def _cg(product, b, Minv, tol, most):
    x, r = torch.zeros_like(b), b.clone()
    z = Minv * r
    p, rz, bb = z.clone(), (r * z).sum(), (b * b).sum()
    for it in range(most):
        q = product(p)
        a = rz / (p * q).sum()
        x, r = x + a * p, r - a * q
        if it % 8 == 7 and float((r * r).sum()) <= tol * tol * float(bb):
            break
        z = Minv * r
        rn = (r * z).sum()
        p, rz = z + (rn / rz) * p, rn
    return x


def _minimise(E, X, Xt):
    """Newton from X to the minimum of the incremental potential."""
    f = lambda Y: None if (e := E.elastic(Y)) is None else float(e + 0.5 * (E.m[:, None] * (Y - Xt).square()).sum())  # noqa: E731
    e0 = f(X)
    for it in range(30):
        g = E.gradient(X, Xt)
        E.linearise(X)
        p = E.solve(-g, 1e-3 if it < 3 else 1e-8)
        a = 1.0
        while a > 1e-6 and ((e := f(X + a * p)) is None or e > e0 + 1e-14 * abs(e0)):
            a /= 2
        X = X + a * p
        e0 = f(X)
        if float(p.square().mean().sqrt()) < 1e-13:
            break
    return X, e0


def _normals(X, faces):
    """Per vertex the normalised sum of its surface triangles' normals."""
    n = np.cross(X[faces[:, 1]] - X[faces[:, 0]], X[faces[:, 2]] - X[faces[:, 0]])
    N = np.zeros_like(X)
    for k in range(3):
        np.add.at(N, faces[:, k], n)
    L = np.linalg.norm(N, axis=1, keepdims=True)
    return N / np.where(L > 0, L, 1.0)


def _surface(tets):
    faces = tets[:, [[0, 2, 1], [0, 3, 2], [0, 1, 3], [1, 2, 3]]].reshape(-1, 3)
    _, inv, n = np.unique(np.sort(faces, axis=1), axis=0, return_inverse=True, return_counts=True)
    return faces[n[inv.reshape(-1)] == 1]


def exact(case, seed):
    """Outputs of the contact-free cases in 64 bits (no contact forms at these
    inputs: the barrier term is zero and the CCD does not cut the steps)."""
    c, kind = case, case["kind"]
    if kind in ("energy", "step", "direction", "gradient", "hessian"):
        X0, tets, X, v = _tet_inputs(c, seed)
        mass = _problem_of(c)["mass"]
        E = _Tet(X0, tets, mass)
        if kind == "energy":
            X = X0 + _smooth(np.random.default_rng(seed), X0, 0.02)
            return dict(energy=E.elastic(E.tensor(X)).reshape(1), inverted=None)
        x = E.tensor(X)
        if kind == "step":
            xt = E.tensor(X + FLOW * _normals(X, _surface(tets)) if c["shape"] == "blob" else X + H * v)
            y, e = _minimise(E, x, xt)
            return dict(X=y, kappa=None, energy=e)
        if kind == "hessian":
            E.linearise(x)
            rhs = np.random.default_rng(seed + 1).normal(0.0, 1.0, X.shape)
            return E.product(E.tensor(rhs)).reshape(-1)
        # a sub-step's predictor starts from the context's own positions, the rest shape
        xt = E.tensor(X0 + H * v)
        g = E.gradient(x, xt)
        if kind == "gradient":
            inertia = 0.5 * (E.m[:, None] * (x - xt).square()).sum()
            return dict(energy=[float(E.elastic(x)), float(inertia), None], gradient=g.reshape(-1))
        E.linearise(x)
        return E.solve(-g, 1e-13).reshape(-1)
    if kind == "flow":
        X, F = _blob_shell(c["n"])
        X = X + _smooth(np.random.default_rng(seed), X, 0.02)
        f = FLOWSHELL
        area = np.linalg.norm(np.cross(X[F[:, 1]] - X[F[:, 0]], X[F[:, 2]] - X[F[:, 0]]), axis=1) / 2
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        faces, w = t(F).long(), t(f["h"] * area * f["thickness"] / 6)
        m = torch.zeros(X.shape[0], dtype=torch.float64, device=dev)
        m.index_add_(0, faces.reshape(-1), t(np.repeat(area * f["thickness"] * f["density"] / 3, 3)))
        deg = torch.zeros_like(m).index_add_(0, faces.reshape(-1), w.repeat_interleave(3)) * 2

        def product(x):
            y = x[faces]
            part = (3 * y - y.sum(1, keepdim=True)) * w[:, None, None]
            return m[:, None] * x + torch.zeros_like(x).index_add_(0, faces.reshape(-1), part.reshape(-1, 3))

        x0 = t(X)
        xt = x0 + f["step"] * t(_normals(X, F))
        p = _cg(product, m[:, None] * xt - product(x0), (1.0 / (m + deg))[:, None], 1e-14, 4000)
        y = x0 + p
        e = 0.5 * ((product(y) - m[:, None] * y) * y).sum() + 0.5 * (m[:, None] * (y - xt).square()).sum()
        return dict(X=y, kappa=None, energy=float(e))
    return None
