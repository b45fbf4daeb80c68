"""Performance cases of the engine: what a user's program has it do.

A program that uses the engine builds a model (mesh, materials, loads), gives
it a state, and then either lets the device loop advance it by some steps and
reads the fields back (``Model.run``, ``Model.state``), calls the reference's
own primitives once per step of its own loop (``GetForce``,
``StableTimeStep``), or trains the learned stress surrogate and runs it in the
loop.  The cases below do that from 1,000 to 4,000,000 elements, in both
precisions, on both element types and on the laws the configurations use.

A pass of a loop case is one segment of a simulation: the state goes in from
page-locked host arrays, the loop's start is set up (initial force and stable
step), ``steps`` central-difference steps run and the fields come back.  The
FP64 mode returns u, v and a.  The mixed mode computes element forces in FP32
and answers for the displacements, the configurations' output; they come back
as FP32 fields, which is what they are accurate to.  (Its accelerations and
velocities carry the FP32 forces' rounding, 1e-4 and more of their size, which
differs with every order of summation.)

``exact`` restates the same segment in plain torch FP64: shape-function
derivatives, F, the textbook form of each law, B^T S, lumped mass, the
central-difference update and the stable step.
"""
import functools
import math

import numpy as np
import torch

import femtech_gb300 as ft
from femtech_gb300 import meshgen as mg

RHO = 1040.0
# brain-tissue parameters of the head-like configuration (material 7 layout)
GOH = [RHO, 1.0e3, 2.19e8, 5.0e3, 10.0, 0.6, 6.0e-3, 0.1]


def listed():
    return [
        # the plain configuration: 10^3 Neo-Hookean cube in FP64, displacements every 100 steps;
        # every launch is far shorter than the chip is wide, so latency is all there is
        dict(name="cube_fp64", kind="block", mat=1, fp64=True, nx=10, ny=10, nz=10, steps=100),
        # the smallest member of the batched ensemble run by itself (a parameter study's one run)
        dict(name="block_small", kind="block", mat=6, fp64=False, nx=21, ny=17, nz=11, steps=100),
        # the accuracy sub-block of the scale configuration, both precisions: the size at which a
        # result is checked against FP64 before a long run
        dict(name="block_check_mixed", kind="block", mat=6, fp64=False, nx=40, ny=40, nz=20, steps=50),
        dict(name="block_check_fp64", kind="block", mat=6, fp64=True, nx=40, ny=40, nz=20, steps=16),
        # the scale configuration: 4.0M C3D8, one-term Ogden, mixed precision
        dict(name="block_4m", kind="block", mat=6, fp64=False, nx=200, ny=200, nz=100, steps=16),
        # a hexahedral tissue model with the reference's viscoelastic law, sizes of no power of
        # two, and a plot step (element strains) at the end
        dict(name="tissue_hex", kind="block", mat=5, fp64=False, nx=83, ny=61, nz=47, steps=16, strain=True),
        # the head-like configuration: 2M C3D4, stiff shell around a fibre-reinforced viscoelastic
        # interior, shell driven by a rigid rotation
        dict(name="head_2m", kind="head", fp64=False, tets=2_000_000, steps=32),
        # the brain drivers' loop: rigid skull from acceleration records, energy balance and
        # injury criteria every step
        dict(name="head_drivers", kind="drivers", fp64=False, tets=300_000, steps=32),
        # a batched ensemble of independent blocks, each at its own stable step
        dict(name="ensemble", kind="ensemble", instances=48, e_min=4_000, e_max=60_000, steps=20),
        # the drop-in use: the reference's own loop calls GetForce and StableTimeStep each step,
        # on a mesh of its examples' size
        dict(name="drop_in_force", kind="force", fp64=True, tets=20_000),
        # the learned surrogate in the loop of the head-like mesh
        dict(name="head_surrogate", kind="surrogate_loop", tets=200_000, steps=16),
        # its training: one epoch over samples of the plain law
        dict(name="surrogate_train", kind="surrogate_train", samples=131_072, batch=8_192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block"] * 5 + ["head", "head", "drivers", "ensemble", "force",
                                       "surrogate_loop", "surrogate_train"])
    if kind == "block":
        fp64 = rng.random() < 0.4
        mat = rng.choice([1, 2, 4, 5, 6, 6, 6, 7])
        n = _log(rng, 1_000, 60_000 if fp64 else 2_000_000)
        ax, ay = rng.uniform(0.6, 1.7), rng.uniform(0.6, 1.7)
        nz = max(3, round((n / (ax * ay)) ** (1 / 3)))
        return dict(kind=kind, mat=mat, fp64=fp64, nx=max(3, round(ax * nz)), ny=max(3, round(ay * nz)),
                    nz=nz, steps=rng.randint(9, 33), strain=rng.random() < 0.25)
    if kind == "head":
        fp64 = rng.random() < 0.25
        return dict(kind=kind, fp64=fp64, tets=_log(rng, 20_000, 200_000 if fp64 else 1_500_000),
                    steps=rng.randint(9, 33))
    if kind == "drivers":
        return dict(kind=kind, fp64=False, tets=_log(rng, 30_000, 600_000), steps=rng.randint(9, 33))
    if kind == "ensemble":
        return dict(kind=kind, instances=rng.randint(3, 64), e_min=4_000, e_max=_log(rng, 8_000, 60_000),
                    steps=rng.randint(5, 20))
    if kind == "force":
        return dict(kind=kind, fp64=rng.random() < 0.7, tets=_log(rng, 5_000, 200_000))
    if kind == "surrogate_loop":
        return dict(kind=kind, tets=_log(rng, 30_000, 400_000), steps=rng.randint(5, 17))
    return dict(kind=kind, samples=_log(rng, 40_000, 250_000), batch=rng.choice([1000, 4096, 8192, 16384]))


# ---------------- inputs ----------------
def _pinned(n):
    if torch.cuda.is_available():
        return torch.zeros(n, dtype=torch.float64, pin_memory=True)
    return torch.zeros(n, dtype=torch.float64)


def _wave(X, height, seed, strain=0.1, speed=0.5, drive=None, t=0.0):
    """Displacements and velocities of shear waves travelling up a base-fixed layer, the motion
    that the driven top face sets up: u = g(z), volume-preserving.  drive: amplitude and angular
    frequency of the top face's x motion, followed linearly."""
    rng = np.random.default_rng(seed)
    u, v = np.zeros_like(X), np.zeros_like(X)
    z = X[:, 2] / height
    for d in (0, 1):
        for k in (1, 2, 3):
            s = np.sin(np.pi * k * z)
            u[:, d] += rng.normal() * strain * height / (2 * np.pi * k) * s
            v[:, d] += rng.normal() * speed / k * s
    if drive is not None:
        a, om = drive
        u[:, 0] += a * math.sin(om * t) * z
        v[:, 0] += a * om * math.cos(om * t) * z
    return u, v


def _block(case, seed):
    nx, ny, nz, mat = case["nx"], case["ny"], case["nz"], case["mat"]
    h = 1.0e-3
    if mat == 1:  # the tension cube: soft Neo-Hookean, top face pulled
        mesh, mats, loads = mg.cube_tension_case(n=1)
        mesh = mg.hex_block(nx, ny, nz, nx * h, ny * h, nz * h, jitter=0.02, seed=seed)
        X, top = mesh["coordinates"], nz * h
        loads = mg.Loads(len(X))
        loads.fix(np.where(np.abs(X[:, 2]) < 1e-9)[0])
        loads.ramp(np.where(np.abs(X[:, 2] - top) < 1e-9)[0], 2, 0.1 * top / 0.01)
        t0 = 2.0e-3
        u, v = _wave(X, top, seed + 1, strain=0.02, speed=0.05)
        u[:, 2] += 0.1 * top / 0.01 * t0 * X[:, 2] / top
        v[:, 2] += 0.1 * top / 0.01 * X[:, 2] / top
        return mesh, mats, loads, u, v, t0
    mesh, mats, loads = mg.ogden_block_case(nx=nx, ny=ny, nz=nz, lx=nx * h, ly=ny * h, lz=nz * h, seed=seed)
    if mat == 2:
        mats = mg.materials([(2, [RHO, 2.0e4, 1.0e6])])
    elif mat == 4:
        mats = mg.materials([(4, [RHO, 1.0e3, 2.0e7, 5.0e3, 10.0])])
    elif mat == 5:
        mats = mg.materials([(5, [RHO, 1.0e3, 2.0e7, 5.0e3, 10.0, 0.5, 6.0e-3, 0.2, 4.0e-2])])
    elif mat == 7:
        mats = mg.materials([(7, [RHO, 1.0e3, 2.0e7] + GOH[3:])])
        cen = mesh["coordinates"][mesh["connectivity"].reshape(-1, 8)].mean(1)
        mesh["fiber"] = mg.smooth_fibers(cen, seed=seed + 2)
    u, v = _wave(mesh["coordinates"], nz * h, seed + 1, drive=loads.fns[1][1][:2], t=1.0e-3)
    return mesh, mats, loads, u, v, 1.0e-3


@functools.lru_cache(maxsize=4)
def _head_mesh(tets):
    """The ellipsoid, its 5 mm shell and its surface nodes (a mesh file in real use)."""
    a, b, c = 0.09, 0.07, 0.06
    h = (4.0 / 3.0 * np.pi * a * b * c * 6.0 / tets) ** (1.0 / 3.0)
    mesh = mg.tet_ellipsoid(a, b, c, h, jitter=0.1, seed=0)
    T = mesh["connectivity"].reshape(-1, 4).astype(np.int64)
    cen = mesh["coordinates"][T].mean(1)
    r = np.sqrt((cen[:, 0] / a) ** 2 + (cen[:, 1] / b) ** 2 + (cen[:, 2] / c) ** 2)
    depth = np.linalg.norm(cen, axis=1) * (1.0 / np.maximum(r, 1e-9) - 1.0)
    mesh["pid"] = np.where(depth < 5.0e-3, 0, 1).astype(np.int32)
    F = np.sort(np.concatenate([T[:, [1, 2, 3]], T[:, [0, 2, 3]], T[:, [0, 1, 3]], T[:, [0, 1, 2]]]), 1)
    n = len(mesh["coordinates"])
    key = (F[:, 0] * n + F[:, 1]) * n + F[:, 2]
    _, first, count = np.unique(key, return_index=True, return_counts=True)
    return mesh, cen, np.unique(F[first[count == 1]])


def _rotation(axis, t, peak=6.0e3, T=0.01):
    th = peak * T / np.pi * (t - T / np.pi * np.sin(np.pi * t / T))
    return axis, th, peak * T / np.pi * (1.0 - np.cos(np.pi * t / T))


def _head(case, seed):
    """The head mid-pulse: rotated with its shell, the interior lagging behind by a smooth field."""
    base, cen, surf = _head_mesh(case["tets"])
    mesh = dict(base, fiber=mg.smooth_fibers(cen, seed=seed + 1, modes=3))
    X = mesh["coordinates"]
    rng = np.random.default_rng(seed)
    axis = rng.normal(size=3)
    axis /= np.linalg.norm(axis)
    E, nu = 6.0e9, 0.3
    mats = mg.materials([(1, [2000.0, E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))]), (7, GOH)])
    loads = mg.Loads(len(X))
    loads.rotation(surf, axis, [0.0, 0.0, 0.0], 6.0e3, 0.01)
    t0 = 1.0e-3
    k, th, om = _rotation(axis, t0)
    r2 = (X[:, 0] / 0.09) ** 2 + (X[:, 1] / 0.07) ** 2 + (X[:, 2] / 0.06) ** 2
    lag = np.clip(1.0 - r2 / 0.64, 0.0, None)[:, None] ** 2  # none in the shell
    ang = th * (1.0 - 0.3 * lag)
    kx, kk = np.cross(k, X), (X @ k)[:, None] * k
    R = X * np.cos(ang) + kx * np.sin(ang) + kk * (1.0 - np.cos(ang))
    v = om * (1.0 - 0.3 * lag) * np.cross(k, R)
    return mesh, mats, loads, R - X, v, t0


def _ensemble(case):
    """The study's blocks: their sizes, aspect ratios and materials belong to the case."""
    return mg.ensemble_case(case["instances"], case["e_min"], case["e_max"], seed=case["instances"])


def _member_wave(X, loads, i, seed):
    """The state of member i; its functions are base, top x, top y and z."""
    return _wave(X, X[:, 2].max(), seed + 7 * i, strain=0.05, drive=loads.fns[3 * i + 1][1][:2], t=1.0e-3)


def _surrogate(props, seed, samples):
    from femtech_gb300.surrogate import Surrogate
    s = Surrogate(props, seed=seed)
    s.generate(samples, seed=seed + 1)
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "surrogate_train":
        s = _surrogate(GOH, seed, case["samples"])
        return dict(case=case, sur=s, start=s.params)
    prec = ft.FP64 if case.get("fp64") else ft.MIXED
    if kind == "ensemble":
        mesh, mats, loads, off = _ensemble(case)
        u = np.zeros_like(mesh["coordinates"])
        v = np.zeros_like(u)
        for i in range(len(off) - 1):
            X = mesh["coordinates"][off[i]:off[i + 1]]
            u[off[i]:off[i + 1]], v[off[i]:off[i + 1]] = _member_wave(X, loads, i, seed)
        n = len(off) - 1
        inst = dict(node_offset=off, tmax=np.full(n, 1.0), reduction=np.full(n, 0.9))
        m = ft.Model(mesh, mats, precision=prec, loads=loads, instances=inst)
        t0 = 1.0e-3
    elif kind == "block":
        mesh, mats, loads, u, v, t0 = _block(case, seed)
        m = ft.Model(mesh, mats, precision=prec, loads=loads)
    else:
        mesh, mats, loads, u, v, t0 = _head(case, seed)
        if kind == "drivers":  # rigid skull, from rest at the start of the records
            mats = mg.materials([(0, [2000.0, 2.3e9, 3.5e9]), (7, GOH)])
            loads = mg.Loads(len(mesh["coordinates"]))
            loads.rigid(mg.rigid_nodes(mesh, mats))
            u, v, t0 = np.zeros_like(u), np.zeros_like(u), 0.0
            # a head that already moves: interior waves
            free = np.ones(len(u), bool)
            free[mg.rigid_nodes(mesh, mats)] = False
            w, x = _wave(mesh["coordinates"], 0.06, seed + 5, strain=0.05, speed=1.0)
            u[free], v[free] = w[free] * 0.1, x[free]
        m = ft.Model(mesh, mats, precision=prec, loads=loads)
    st = dict(case=case, model=m, t0=t0)
    if kind == "force":
        rng = np.random.default_rng(seed + 9)
        st["u"] = u.ravel() + rng.normal(0.0, 1.0e-6, u.size)
        st["dt"] = 1.0e-7
        return st
    if kind == "drivers":
        m.set_rigid_body(mg.pulse_records(seed=seed + 3))
        m.set_energy(True)
        m.set_injury(np.where(mesh["pid"] == 1)[0])
    if kind == "surrogate_loop":
        s = _surrogate(GOH, seed, 262_144)
        s.train(epochs=1, batch=8192)
        m.set_surrogate(s)
        st["sur"] = s
    n3 = u.size
    for k, x in (("u0", u), ("v0", v)):
        st["_" + k] = _pinned(n3)
        st["_" + k].numpy()[:] = x.ravel()
        st[k] = st["_" + k].numpy()
    keys = "uva" if case.get("fp64") else "u"
    st["pin"] = {k: _pinned(n3) for k in keys}
    st["out"] = {k: p.numpy() for k, p in st["pin"].items()}
    if not case.get("fp64"):
        st["f32"] = {k: torch.zeros(n3, dtype=torch.float32) for k in keys}
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "surrogate_train":
        s = st["sur"]
        s.params = st["start"]
        loss = s.train(epochs=1, batch=case["batch"])
        return dict(params=s.params, loss=np.float32(loss))
    m = st["model"]
    if kind == "force":
        return dict(fi=_typed(case, m.GetForce(st["u"], st["dt"])), dt=_typed(case, m.StableTimeStep(st["u"])))
    m.set_state(st["u0"], st["v0"], None, st["t0"])
    m.init_explicit(0.9, 0.0, 1.0)
    m.run(case["steps"])
    s = m.state(out=st["out"])
    if case.get("fp64"):
        res = {k: st["pin"][k] for k in "uva"}
    else:
        res = {"u": st["f32"]["u"].copy_(st["pin"]["u"])}
    res["dt"] = _typed(case, s["dt"])
    if case.get("strain"):
        E, hi, lo, sh = m.element_strain()
        res.update(E=_typed(case, E), ps_max=_typed(case, hi), ps_min=_typed(case, lo), shear=_typed(case, sh))
    if kind == "drivers":
        rec = m.injury()
        # the strain criteria (rates are differences of FP32 strains over one step: rounding)
        res["mps"] = _typed(case, rec["ps"])
        res["csdm"] = rec["flags"] & (ft.INJ_MPS15 | ft.INJ_MPS30)
        res["record"] = _typed(case, np.array([rec[k] for k in ("max_strain", "min_strain", "max_shear", "mps95")]))
        e = m.energy()
        res["energy"] = _typed(case, np.array([e["internal_work"], e["external_work"], e["kinetic"]]))
    return res


def _typed(case, x):
    """Host results in the precision that the model computes them in."""
    return x if case.get("fp64") else np.asarray(x, np.float32)


# ---------------- work ----------------
def _sizes(case):
    """(elements, nodes, corners per element) of a case."""
    if case["kind"] == "block":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        return nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1), 8
    if case["kind"] == "ensemble":
        lo, hi = case["e_min"], case["e_max"]
        e = case["instances"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
        return e, 1.1 * e, 8
    return case["tets"], 0.176 * case["tets"], 4


#: floating-point operations of one element's force and stable step: kinematics and B^T S of a
#: Gauss point, each law, the element's characteristic length
_FLOPS = {8: (8, 300, 700), 4: (1, 200, 150)}
_LAW = {0: 0, 1: 120, 2: 40, 4: 230, 5: 300, 6: 300, 7: 330}


def work(case):
    kind = case["kind"]
    if kind == "surrogate_train":
        n = case["samples"] // case["batch"] * case["batch"]
        macs = 16 * 128 + 2 * 128 * 128 + 128 * 8
        # forward, dW, and dX of every layer but the first; features and targets read once
        return dict(bytes=n * (32 + 32) + 2 * 4 * 36_232, flops=2 * n * (3 * macs - 16 * 128))
    e, n, nc = _sizes(case)
    word = 8 if case.get("fp64") else 4
    gp, kin, rest = _FLOPS[nc]
    mat = case.get("mat", 6 if kind == "ensemble" else 7)
    flops = e * (gp * (kin + _LAW[mat]) + rest)
    hist = {5: 18, 7: 12}.get(mat, 0) * gp * word
    # a step: connectivity, reference coordinates, history read and written, u and v_half read and
    # written in FP64, mass
    step = e * (4 * nc + 2 * hist) + n * (3 * word + 96 + 8)
    if kind == "force":
        return dict(bytes=step + 48 * n, flops=2 * flops)
    if kind == "surrogate_loop":
        flops += e * 2 * (16 * 128 + 2 * 128 * 128 + 128 * 8)
    k = case["steps"]
    # a mesh that stays on the chip is read once for all steps, a larger one at each step
    return dict(bytes=(step if step < 100e6 else k * step) + 96 * n, flops=k * flops)


# ---------------- the same segments in plain FP64 ----------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _mm(A, B):
    """A B of two batches of small matrices."""
    return sum(A[:, :, k, None] * B[:, None, k, :] for k in range(A.shape[2]))


def _det(A):
    return (A[:, 0] * torch.linalg.cross(A[:, 1], A[:, 2])).sum(1)


def _inv(A):
    c = [torch.linalg.cross(A[:, (i + 1) % 3], A[:, (i + 2) % 3]) for i in range(3)]
    return torch.stack(c, 2) / _det(A)[:, None, None]


def _tr(A):
    return A.diagonal(dim1=1, dim2=2).sum(1)[:, None, None]


class _Exact:
    """One instance: mesh, laws and loads as FP64 tensors, and the driver's loop."""

    def __init__(self, mesh, mats, loads):
        d = _dev()
        self.X = torch.as_tensor(np.asarray(mesh["coordinates"]).reshape(-1, 3), device=d)
        nc = int(mesh["eptr"][1])
        self.nc = nc
        self.conn = torch.as_tensor(np.asarray(mesh["connectivity"]).reshape(-1, nc).astype(np.int64), device=d)
        pid = torch.as_tensor(np.asarray(mesh["pid"]).astype(np.int64), device=d)
        self.prop = torch.as_tensor(np.asarray(mats["properties"]).reshape(-1, 9), device=d)
        self.groups = [(int(mt), self.prop[p], torch.nonzero(pid == p).ravel())
                       for p, mt in enumerate(mats["materialID"]) if bool((pid == p).any())]
        self.fib = None if mesh.get("fiber") is None else torch.as_tensor(mesh["fiber"], device=d)
        if nc == 8:
            s = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                              [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=torch.float64, device=d)
            q = 0.577350269189626 * torch.tensor([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)],
                                                 dtype=torch.float64, device=d)
            one = 1.0 + q[:, None, :] * s[None]  # [gp, corner, direction]
            self.N = one.prod(-1) / 8
            self.dN = torch.stack([s[:, 0] * one[..., 1] * one[..., 2], s[:, 1] * one[..., 0] * one[..., 2],
                                   s[:, 2] * one[..., 0] * one[..., 1]], -1) / 8
            self.w = 1.0
        else:
            self.N = torch.full((1, 4), 0.25, dtype=torch.float64, device=d)
            self.dN = torch.tensor([[[1, 0, 0], [0, 1, 0], [0, 0, 1], [-1, -1, -1]]], dtype=torch.float64, device=d)
            self.w = 1.0 / 6.0
        self.hist = {}
        x = self.X[self.conn]
        self.grad, self.wj = [], []
        m = torch.zeros(len(self.X), dtype=torch.float64, device=d)
        rho = self.prop[pid, 0]
        for g in range(len(self.N)):
            Jm = torch.einsum("eai,aj->eij", x, self.dN[g])
            self.grad.append(torch.einsum("aj,ejk->eak", self.dN[g], _inv(Jm)))
            self.wj.append(self.w * _det(Jm).abs())
            for a in range(nc):
                m.index_add_(0, self.conn[:, a], rho * self.wj[g] * self.N[g, a])
        self.m = m[:, None]
        mu, lam = self.prop[pid, 1], self.prop[pid, 2]
        nu = 0.5 * lam / (lam + mu)
        self.c = torch.sqrt(lam * (1.0 / nu - 1.0) / rho)
        self.fn = None if loads is None else torch.as_tensor(np.asarray(loads.dof_fn).reshape(-1, 3), device=d)
        self.fns = [] if loads is None else loads.fns
        self.free = torch.ones_like(self.X, dtype=torch.bool) if self.fn is None else self.fn == mg.BC_FREE
        self.act = self.free.any(1)[self.conn].any(1)

    def stress(self, key, mat, p, at, F, dt):
        I = torch.eye(3, dtype=torch.float64, device=F.device)
        J = _det(F)[:, None, None]
        C = _mm(F.mT, F)
        if mat == 0:
            return torch.zeros_like(F)
        if mat == 2:
            E = (C - I) / 2
            return 2 * p[1] * E + p[2] * _tr(E) * I
        Ci = _inv(C)
        if mat == 1:
            return p[1] * (I - Ci) + p[2] * torch.log(J) * Ci
        vol = 0.5 * (p[2] + 2 * p[1] / 3) * (J * J - 1) * Ci
        if mat == 6:
            al = float(p[3])
            A = _power(C - I, al / 2 - 1)  # C^(al/2 - 1)
            tr = _tr(_mm(A, C))
            return 2 * p[1] / al * J ** (-al / 3) * (A - tr / 3 * Ci) + vol
        j = J ** (-2.0 / 3.0)
        kap = float(p[7]) if mat == 7 else 1.0 / 3.0
        B = _mm(F, F.mT)
        Ea = kap * (j * _tr(B) - 3)
        if mat == 7:
            a0 = self.fib[at]
            a = _mm(F, a0.repeat(len(F) // len(a0), 1)[:, :, None])
            aa = (a * a).sum(1, keepdim=True)
            Ea = Ea + (1 - 3 * kap) * (j * aa - 1)
        dW = torch.where(Ea > 0, p[3] * Ea * torch.exp(p[4] * Ea * Ea), torch.zeros_like(Ea))
        W = (p[1] + 2 * dW * kap) * j * (B - _tr(B) / 3 * I)
        if mat == 7:
            W = W + 2 * dW * (1 - 3 * kap) * j * (a * a.mT - aa / 3 * I)
        Fi = _inv(F)
        iso = _mm(_mm(Fi, W), Fi.mT)
        S = iso + vol
        terms = {5: ((5, 6), (7, 8)), 7: ((5, 6),)}.get(mat, ())
        if terms:
            old, H = self.hist.get(key, (torch.zeros_like(iso), [torch.zeros_like(iso) for _ in terms]))
            new = []
            for (kg, kt), h in zip(terms, H):
                r = dt / float(p[kt])
                h = math.exp(-r) * h + float(p[kg]) * -math.expm1(-r) / r * (iso - old)
                new.append(h)
                S = S + h
            self.hist[key] = (iso, new)
        return S

    def force(self, u, dt):
        f = torch.zeros_like(u)
        x = (self.X + u)[self.conn]
        G, E = len(self.N), len(self.conn)
        # the Gauss points of a small mesh together, those of a large one each for itself
        for gs in [range(G)] if G * E <= 4_000_000 else [[g] for g in range(G)]:
            F = torch.cat([_mm(x.mT, self.grad[g]) for g in gs])
            P = torch.empty_like(F)
            for mat, p, at in self.groups:
                if len(self.groups) == 1:
                    P = _mm(F, self.stress((gs[0], mat), mat, p, slice(None), F, dt))
                else:
                    P[at] = _mm(F[at], self.stress((gs[0], mat), mat, p, at, F[at], dt))
            for k, g in enumerate(gs):
                fe = self.wj[g][:, None, None] * _mm(self.grad[g], P[k * E:(k + 1) * E].mT)
                for a in range(self.nc):
                    f.index_add_(0, self.conn[:, a], fe[:, a])
        return f

    def strain(self, u):
        x = (self.X + u)[self.conn]
        E = 0
        for g in range(len(self.N)):
            F = _mm(x.mT, self.grad[g])
            E = E + (_mm(F.mT, F) - torch.eye(3, dtype=torch.float64, device=F.device)) / (2 * len(self.N))
        w = torch.linalg.eigvalsh(E.cpu())
        hi, lo = w[:, 2], w[:, 0]
        return E.mT.reshape(-1, 9), hi.clamp(min=0), lo.clamp(max=0), (hi - lo) / 2

    def stable(self, u):
        x = (self.X + u)[self.conn]
        if self.nc == 4:
            v6 = _det(torch.stack([x[:, k] - x[:, 3] for k in range(3)], 1)).abs()
            n = [torch.linalg.cross(x[:, b] - x[:, a], x[:, c] - x[:, a]).norm(dim=1)
                 for a, b, c in ((1, 2, 3), (2, 3, 0), (3, 0, 1), (0, 1, 2))]
            l = v6 / torch.stack(n).amax(0)
        else:
            vol = sum(_det(torch.einsum("eai,aj->eij", x, self.dN[g])) for g in range(8))
            area = torch.zeros_like(vol)
            t = 1.0 / math.sqrt(3.0)
            for i, j, k, n in ((0, 1, 2, 3), (4, 5, 6, 7), (0, 3, 7, 4), (1, 2, 6, 5), (0, 1, 5, 4), (3, 2, 6, 7)):
                p, q, r, s = x[:, i], x[:, j], x[:, k], x[:, n]
                cD, c1, c2 = (p - q + r - s) / 4, (-p + q + r - s) / 4, (-p - q + r + s) / 4
                flat = (cD < 1e-6).all(1)
                quad = sum(torch.linalg.cross(c1 + b * cD, c2 + a * cD).norm(dim=1) for a in (-t, t) for b in (-t, t))
                area = torch.maximum(area, torch.where(flat, 4 * torch.linalg.cross(c1, c2).norm(dim=1), quad))
            l = vol / area
        return float((l / self.c)[self.act].min())

    def bounds(self, t, u, v, a):
        for i, (kind, p) in enumerate(self.fns):
            at = self.fn == i
            if kind == mg.BCK_ROT:
                n = at.any(1)
                k = torch.tensor(p[:3], dtype=torch.float64, device=u.device)
                _, th, om = _rotation(k, t, p[6], p[7])
                r = self.X[n]
                R = r * math.cos(th) + torch.linalg.cross(k.expand_as(r), r) * math.sin(th) + \
                    (r @ k)[:, None] * k * (1 - math.cos(th))
                u[n], v[n], a[n] = R - r, om * torch.linalg.cross(k.expand_as(R), R), 0.0
                continue
            if kind == mg.BCK_FIXED:
                x, y = p[0], 0.0
            elif kind == mg.BCK_RAMP:
                x, y = p[0] * t, p[0]
            else:
                x, y = p[0] * math.sin(p[1] * t), p[0] * p[1] * math.cos(p[1] * t)
            u[at], v[at], a[at] = x, y, 0.0

    def loop(self, u, v, t, steps):
        u, v = (torch.as_tensor(x.reshape(-1, 3), device=self.X.device).clone() for x in (u, v))
        a = torch.zeros_like(u)
        self.bounds(t, u, v, a)
        dt = 0.9 * self.stable(u)
        a = torch.where(self.free, -self.force(u, dt) / self.m, a)
        for _ in range(steps):
            t1 = t + dt
            th = 0.5 * (t + t1)
            vh = v + (th - t) * a
            u = torch.where(self.free, u + dt * vh, u)
            self.bounds(t1, u, v, a)
            a = torch.where(self.free, -self.force(u, dt) / self.m, a)
            v = torch.where(self.free, vh + (t1 - th) * a, v)
            t, dt = t1, 0.9 * self.stable(u)
        return u, v, a, dt


def _power(M, q, terms=50):
    """(I + M)^q for symmetric 3x3 M of norm well below 1: the binomial series, with every power
    of M written on I, M and M^2 by Cayley-Hamilton."""
    M2 = _mm(M, M)
    i1, t2 = _tr(M).ravel(), _tr(M2).ravel()
    i2 = (i1 * i1 - t2) / 2
    i3 = _det(M)
    a, b, c = torch.zeros_like(i1), torch.ones_like(i1), torch.zeros_like(i1)
    s = [torch.ones_like(i1), torch.zeros_like(i1), torch.zeros_like(i1)]
    co = 1.0
    for k in range(1, terms + 1):
        co *= (q - k + 1) / k
        for x, y in zip(s, (a, b, c)):
            x.add_(y, alpha=co)
        a, b, c = c * i3, a - c * i2, b + c * i1
    I = torch.eye(3, dtype=M.dtype, device=M.device)
    return s[0][:, None, None] * I + s[1][:, None, None] * M + s[2][:, None, None] * M2


def exact(case, seed):
    kind = case["kind"]
    if kind in ("drivers", "surrogate_loop", "surrogate_train"):
        return None  # a network in BF16, or a sampled rigid-body integrator with criteria
    if kind == "ensemble":
        mesh, mats, loads, off = _ensemble(case)
        if len(mesh["pid"]) * case["steps"] > 40_000_000:
            return None
        conn, props = mesh["connectivity"].reshape(-1, 8), mats["properties"].reshape(-1, 9)
        us, dt0 = [], None
        for i in range(len(off) - 1):
            X, at = mesh["coordinates"][off[i]:off[i + 1]], mesh["pid"] == i
            part = dict(coordinates=X, eptr=np.array([0, 8]), connectivity=conn[at] - off[i],
                        pid=np.zeros(int(at.sum()), np.int32))
            own = mg.Loads(len(X))
            own.dof_fn, own.fns = loads.dof_fn[3 * off[i]:3 * off[i + 1]], loads.fns
            e = _Exact(part, dict(materialID=[6], properties=props[i]), own)
            u, v = _member_wave(X, loads, i, seed)
            u, _, _, dt = e.loop(u, v, 1.0e-3, case["steps"])
            us.append(u)
            dt0 = dt if dt0 is None else dt0
        return dict(u=torch.cat(us).ravel().cpu(), dt=dt0)
    mesh, mats, loads, u, v, t0 = _block(case, seed) if kind == "block" else _head(case, seed)
    if len(mesh["pid"]) * case.get("steps", 1) * (8 if kind == "block" else 1) > 550_000_000:
        return None
    e = _Exact(mesh, mats, loads)
    if kind == "force":
        rng = np.random.default_rng(seed + 9)
        w = torch.as_tensor(u.ravel() + rng.normal(0.0, 1.0e-6, u.size), device=e.X.device).reshape(-1, 3)
        return dict(fi=e.force(w, 1.0e-7).ravel().cpu(), dt=e.stable(w))
    u, v, a, dt = e.loop(u, v, t0, case["steps"])
    res = dict(u=u.ravel().cpu(), dt=dt)
    if case.get("fp64"):
        res.update(v=v.ravel().cpu(), a=a.ravel().cpu())
    if case.get("strain"):
        E, hi, lo, sh = e.strain(u)
        res.update(E=E.cpu(), ps_max=hi, ps_min=lo, shear=sh)
    return res
