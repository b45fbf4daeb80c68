"""The FP64 C3D8 step bounds (hexgp_dt_bounds) where a model has more than one
part of one law: several element groups (laws with and without history), several
instances, elements left out of the minimum because all their nodes are held
(the smallest ones here), and patches of the caller's size; in the dt pass
(StableTimeStep), the initial force pass and the passes of a run.  Every group is
above the size from which the bounds are used.

The step is the FP64 evaluation's of every element that counts: 1e-12, its
rounding, as in test_fp64_step_bounds."""
import numpy as np
import pytest

import femtech_gb300 as ft
from femtech_gb300 import meshgen as mg

H = 1.0e-3
LAWS = [(1, [1000.0, 3.4e3, 2.0e6]),
        (5, [1040.0, 1.0e3, 2.0e7, 5.0e3, 10.0, 0.5, 6.0e-3, 0.2, 4.0e-2]),
        (7, [1040.0, 1.0e3, 2.0e7, 5.0e3, 10.0, 0.6, 6.0e-3, 0.1])]


def block(nx, ny, nz, seed):
    """Three parts side by side, the two lowest layers of elements thinner than the rest."""
    mesh = mg.hex_block(nx, ny, nz, nx * H, ny * H, nz * H, jitter=0.1, seed=seed)
    X = mesh["coordinates"].copy()
    cen = X[mesh["connectivity"].reshape(-1, 8)].mean(1)
    X[:, 2] -= 0.5 * np.minimum(X[:, 2], 2.0 * H)
    mesh["coordinates"] = X
    mesh["pid"] = np.minimum(cen[:, 0] / (nx * H) * 3, 2).astype(np.int32)
    mesh["fiber"] = mg.smooth_fibers(cen, seed=seed)
    return mesh


def waves(X, seed):
    rng = np.random.default_rng(seed)
    free = np.clip((X[:, 2] - X[:, 2].min()) / H - 1.5, 0.0, 1.0)[:, None]  # (at rest where held)
    return (0.03 * H * free * np.sin(X[:, [1, 2, 0]] * 700.0) + rng.normal(0.0, 0.01 * H, X.shape) * (free > 0)).ravel()


def held_base(X):
    return np.where(X[:, 2] <= X[:, 2].min() + 1.25 * H)[0]  # the thin layers' nodes


@pytest.mark.gpu
@pytest.mark.parametrize("patch", [0, 32, 128])
def test_groups_and_skipped_elements(patch):
    from oracle.oracle import Oracle
    mesh = block(27, 18, 17, 3)  # 2,754 elements of each law
    X, mats = mesh["coordinates"], mg.materials(LAWS)
    loads = mg.Loads(len(X))
    loads.fix(held_base(X))
    o = Oracle(mesh, mats)
    held = np.zeros(X.size, np.int32)
    held[(3 * held_base(X)[:, None] + np.arange(3)).ravel()] = 1
    u = waves(X, 4)
    m = ft.Model(mesh, mats, precision=ft.FP64, loads=loads, patch_size=patch)
    want = o.stable_time_step(u, held)
    assert o.stable_time_step(u, 0 * held) < 0.9 * want  # (the held elements would decide it)
    assert abs(m.StableTimeStep(u) - want) <= 1e-12 * want
    m.set_state(u, np.zeros_like(u), None, 0.0)
    m.init_explicit(0.9, 0.0, 1.0e9)
    assert abs(m.state()["dt"] - 0.9 * want) <= 1e-12 * want
    for steps in (1, 3, 16):
        m.run(steps)
        s = m.state()
        want = 0.9 * o.stable_time_step(s["u"], held)
        assert abs(s["dt"] - want) <= 1e-12 * want, steps
    m.close()


@pytest.mark.gpu
def test_instances():
    from oracle.oracle import Oracle
    parts = [block(27, 18, 17, 5), block(9, 5, 4, 6), block(30, 19, 17, 7)]
    mats = mg.materials(LAWS)
    n = np.cumsum([0] + [len(p["coordinates"]) for p in parts])
    mesh = dict(coordinates=np.concatenate([p["coordinates"] * (1 + 0.3 * i) + [i, 0, 0] for i, p in enumerate(parts)]),
                connectivity=np.concatenate([p["connectivity"] + k for p, k in zip(parts, n)]).astype(np.int32))
    for k in ("etype", "pid", "fiber"):
        mesh[k] = np.concatenate([p[k] for p in parts])
    mesh["eptr"] = np.arange(0, 8 * len(mesh["etype"]) + 1, 8, dtype=np.int32)
    oracles = [Oracle(dict(p, coordinates=mesh["coordinates"][a:b]), mats)
               for p, a, b in zip(parts, n[:-1], n[1:])]
    u = np.concatenate([waves(mesh["coordinates"][a:b] - [i, 0, 0], i) for i, (a, b) in enumerate(zip(n[:-1], n[1:]))])
    m = ft.Model(mesh, mats, precision=ft.FP64,
                 instances=dict(node_offset=n, tmax=[1.0e9] * 3, reduction=[0.9, 0.8, 0.7]))
    m.set_state(u, np.zeros_like(u), None, 0.0)
    m.init_explicit()
    for steps in (0, 2, 17):
        if steps:
            m.run(steps)
        s, c = m.state()["u"], m.instance_clocks()
        for i, (a, b) in enumerate(zip(n[:-1], n[1:])):
            want = (0.9, 0.8, 0.7)[i] * oracles[i].stable_time_step(s[3 * a:3 * b], np.zeros(3 * (b - a), np.int32))
            # (metres from the origin: the coordinates' own rounding over a thin layer's edge)
            assert abs(c["dt"][i] - want) <= (1e-12 + 8 * 2.5e-16 * (i + 0.05) / (0.5 * H)) * want, (i, steps)
    m.close()
