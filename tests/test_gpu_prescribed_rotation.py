"""Prescribed rigid rotations in the passes outside a fused step (the boundary
values at the start of a simulation, the half-step that opens a run): DOFs of
one node on different rotation functions, more functions than the passes hold
trigonometry for (8), and blocks that hold nodes of two instances at different
times, against Rodrigues' formula.

Tolerances: those of the oracle's own closed-form test, 1e-15 for u (radii of
1e-2) and 1e-12 for v, as both sides round a handful of FP64 operations."""
import numpy as np
import pytest

import femtech_gb300 as ft
from femtech_gb300 import meshgen as mg

T0, A0, T = 0.004, 6.0e3, 0.01


def rotated(X, axis, t):
    k = axis / np.linalg.norm(axis)
    K = np.array([[0, -k[2], k[1]], [k[2], 0, -k[0]], [-k[1], k[0], 0]])
    th = A0 * T / np.pi * (t - T / np.pi * np.sin(np.pi * t / T))
    om = A0 * T / np.pi * (1 - np.cos(np.pi * t / T))
    R = np.eye(3) + np.sin(th) * K + (1 - np.cos(th)) * K @ K
    x = X @ R.T
    return x - X, om * np.cross(k, x)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [ft.FP64, ft.MIXED])
@pytest.mark.parametrize("nfn", [1, 3, 8, 9])
def test_prescribed_rotations(precision, nfn):
    parts = [mg.hex_block(3, 2, 2, 0.012, 0.01, 0.01), mg.hex_block(2, 2, 3, 0.006, 0.007, 0.01)]
    n = [len(p["coordinates"]) for p in parts]
    E = sum(len(p["etype"]) for p in parts)
    mesh = dict(coordinates=np.concatenate([p["coordinates"] for p in parts]),
                connectivity=np.concatenate([parts[0]["connectivity"],
                                             parts[1]["connectivity"] + n[0]]).astype(np.int32),
                eptr=np.arange(0, 8 * E + 1, 8, dtype=np.int32), etype=np.zeros(E, np.int32),
                pid=np.zeros(E, np.int32))
    X, N = mesh["coordinates"], n[0] + n[1]
    rng = np.random.default_rng(nfn)
    axes = rng.normal(size=(nfn, 3))
    loads = mg.Loads(N)
    for k in range(nfn):
        loads.rotation(np.arange(0), axes[k], [0.0, 0.0, 0.0], A0, T)
    fn = (np.arange(N)[:, None] * 2 + np.arange(3)) % nfn
    fn[rng.random(fn.shape) < 0.2] = -1
    loads.dof_fn = fn.ravel().astype(np.int32)
    inst = dict(node_offset=np.array([0, n[0], N], np.int32), tmax=np.array([1.0, 1.0]),
                reduction=np.array([0.9, 0.5]))
    m = ft.Model(mesh, mg.materials([(1, [1000.0, 3.4e3, 2.0e5])]), precision=precision,
                 loads=loads, instances=inst)

    def check(s, t):
        ref_u, ref_v = np.zeros((N, 3)), np.zeros((N, 3))
        for i, sl in enumerate((slice(0, n[0]), slice(n[0], N))):
            for k in range(nfn):
                u, v = rotated(X[sl], axes[k], t[i])
                on = fn[sl] == k
                ref_u[sl][on], ref_v[sl][on] = u[on], v[on]
        on = fn >= 0
        np.testing.assert_allclose(s["u"].reshape(-1, 3)[on], ref_u[on], rtol=0, atol=1e-15)
        np.testing.assert_allclose(s["v"].reshape(-1, 3)[on], ref_v[on], rtol=0, atol=1e-12)
        assert np.all(s["a"].reshape(-1, 3)[on] == 0.0)

    m.set_state(np.zeros(3 * N), np.zeros(3 * N), None, T0)
    m.init_explicit(0.9, 0.0, 1.0)
    check(m.state(), [T0, T0])
    m.run(1)
    t = m.instance_clocks()["time"]
    assert t[0] != t[1]
    check(m.state(), t)
    m.close()
