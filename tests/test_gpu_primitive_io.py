"""The single primitives' arrays in and out (internal force, stable step): node
counts around one block of the transfer kernels and on both sides of the bound
between page-locked memory in place and link copies (16,384 nodes), against the
FP64 oracle; both outputs, either one alone, no displacements, and an error,
which leaves the outputs as they were.

Tolerances: FP64 1e-10 of the force's 2-norm and 1e-12 of the step, mixed 2e-4
and 5e-6, the bounds of the force tests."""
import numpy as np
import pytest

import femtech_gb300 as ft
from femtech_gb300 import meshgen as mg


@pytest.mark.gpu
@pytest.mark.parametrize("prec,ftol,dtol", [(ft.FP64, 1e-10, 1e-12), (ft.MIXED, 2e-4, 5e-6)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 7, 3), (16, 14, 0), (24, 24, 24), (25, 25, 24)])
def test_force_and_step(shape, prec, ftol, dtol):
    from oracle.oracle import Oracle
    nx, ny, nz = shape[0], shape[1], max(shape[2], 1)
    h = 1.0e-3
    mesh = mg.hex_block(nx, ny, nz, nx * h, ny * h, nz * h, jitter=0.1, seed=1)
    mats = mg.materials([(1, [1000.0, 3.4e3, 2.0e6])])
    X = mesh["coordinates"]
    rng = np.random.default_rng(2)
    u = (X @ (0.03 * rng.normal(size=(3, 3))).T).ravel()
    n = u.size
    ref = Oracle(mesh, mats).get_force(u, 0.0)
    ref_dt = Oracle(mesh, mats).stable_time_step(u, np.zeros(n, np.int32))
    m = ft.Model(mesh, mats, precision=prec)
    L = ft.lib()

    def call(uu, fi, fn):
        p = [None if x is None else x.ctypes.data for x in (fi, fn)]
        return L.ftgpu_get_force(m.h, uu, 0.0, *p)

    fi, fn = np.full(n, 7.0), np.full(n, 7.0)
    for _ in range(2):
        assert call(u, fi, fn) == 0
        assert np.linalg.norm(fi - ref) <= ftol * np.linalg.norm(ref)
        assert np.array_equal(fn, -fi)
        assert abs(m.StableTimeStep(u) - ref_dt) <= dtol * ref_dt
    only = np.full(n, 7.0)
    assert call(u, None, only) == 0 and np.array_equal(only, fn)
    assert call(u, None, None) == 0
    assert np.array_equal(m.GetForce(u), fi)
    assert not np.any(m.GetForce(np.zeros(n)))
    if nz == 1:  # turning a single layer's lower face inverts nothing
        return m.close()
    bad = u.copy()
    bad.reshape(-1, 3)[: X.shape[0] // 2] -= 2.0 * X[: X.shape[0] // 2]  # mirrored
    only[:] = 7.0
    assert call(bad, only, None) == ft.ERR_INVERTED and np.all(only == 7.0)
    m.close()
