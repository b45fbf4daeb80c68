"""The eight-lane C3D8 pass (ft_hexgp.cuh) at the edges of its blocks, against
the FP64 oracle: element counts around one warp (4 elements), one block (32)
and a patch, every law, both precisions, and the Ogden law on both sides of its
series bounds.

Tolerances, on the force's 2-norm: FP64 1e-8 (the oracle forms det F - 1 and
C^-1 - I by subtraction, 1e-16 K against pressures of 1e-6 K and more, times
the corner forces' cancellation; the bound of the existing tests of the same
laws); mixed 2e-4, the bound of the force tests for FP32 element arithmetic on
FP32 displacements."""
import numpy as np
import pytest

import femtech_gb300 as ft
from femtech_gb300 import meshgen as mg

LAWS = {
    0: [1000.0, 1.0e3, 2.0e6],
    1: [1000.0, 3.4e3, 2.0e6],
    2: [1000.0, 2.0e4, 1.0e6],
    3: [1000.0, 2.0e4, 1.0e6],
    4: [1040.0, 1.0e3, 2.0e7, 5.0e3, 10.0],
    5: [1040.0, 1.0e3, 2.0e7, 5.0e3, 10.0, 0.5, 6.0e-3, 0.2, 4.0e-2],
    6: [1040.0, 1.5e3, 2.0e7, 5.0],
    7: [1040.0, 1.0e3, 2.0e7, 5.0e3, 10.0, 0.6, 6.0e-3, 0.1],
}


def case(shape, mat, strain, seed=0, alpha=None):
    nx, ny, nz = shape
    h = 1.0e-3
    mesh = mg.hex_block(nx, ny, nz, nx * h, ny * h, nz * h, jitter=0.1, seed=seed)
    props = list(LAWS[mat])
    if alpha is not None:
        props[3] = alpha
    X = mesh["coordinates"]
    rng = np.random.default_rng(seed + 1)
    G = rng.normal(size=(3, 3))
    G = strain * (G - np.eye(3) * np.trace(G) / 3) / 2
    u = X @ G.T + rng.normal(0.0, 0.02 * strain * h, X.shape)
    if mat == 7:
        mesh["fiber"] = mg.smooth_fibers(X[mesh["connectivity"].reshape(-1, 8)].mean(1), seed=seed)
    return mesh, mg.materials([(mat, props)]), u.ravel()


def check(mesh, mats, u, prec, tol):
    from oracle.oracle import Oracle
    o = Oracle(mesh, mats)
    m = ft.Model(mesh, mats, precision=prec)
    for dt in (1.0e-6, 2.0e-6):  # the second call runs on the first one's history
        ref, got = o.get_force(u, dt), m.GetForce(u, dt)
        assert np.linalg.norm(got - ref) <= tol * max(np.linalg.norm(ref), 1e-30)
    dref = o.stable_time_step(u, np.zeros(len(u), np.int32))
    dgot = m.StableTimeStep(u)
    m.close()
    assert abs(dgot - dref) <= (1e-12 if prec == ft.FP64 else 5e-6) * dref


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(ft.FP64, 1e-8), (ft.MIXED, 2e-4)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 1), (5, 1, 1), (31, 1, 1), (11, 3, 1), (13, 10, 1),
                                   (17, 11, 9)])
def test_block_edges(shape, prec, tol):
    check(*case(shape, 6, 0.05, seed=shape[0]), prec, tol)


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(ft.FP64, 1e-8), (ft.MIXED, 2e-4)])
@pytest.mark.parametrize("mat", [1, 2, 3, 4, 5, 7])
def test_laws(mat, prec, tol):
    check(*case((7, 5, 3), mat, 0.08, seed=mat), prec, tol)


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(ft.FP64, 1e-8), (ft.MIXED, 2e-4)])
@pytest.mark.parametrize("alpha", [5.0, -5.0, 8.0, 2.0])
@pytest.mark.parametrize("strain", [1e-4, 0.02, 0.06, 0.12, 0.2, 0.3])
def test_ogden_series_and_eigen(strain, alpha, prec, tol):
    """Every count of series terms and the eigen-decomposition beyond them."""
    check(*case((4, 4, 4), 6, strain, seed=3, alpha=alpha), prec, tol)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(14, 14, 13), (43, 9, 8)])
@pytest.mark.parametrize("scale,shift", [(1.0, 0.0), (1.0, 1e3), (5e3, 0.0), (1e-6, 0.0)])
@pytest.mark.parametrize("kind", ["jitter", "box", "sliver"])
def test_fp64_step_bounds(kind, scale, shift, shape):
    """Meshes large enough for the FP32 bounds in front of the FP64 stable step:
    no two elements alike, all alike (parallelogram faces, every bound equal),
    and thin ones; far from the origin, and sizes at which the bounds leave the
    twist test open (edges of 5 m) or their range (1e-9 m).  The step is that of
    the FP64 evaluation of every element: its rounding, 1e-12, plus the
    coordinates' own, 1e-16 of their size over an edge."""
    from oracle.oracle import Oracle
    mesh, mats, u = case(shape, 1, 0.05 if kind == "jitter" else 0.0, seed=5)
    h = 1.0e-3
    if kind != "jitter":
        mesh = mg.hex_block(*shape, shape[0] * h, shape[1] * h, shape[2] * h)
        u = np.zeros_like(u)
    X = mesh["coordinates"].copy()
    if kind == "sliver":
        rng = np.random.default_rng(2)
        X[:, 2] *= 1e-3
        X += rng.uniform(-1, 1, X.shape) * [0.1 * h, 0.1 * h, 1e-4 * h]
    mesh["coordinates"] = X * scale + shift
    u = u * scale
    m = ft.Model(mesh, mats, precision=ft.FP64)
    ref = Oracle(mesh, mats).stable_time_step(u, np.zeros(len(u), np.int32))
    tol = 1e-12 + 1e-16 * shift / (h * scale * (1e-3 if kind == "sliver" else 1.0)) * 8
    assert abs(m.StableTimeStep(u) - ref) <= tol * ref
    m.set_state(u, np.zeros_like(u), None, 0.0)
    m.init_explicit(1.0, 0.0, 1.0e9)
    assert abs(m.state()["dt"] - ref) <= tol * ref
    m.close()
