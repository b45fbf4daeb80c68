"""The reductions that close a step beside the step's chain (k_injury_select,
k_energy_reduce) against the timing graph, which runs them in it: with either
one and both, with one element group and two, with driven nodes and without,
over one graph (16 steps), tails and several graphs.  Exact: the same kernels
on the same inputs in the same order."""
import ctypes as C

import numpy as np
import pytest

import femtech_gb300 as ft
from femtech_gb300 import meshgen as mg


def model(prec, groups, driven, energy, injury):
    mesh = mg.hex_block(8, 7, 6, 8e-3, 7e-3, 6e-3, jitter=0.1, seed=4)
    X = mesh["coordinates"]
    parts = [(2, [1000.0, 2.0e4, 1.0e6]), (4, [1040.0, 1.0e3, 2.0e7, 5.0e3, 10.0])]
    mesh["pid"] = (np.arange(len(mesh["pid"])) % groups).astype(np.int32)
    loads = mg.Loads(len(X))
    if driven:
        loads.rotation(np.where(X[:, 2] < 1e-9)[0], [0.2, 0.5, 1.0], [0.0, 0.0, 0.0], 6e3, 0.01)
    m = ft.Model(mesh, mg.materials(parts[:groups]), precision=prec, loads=loads)
    v = 2.0 * np.sin(X[:, [1, 2, 0]] * 900.0)
    m.set_state(u=(1e-5 * np.sin(X * 700.0)).ravel(), v=v.ravel())
    if injury:
        m.set_injury(np.arange(0, len(mesh["pid"]), 3).astype(np.int32))
    m.set_energy(energy)
    m.init_explicit(0.9, 0.0, 1.0)
    return m


@pytest.mark.gpu
@pytest.mark.parametrize("energy,injury", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("groups,driven", [(1, False), (1, True), (2, True)])
@pytest.mark.parametrize("prec", [ft.FP64, ft.MIXED])
def test_beside_and_within(prec, groups, driven, energy, injury):
    def results(m):
        out = dict(m.energy()) if energy else {}
        if injury:
            out.update({"inj_" + k: x for k, x in m.injury().items()})
        return out

    a, b = model(prec, groups, driven, energy, injury), model(prec, groups, driven, energy, injury)
    L = ft.lib()
    n, x, y = C.c_int(), C.c_double(), C.c_double()
    a.run(16)
    assert L.ftgpu_run_profiled(b.h, 16, C.byref(n), C.byref(x), C.byref(y)) == 0
    ra, rb = results(a), results(b)
    for k in ra:
        np.testing.assert_array_equal(ra[k], rb[k], err_msg=k)
    # the same steps in several graphs and tails
    c = model(prec, groups, driven, energy, injury)
    c.run(16), c.run(16), c.run(7), a.run(23)
    rc, ra = results(c), results(a)
    for k in ra:
        np.testing.assert_allclose(rc[k], ra[k], rtol=1e-12 if prec == ft.FP64 else 1e-4,
                                   atol=0 if prec == ft.FP64 else 1e-6, err_msg=k)
    for m in (a, b, c):
        m.close()
