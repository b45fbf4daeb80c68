"""Small results of several arrays (element_strain, injury) cost one trip from the
device: asking for all of them takes hardly longer than for one.  The least of 200
calls each, in turn, into arrays that are there; a copy per array took 1.4 times as
long and more, 1.2 lies between.
And the arrays are the same, whichever are asked for, on both sides of the size up
to which they come together (512 KB: some 5,400 elements' strains, 42,000 listed
elements)."""
import ctypes as C
import time

import numpy as np
import pytest

import femtech_gb300 as ft
from femtech_gb300 import meshgen as mg

H = 1.0e-3


def model(n):
    mesh = mg.hex_block(*n, *[k * H for k in n], jitter=0.1, seed=1)
    m = ft.Model(mesh, mg.materials([(2, [1000.0, 2.0e4, 1.0e6])]))
    E = len(mesh["etype"])
    m.set_injury(np.random.default_rng(0).permutation(E).astype(np.int32))
    v = 2.0 * np.sin(mesh["coordinates"][:, [1, 2, 0]] * 900.0)
    m.set_state(v=v.ravel())
    m.init_explicit(0.9, 0.0, 1.0)
    m.run(3)
    return m, E


def arrays(which, E, want):
    if which == "strain":
        return [np.full(k * E, -7.0) if w else None for k, w in zip((9, 1, 1, 1), want)]
    made = [np.zeros(C.sizeof(ft.Injury), np.uint8), np.full(E, -7, np.int32), np.full(E, -7.0)]
    return [x if w else None for x, w in zip(made, want)]


def call(which, m, out):
    L = ft.lib()
    f = L.ftgpu_element_strain if which == "strain" else L.ftgpu_get_injury
    f.argtypes = [C.c_void_p] * (1 + len(out))
    args = [None if x is None else x.ctypes.data for x in out]
    t0 = time.perf_counter()
    rc = f(m.h, *args)
    t0 = time.perf_counter() - t0
    assert rc == 0
    return t0


PARTS = {"strain": 4, "injury": 3}


@pytest.mark.gpu
@pytest.mark.parametrize("which", PARTS)
def test_all_arrays_cost_one_trip(which):
    parts = PARTS[which]
    m, E = model((6, 6, 6))
    every, one = (arrays(which, E, [k or i == parts - 1 for i in range(parts)]) for k in (True, False))
    times = [(call(which, m, every), call(which, m, one)) for _ in range(200)]
    m.close()
    least = np.min(times, 0)
    assert least[0] <= 1.2 * least[1]


@pytest.mark.gpu
@pytest.mark.parametrize("which,n", [("strain", (3, 2, 2)), ("strain", (18, 17, 17)), ("strain", (18, 18, 17)),
                                     ("injury", (3, 2, 2)), ("injury", (35, 35, 34)), ("injury", (36, 35, 35))])
def test_any_choice_of_arrays(which, n):
    parts = PARTS[which]
    m, E = model(n)
    full = arrays(which, E, [True] * parts)
    call(which, m, full)
    assert all((x != -7).any() for x in full)
    for mask in range(2 ** parts - 1):
        some = arrays(which, E, [bool(mask >> i & 1) for i in range(parts)])
        call(which, m, some)
        for x, y in zip(some, full):
            if x is not None:
                np.testing.assert_array_equal(x, y)
    m.close()
