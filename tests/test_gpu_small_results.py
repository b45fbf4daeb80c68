"""Small results of several arrays (element_strain, injury) cost one trip from the
device: asking for all of them takes hardly longer than for one.  Medians over 60
calls in turn; a copy per array took 1.3 times as long and more, 1.2 lies between.
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


def strain(m, E, want):
    f = ft.lib().ftgpu_element_strain
    out = [np.full(k * E, -7.0) if w else None for k, w in zip((9, 1, 1, 1), want)]
    f.argtypes = [C.c_void_p] * 5
    assert f(m.h, *[None if x is None else x.ctypes.data for x in out]) == 0
    return out


def injury(m, E, want):
    f = ft.lib().ftgpu_get_injury
    f.argtypes = [C.c_void_p] * 4
    rec = ft.Injury() if want[0] else None
    out = [np.full(E, -7, np.int32) if want[1] else None, np.full(E, -7.0) if want[2] else None]
    assert f(m.h, None if rec is None else C.byref(rec), *[None if x is None else x.ctypes.data for x in out]) == 0
    return [None if rec is None else np.frombuffer(bytes(rec), np.uint8)] + out


CALLS = {"strain": (strain, 4), "injury": (injury, 3)}


@pytest.mark.gpu
@pytest.mark.parametrize("which", CALLS)
def test_all_arrays_cost_one_trip(which):
    call, parts = CALLS[which]
    m, E = model((6, 6, 6))
    times = {parts: [], 1: []}
    for _ in range(60):
        for k, t in times.items():
            want = [k == parts or i == parts - 1 for i in range(parts)]
            t0 = time.perf_counter()
            call(m, E, want)
            t.append(time.perf_counter() - t0)
    m.close()
    assert np.median(times[parts]) <= 1.2 * np.median(times[1])


@pytest.mark.gpu
@pytest.mark.parametrize("which,n", [("strain", (3, 2, 2)), ("strain", (18, 17, 17)), ("strain", (18, 18, 17)),
                                     ("injury", (3, 2, 2)), ("injury", (35, 35, 34)), ("injury", (36, 35, 35))])
def test_any_choice_of_arrays(which, n):
    call, parts = CALLS[which]
    m, E = model(n)
    full = call(m, E, [True] * parts)
    assert all((x != -7).any() for x in full)
    for mask in range(2 ** parts - 1):
        want = [bool(mask >> i & 1) for i in range(parts)]
        for w, x, y in zip(want, call(m, E, want), full):
            assert (x is None) == (not w)
            if w:
                np.testing.assert_array_equal(x, y)
    m.close()
