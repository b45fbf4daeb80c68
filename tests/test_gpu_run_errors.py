"""A run whose error shows up in the first of several graphs ends with that graph:
the steps taken, the clocks and the fields are those of its 16th step, although
further graphs may already be queued behind it.  An inverted element, and a step
below FailureTimeStep in one instance of two (the other has nothing to do with
it and runs to the same 16th step).  And a run that is past its end."""
import time

import numpy as np
import pytest

import femtech_gb300 as ft
from femtech_gb300 import meshgen as mg

H = 1.0e-3
LAW = mg.materials([(2, [1000.0, 2.0e4, 1.0e6])])


def block(n=4):
    return mg.hex_block(n, n, n, n * H, n * H, n * H, jitter=0.05, seed=2)


def pressed(mesh, per_step, dt, nodes=None):
    """Base held, top pressed down by per_step edges a step of dt."""
    X = mesh["coordinates"]
    top = X[:, 2].max()
    loads = mg.Loads(len(X))
    loads.fix(np.where(np.abs(X[:, 2]) < 1e-9)[0])
    on = np.abs(X[:, 2] - top) < 1e-9
    if nodes is not None:
        on &= nodes
    loads.ramp(np.where(on)[0], 2, -per_step * H / dt)
    return loads


def stable(mesh, prec):
    m = ft.Model(mesh, LAW, precision=prec)
    dt = m.StableTimeStep(np.zeros(mesh["coordinates"].size))
    m.close()
    return dt


@pytest.mark.gpu
@pytest.mark.parametrize("criteria", [False, True])
@pytest.mark.parametrize("prec", [ft.FP64, ft.MIXED])
def test_inversion_ends_the_run_with_its_graph(prec, criteria):
    mesh = block()
    # (1.5 edges in the first step: its top layer turns inside out at once)
    loads = pressed(mesh, 1.5, 0.9 * stable(mesh, prec))
    last = None
    for steps in (16, 64, 200):
        m = ft.Model(mesh, LAW, precision=prec, loads=loads)
        if criteria:
            m.set_energy(True)
            m.set_injury(np.arange(64, dtype=np.int32))
        m.set_state(time=0.0)
        m.init_explicit(0.9, 0.0, 1.0e9)
        with pytest.raises(ft.FtgpuError) as e:
            m.run(steps)
        assert e.value.status == ft.ERR_INVERTED
        c = m.instance_clocks()
        assert c["step"][0] == 16
        if steps > 16:  # (a run of 16 steps ends there by its limit)
            assert c["done"][0] == 0
            now = [m.state()["u"], c["time"], c["dt"]]
            if criteria:
                now += [m.injury()["ps"], m.injury()["steps"], list(m.energy().values())]
                assert m.injury()["steps"] == 16
            for x, y in zip(last or now, now):
                np.testing.assert_array_equal(x, y)
            last = now
        m.close()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [ft.FP64, ft.MIXED])
def test_failed_step_of_one_instance_ends_the_run_with_its_graph(prec):
    a, b = block(), block()
    n = len(a["coordinates"])
    mesh = dict(coordinates=np.concatenate([a["coordinates"], b["coordinates"] + [1.0, 0, 0]]),
                connectivity=np.concatenate([a["connectivity"], b["connectivity"] + n]).astype(np.int32))
    E = len(a["etype"])
    mesh.update(etype=np.zeros(2 * E, np.int32), pid=np.zeros(2 * E, np.int32),
                eptr=np.arange(0, 16 * E + 1, 8, dtype=np.int32))
    dt = stable(a, prec)
    second = np.arange(2 * n) >= n
    loads = pressed(mesh, 0.05, 0.9 * dt, second)  # (below 0.8 of the start's step after a few)
    m = ft.Model(mesh, LAW, precision=prec, loads=loads,
                 instances=dict(node_offset=[0, n, 2 * n], tmax=[1.0e9, 1.0e9], reduction=[0.9, 0.9],
                                failure_dt=[0.0, 0.8 * dt]))
    m.set_state(time=0.0)
    m.init_explicit()
    with pytest.raises(ft.FtgpuError) as e:
        m.run(100)
    assert e.value.status == ft.ERR_DT
    c = m.instance_clocks()
    assert c["step"][0] == 16 and 1 <= c["step"][1] < 16
    assert c["done"][0] == 0 and c["done"][1] == 4
    m.close()


@pytest.mark.gpu
def test_a_run_past_its_end_takes_one_empty_graph():
    """Every graph of a run that is past its tMax is empty: it takes as long as a
    run of one graph's 16 steps (a second graph ahead of the first one's clocks
    took 1.6 times that; 1.3 lies between, the least of 40 each in turn)."""
    mesh = mg.hex_block(40, 40, 20, 40 * H, 40 * H, 20 * H)
    m = ft.Model(mesh, LAW)
    m.set_state(time=0.0)
    m.init_explicit(0.9, 0.0, 20.5 * 0.9 * m.StableTimeStep(np.zeros(mesh["coordinates"].size)))
    assert m.run(10 ** 6) == 21
    times = {16: [], 10 ** 6: []}
    for _ in range(40):
        for steps, t in times.items():
            t0 = time.perf_counter()
            assert m.run(steps) == 0
            t.append(time.perf_counter() - t0)
    m.close()
    assert min(times[10 ** 6]) <= 1.3 * min(times[16])
