"""The running extremes of the injury criteria where some elements' shear is NaN.

Beside a double root (a uniaxial stretch along an oblique axis) the argument of
the trigonometric roots' arc cosine rounds to either side of one; just outside,
the three roots are NaN, the element's MPS falls to zero and its shear is no
number.  Such an element must not hide another one's larger shear, wherever the
two sit in a patch.  Separate elements carry such stretches (up to 3 %, shears
up to 0.016), one carries distinct principal strains and the largest shear; for
both passes of C3D8 elements (eight lanes up to 20,000 in mixed precision, a
thread each above) and for C3D4 in both precisions.

Tolerance 1e-4: the roots' own FP32 rounding, some 1e-6 of an angle of order
one, times the ratio of a root to the shear, with room."""
import numpy as np
import pytest

import femtech_gb300 as ft
from femtech_gb300 import meshgen as mg

HEX = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]], float)
TET = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)


def separate(corners, n, h=1.0e-3):
    """n elements that share no node, on a grid of pitch 2 h; and each node's place in its element."""
    k = int(np.ceil(n ** (1 / 3)))
    at = np.stack(np.unravel_index(np.arange(n), (k, k, k)), 1) * 2.0 * h
    nc = len(corners)
    X = (at[:, None] + corners * h).reshape(-1, 3)
    mesh = dict(coordinates=X, eptr=np.arange(0, nc * n + 1, nc, dtype=np.int32),
                connectivity=np.arange(nc * n, dtype=np.int32),
                etype=np.full(n, 0 if nc == 8 else 1, np.int32), pid=np.zeros(n, np.int32))
    return mesh, np.broadcast_to(corners * h, (n, nc, 3))


@pytest.mark.gpu
@pytest.mark.parametrize("corners,n,prec", [(TET, 300, ft.MIXED), (TET, 300, ft.FP64), (HEX, 300, ft.MIXED),
                                            (HEX, 300, ft.FP64), (HEX, 20_400, ft.MIXED)])
def test_nan_shear_hides_no_other(corners, n, prec):
    mesh, local = separate(corners, n)
    m = ft.Model(mesh, mg.materials([(2, [1000.0, 2.0e4, 1.0e6])]), precision=prec)
    m.set_injury(np.arange(n, dtype=np.int32))
    stretch = np.array([0.06, -0.01, -0.05])
    green = stretch + 0.5 * stretch ** 2
    shear = 0.5 * (green.max() - green.min())
    for trial in range(24):
        rng = np.random.default_rng(trial)
        axis = rng.normal(size=(n, 3))
        axis /= np.linalg.norm(axis, axis=1, keepdims=True)
        G = rng.uniform(0.01, 0.03, n)[:, None, None] * axis[:, :, None] * axis[:, None]
        one = int(rng.integers(n))
        Q = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        G[one] = Q @ np.diag(stretch) @ Q.T
        u = np.einsum("eij,eaj->eai", G, local)
        m.set_state(u=u.ravel(), v=np.zeros(u.size))
        m.init_explicit(1.0e-6, 0.0, 1.0)  # (a step so short that the strains stay as given)
        m.run(1)
        r = m.injury()
        assert abs(r["max_shear"] - shear) <= 1e-4 * shear, trial
        assert r["max_shear_elem"] == one and r["max_strain_elem"] == one and r["min_strain_elem"] == one
    m.close()
