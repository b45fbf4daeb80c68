"""Element strains of a mesh whose results exceed the direct copy (4 MB), so
that they come back through the threads' pieces: shares that are no multiple
of a piece, into pageable and page-locked arrays, and the second call on the
kept buffers.  The values are those of the small blocks that the same kernels
are tested on; here every copy has to return the same bytes."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(36, 35, 35), (57, 41, 37)])
def test_large_strain_results(shape):
    import torch

    import femtech_gb300 as ft
    from femtech_gb300 import meshgen as mg
    nx, ny, nz = shape
    mesh = mg.hex_block(nx, ny, nz, nx * 1e-3, ny * 1e-3, nz * 1e-3, jitter=0.1, seed=1)
    m = ft.Model(mesh, mg.materials([(2, [1000.0, 2.0e4, 1.0e6])]), precision=ft.FP64)
    X = mesh["coordinates"]
    u = 1e-2 * np.sin(X * 300.0) * 1e-3
    m.set_state(u=u.ravel())
    a = m.element_strain()
    nE = len(mesh["pid"])
    pin = [torch.zeros(k * nE, dtype=torch.float64, pin_memory=True).numpy() for k in (9, 1, 1, 1)]
    L = ft.lib()
    assert L.ftgpu_element_strain(m.h, *pin) == 0
    for x, y in zip(a, pin):
        np.testing.assert_array_equal(x.ravel(), y)
    L.ftgpu_element_strain.argtypes = [C.c_void_p] * 5
    only = np.zeros(nE)
    assert L.ftgpu_element_strain(m.h, None, None, None, only.ctypes.data) == 0
    np.testing.assert_array_equal(only, a[3])
    E = a[0].reshape(-1, 3, 3)
    np.testing.assert_array_equal(E, E.transpose(0, 2, 1))
    m.close()
