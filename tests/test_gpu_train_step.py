"""The tcgen05 training step (ft_train_tc.cuh) at the edges of its tiles and
slices, against the warp-level mma.sync kernels.

Both paths round the same BF16 operands and activations; FP32 sums in another
order flip a BF16 rounding (2^-9 of one activation) here and there, so the
gradient blocks agree to a few 1e-3 in the 2-norm (the bound that the
existing cross-check of the two paths uses)."""
import numpy as np
import pytest

from test_surrogate import PROPS7, mo, rand_batch, rand_params


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 128, 129, 511, 513, 769, 19_585])
def test_training_step_edges(n):
    """One row, the edges of a 128-row tile, both sides of the one-slice limit
    of 512 rows, a last slice of one row, and more tiles than SMs."""
    from femtech_gb300.surrogate import Surrogate
    s = Surrogate(PROPS7, seed=n)
    rng = np.random.default_rng(n)
    s.params = rand_params(rng).astype(np.float32)
    x, t = rand_batch(rng, n)
    out = {}
    for tc in (True, False):
        s.gemm_path(tc)
        g, loss = s.gradient(x, t)
        out[tc] = (g, loss, s.forward(x))
    s.close()
    (g1, l1, y1), (g0, l0, y0) = out[True], out[False]
    assert abs(l1 - l0) <= 1e-4 * l0 + 2e-3 * l0 / np.sqrt(n)
    assert np.abs(y1 - y0).max() <= 2e-3 * np.abs(y0).max()
    for k, (a, b) in mo.OFF.items():
        err = np.linalg.norm(g1[a:b] - g0[a:b]) / max(np.linalg.norm(g0[a:b]), 1e-30)
        assert err < 5e-3, (k, err)


def infer(s, x):
    import ctypes as C
    f = s.L.ftgpu_surrogate_infer
    f.argtypes = [C.c_void_p, C.c_longlong, C.c_void_p, C.c_void_p]
    y = np.zeros((len(x), 8), np.float32)
    assert f(s.h, len(x), x.ctypes.data, y.ctypes.data) == 0
    return y


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 128, 129, 19_456, 19_457, 77_825])
def test_inference_tiles(n):
    """The in-loop inference kernel at the edges of its tiles and of its
    distribution over SMs and slots (152 x 128 rows, four slots), against the
    training forward: 1e-2 of max |y|, the existing bound for BF16 activations
    whose roundings flip."""
    from femtech_gb300.surrogate import Surrogate
    s = Surrogate(PROPS7, seed=n)
    rng = np.random.default_rng(n)
    s.params = rand_params(rng).astype(np.float32)
    x = rand_batch(rng, n)[0].astype(np.float32)
    y = s.forward(x)
    assert np.abs(infer(s, x) - y).max() <= 1e-2 * np.abs(y).max()
    s.close()


@pytest.mark.gpu
def test_inference_follows_the_parameters():
    """The weights' images are laid out again when training or a new parameter
    vector changes them."""
    from femtech_gb300.surrogate import Surrogate
    s = Surrogate(PROPS7, seed=5)
    s.generate(20_000, seed=6)
    x = s.samples(500)[0]
    first = infer(s, x)
    s.train(epochs=1, batch=1000)
    y = s.forward(x)
    trained = infer(s, x)
    assert np.abs(trained - y).max() <= 1e-2 * np.abs(y).max()
    assert np.abs(trained - first).max() > 0
    p = s.params
    s.params = rand_params(np.random.default_rng(1)).astype(np.float32)
    assert np.abs(infer(s, x) - trained).max() > 0
    s.params = p
    np.testing.assert_array_equal(infer(s, x), trained)
    s.close()
