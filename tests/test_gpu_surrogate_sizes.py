"""The surrogate's kernels against the CPU oracle at the sizes where their split
changes: tiles of 4 and of 16 samples (the line lies at eight per SM), partial tiles,
runs of samples that follow their input copies, one and the most inputs, training
sets of one tile up to more tiles than SMs.  Tolerances as in test_gpu_surrogate."""
import numpy as np
import pytest

import mlp_oracle as mo
from nonstationary_mra_b200.fit import Surrogate

pytestmark = pytest.mark.gpu


def data(n, n_in):
    rng = np.random.default_rng(n + n_in)
    x = rng.standard_normal((n, n_in)).astype(np.float32)
    return x, np.sin(x[:, 0]).astype(np.float32)


@pytest.mark.parametrize("n,n_in", [(1, 19), (3, 1), (4, 64), (5, 19), (17, 64), (1184, 19), (1185, 19), (2400, 1)])
def test_input_gradient(n, n_in):
    net = Surrogate(n_in, seed=n)
    x, _ = data(n, n_in)
    y, gx = net.predict(x, with_grad=True)
    y_ref, gx_ref = mo.input_grad(net.params(), x, n_in)
    np.testing.assert_allclose(y, y_ref, rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(gx, gx_ref, rtol=1e-3, atol=1e-5 * np.abs(gx_ref).max())
    net.close()


@pytest.mark.parametrize("n,n_in", [(1, 19), (127, 1), (128, 64), (129, 19), (18944, 19), (18945, 19), (57000, 64)])
def test_values(n, n_in):
    net = Surrogate(n_in, seed=n)
    x, _ = data(n, n_in)
    y_ref, _ = mo.forward(net.params(), x, n_in)
    np.testing.assert_allclose(net.predict(x), y_ref, rtol=1e-4, atol=1e-5)
    net.close()


@pytest.mark.parametrize("n,n_in", [(1, 19), (16, 64), (17, 1), (2368, 19), (2369, 19)])
def test_parameter_gradient(n, n_in):
    net = Surrogate(n_in, seed=n)
    x, t = data(n, n_in)
    net.set_data(x, t)
    g, loss = net.grad()
    loss_ref, g_ref = mo.loss_and_grad(net.params(), x, t, n_in)
    assert abs(loss - loss_ref) <= 1e-5 * abs(loss_ref)
    assert np.linalg.norm(g - g_ref) <= 1e-4 * np.linalg.norm(g_ref)
    net.close()
