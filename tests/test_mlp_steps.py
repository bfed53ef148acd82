"""The surrogate's training step and forward pass at the sizes where their
tiling changes: widths and batches that are not multiples of the 16 x 8 tiles,
one row, one hidden layer, more rows than a launch takes, and networks too wide
for the forward kernel's shared memory (GPU)."""
import numpy as np
import pytest

from bnm_cuda_b200 import surrogate as S

# (inputs, hidden, hidden layers, outputs, batch)
SIZES = [(19, 256, 4, 4, 64), (3, 33, 1, 1, 1), (16, 16, 1, 16, 16), (17, 40, 2, 5, 17), (19, 200, 3, 4, 100),
         (1, 8, 2, 2, 250), (33, 500, 2, 9, 31)]


def _adam_first_step(w, g, lr):
    """The first Adam step from w in FP32, every operation rounded to nearest (the moments start at zero)."""
    f = np.float32
    b1, b2, eps = f(0.9), f(0.999), f(1e-8)
    m, v = (f(1) - b1) * g, (f(1) - b2) * g * g
    return w - f(lr) * (m / (f(1) - b1)) / (np.sqrt(v / (f(1) - b2)) + eps)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", SIZES)
def test_step_matches_oracle_and_adam(sizes):
    from oracle import mlp_oracle

    n_in, hidden, layers, out, batch = sizes
    rng = np.random.default_rng(sum(sizes))
    m = S.MLP(n_in, out, hidden=hidden, layers=layers, max_batch=batch, seed=3)
    flat = m.get_params()
    X = rng.standard_normal((batch, n_in)).astype(np.float32)
    T = rng.standard_normal((batch, out)).astype(np.float32)
    loss, g = m.loss_and_grads(X, T)
    dims = [n_in] + [hidden] * layers + [out]
    loss_ref, g_ref, _ = mlp_oracle.loss_and_grads(flat, dims, X, T)
    assert loss == pytest.approx(loss_ref, rel=1e-4)
    assert np.linalg.norm(g - g_ref) <= 1e-3 * np.linalg.norm(g_ref) + 1e-9
    # one step from here uses this gradient (one batch: the order of its rows changes sums' rounding only)
    lr = 1e-2
    losses = m.fine_tune(X, T, epochs=1, batch=batch, lr=lr, seed=0)
    assert losses[0] == pytest.approx(loss, rel=1e-5)
    got = m.get_params()
    if batch == 1:  # a single row has one order: the update is the FP32 formula, bit for bit
        np.testing.assert_array_equal(got, _adam_first_step(flat, g, lr))
    # elsewhere the step is lr times the gradient's sign where the gradient is far from rounding
    big = np.abs(g) > 1e-3 * np.abs(g).max()
    np.testing.assert_allclose((flat - got)[big], lr * np.sign(g)[big], rtol=1e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,hidden,layers,out,n", [(19, 256, 4, 4, 1), (19, 256, 4, 4, 15), (5, 24, 1, 3, 8193),
                                                      (40, 3300, 1, 2, 70)])
def test_predict_matches_forward_oracle(n_in, hidden, layers, out, n):
    from oracle import mlp_oracle

    rng = np.random.default_rng(n)
    m = S.MLP(n_in, out, hidden=hidden, layers=layers, max_batch=64, seed=1)
    X = rng.standard_normal((n, n_in)).astype(np.float32)
    y = m.predict(X)
    dims = [n_in] + [hidden] * layers + [out]
    # the oracle rounds where the device does: what is left is FP32 summation and rare BF16 rounding flips
    ref = mlp_oracle.loss_and_grads(m.get_params(), dims, X, np.zeros((n, out), np.float32))[2]
    assert np.linalg.norm(y - ref) <= 1e-3 * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,hidden,layers,out", [(19, 256, 4, 4), (3, 8, 1, 1), (17, 264, 2, 5), (33, 500, 2, 9)])
def test_predict_rows_do_not_depend_on_the_call(n_in, hidden, layers, out):
    """Large calls read the weights at their use, small ones copy them ahead: the same bits per row."""
    m = S.MLP(n_in, out, hidden=hidden, layers=layers, max_batch=64, seed=1)
    X = np.random.default_rng(hidden).standard_normal((5000, n_in)).astype(np.float32)
    y = m.predict(X)
    for n in (1, 16, 17, 333, 2368):
        np.testing.assert_array_equal(m.predict(X[:n]), y[:n])
        np.testing.assert_array_equal(m.predict(X[-n:]), y[-n:])
