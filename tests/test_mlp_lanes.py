"""The surrogate's kernels off their usual path (GPU): training steps in which
the lanes of a warp go different ways (gradients so small that some weights of a
lane take Adam's plain expression, rows past the batch, layers whose last 32
outputs are not full); forward passes over several clusters; calls around the
size of the locked buffer."""
import numpy as np
import pytest

from bnm_cuda_b200 import surrogate as S


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,hidden,layers,out", [(19, 200, 2, 4), (5, 8, 1, 1), (37, 40, 3, 3), (16, 33, 2, 17)])
def test_small_gradients_take_the_same_formula(n_in, hidden, layers, out):
    from oracle import mlp_oracle

    rng = np.random.default_rng(hidden)
    X = rng.uniform(0.5, 1.5, (1, n_in)).astype(np.float32)
    X[0, rng.permutation(n_in)[: n_in // 2]] *= np.float32(1e-13)  # squares of these gradients are below 1e-27
    T = rng.standard_normal((1, out)).astype(np.float32)
    m = S.MLP(n_in, out, hidden=hidden, layers=layers, max_batch=16, seed=5)
    w = m.get_params()
    loss, g = m.loss_and_grads(X, T)
    dims = [n_in] + [hidden] * layers + [out]
    ref = mlp_oracle.loss_and_grads(w, dims, X, T)[1]
    first = slice(0, n_in * hidden)
    for c in range(n_in):  # small columns too: products of one BF16 value each, a rounding flip is 2^-8
        a, b = g[first].reshape(hidden, n_in)[:, c], ref[first].reshape(hidden, n_in)[:, c]
        assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b)
    losses = m.fine_tune(X, T, epochs=1, batch=1, lr=1e-2, seed=0)
    assert losses[0] == pytest.approx(loss, rel=1e-5)
    # the first step from zero moments in FP32, every operation rounded to nearest
    f = np.float32
    b1, b2 = f(0.9), f(0.999)
    mm, v = (f(1) - b1) * g, (f(1) - b2) * g * g
    want = w - f(1e-2) * (mm / (f(1) - b1)) / (np.sqrt(v / (f(1) - b2)) + f(1e-8))
    np.testing.assert_array_equal(m.get_params(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("n,max_batch", [(1, 1), (33, 1024), (300, 256), (1500, 1024)])
def test_wide_forward_does_not_depend_on_the_split(n, max_batch):
    """Networks too wide for the forward kernel's shared memory: rows in one or several clusters, odd blocks left
    over; a row's result is what it gives alone."""
    from oracle import mlp_oracle

    n_in, hidden, layers, out = 21, 3300, 2, 3
    m = S.MLP(n_in, out, hidden=hidden, layers=layers, max_batch=max_batch, seed=2)
    X = np.random.default_rng(n).standard_normal((n, n_in)).astype(np.float32)
    y = m.predict(X)
    for i in sorted({0, n // 2, n - 1}):
        np.testing.assert_array_equal(m.predict(X[i:i + 1])[0], y[i])
    some = X[:40]
    ref = mlp_oracle.loss_and_grads(m.get_params(), [n_in] + [hidden] * layers + [out], some,
                                    np.zeros((len(some), out), np.float32))[2]
    # the oracle rounds where the device does: what is left is FP32 summation and rare BF16 rounding flips
    assert np.linalg.norm(y[:40] - ref) <= 1e-3 * np.linalg.norm(ref)


@pytest.mark.gpu
def test_long_trainings_of_large_batches_stay_in_bounded_memory():
    """The rows of a launch's steps are bounded, whatever the batch: 150 steps of 65,536 rows are 37 MB of indices, of
    which 16 are on the device at once; and where a training is cut into launches does not show in its result."""
    import torch

    n, epochs = 65536, 150
    x, t = np.full((n, 2), 0.7, np.float32), np.full((n, 1), 0.3, np.float32)  # equal rows: their order does not matter
    m = [S.MLP(2, 1, hidden=8, layers=1, max_batch=n, seed=7) for _ in range(2)]
    for k in m:
        k.fine_tune(x, t, epochs=1, batch=n, lr=1e-3)  # the training set is on the device
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    once = m[0].fine_tune(x, t, epochs=epochs, batch=n, lr=1e-3)
    assert free - torch.cuda.mem_get_info()[0] <= 24 << 20
    parts = np.concatenate([m[1].fine_tune(x, t, epochs=10, batch=n, lr=1e-3) for _ in range(epochs // 10)])
    np.testing.assert_array_equal(once, parts)
    np.testing.assert_array_equal(m[0].get_params(), m[1].get_params())


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,max_batch", [(4100, 96), (4100, 32), (19, 64)])
def test_predict_around_the_locked_buffer(n_in, max_batch):
    """1 MiB of rows: more than that goes through the device's buffer where it holds more (4100 inputs: 63 rows, so 48),
    else in pieces; the buffer grows with the calls."""
    rows = (1 << 20) // (4 * (n_in + 3)) // 16 * 16
    m = S.MLP(n_in, 3, hidden=40, layers=1, max_batch=max_batch, seed=2)
    X = np.random.default_rng(n_in).standard_normal((3 * rows + 5, n_in)).astype(np.float32)
    y = m.predict(X)
    for n in (1, 17, rows - 1, rows, rows + 1, 2 * rows + 7):
        np.testing.assert_array_equal(m.predict(X[:n]), y[:n])
    ref = np.concatenate([m.predict(X[i:i + 1]) for i in (0, rows, 3 * rows + 4)])
    np.testing.assert_array_equal(y[[0, rows, 3 * rows + 4]], ref)


@pytest.mark.gpu
def test_more_layers_than_a_grid_has_rows():
    layers = 65600
    m = S.MLP(1, 1, hidden=1, layers=layers, max_batch=1, seed=0)
    w = np.tile(np.float32([1, 0]), layers + 1)  # every layer passes its input on
    w[-1] = 0.25
    m.set_params(w)
    np.testing.assert_array_equal(m.get_params(), w)
    np.testing.assert_array_equal(m.predict(np.float32([[1.5]])), np.float32([[1.75]]))
