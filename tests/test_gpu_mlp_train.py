"""The persistent training kernel (k_train) at widths where its tiling has
edges, and the graph path deeper networks take: one Adam step on 256 rows
against the gradients of grad() on the same rows.

The first Adam step from zero moments is lr * g / (|g| + 1e-8).  The two
gradients sum the same 256 products per weight in another row order: FP32
accumulation differs by at most 256 * 2^-24 of the sum of magnitudes, taken
here as eps = 2e-5 * max|g| of the layer (16 times a typical case), so the
step differs by at most lr * min(2, 2 eps / (|g| + 1e-8)), plus the rounding
of the weight itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LR = 1e-3


@pytest.mark.parametrize("dims", [
    [32, 256, 256, 256, 59],          # the surrogate
    [1, 2], [16, 16], [5, 17, 3],     # one layer, padded widths
    [40, 129, 31], [256, 128, 130, 2], [33, 64, 256],
    [256, 256, 256, 256, 256, 256, 10],   # more weight tiles than SMs: the graph
])
def test_first_step_matches_gradients(built, dims):
    rng = np.random.default_rng(sum(dims))
    x = rng.uniform(-1, 1, (256, dims[0])).astype(np.float32)
    t = rng.uniform(0, 1, (256, dims[-1])).astype(np.float32)
    t[:, -1] = t[:, -1] > 0.5
    net = built.Mlp(dims, seed=4)
    try:
        p0 = net.get_params()
        g, loss = net.grad(x, t)
        losses, _ = net.train(x, t, epochs=1, lr=LR, seed=2)
        p1 = net.get_params()
        y = net.forward(x)  # the refreshed BF16 copies
    finally:
        net.close()
    assert abs(losses[0] - loss) <= 1e-5 * abs(loss)
    assert np.all(np.isfinite(y))
    o = 0
    for a, b in zip(dims[:-1], dims[1:]):
        for n in (a * b, b):
            gl, w0, w1 = g[o:o + n].astype(np.float64), p0[o:o + n].astype(np.float64), p1[o:o + n]
            eps = 2e-5 * np.abs(gl).max()
            want = w0 - LR * gl / (np.abs(gl) + 1e-8)
            tol = LR * np.minimum(2.0, 2 * eps / (np.abs(gl) + 1e-8)) + 2.0 ** -22 * np.abs(w0) + 1e-9
            bad = np.abs(w1 - want) > tol
            assert not bad.any(), (dims, n, np.abs(w1 - want)[bad][:4], tol[bad][:4])
            o += n


def test_rounds_of_different_size_reuse_buffers(built):
    # a second, smaller call and a larger one on the same network equal fresh
    # networks given the same sequence
    rng = np.random.default_rng(9)
    x = rng.uniform(-1, 1, (1500, 32)).astype(np.float32)
    t = rng.uniform(0, 1, (1500, 59)).astype(np.float32)
    t[:, -1] = t[:, -1] > 0.5
    out = []
    for _ in range(2):
        net = built.Mlp([32, 256, 256, 256, 59], seed=4)
        for k, rows in enumerate((700, 300, 1500)):
            net.train(x[:rows], t[:rows], epochs=3, lr=LR, seed=k + 1)
        out.append(net.get_params())
        net.close()
    np.testing.assert_array_equal(out[0], out[1])
