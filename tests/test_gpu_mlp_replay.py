"""Training over many steps, epochs and calls of different size against a host
replay: the same orders (std::shuffle of the same generator), the gradients of
grad() on each batch at the replay's parameters, and Adam in float64 with one
set of moments and one step count across the calls.  Weights of an earlier
step, an order or rows left from an earlier epoch or call, or moments that do not
carry over would show.

Tolerance, on the relative L2 difference of each tensor's total change: twice
what the replay itself changes by on the CPU when every gradient is off by
uniform noise of 2e-5 of its tensor's largest (16 times the typical FP32
summation difference), e.g. 8.4e-2 for the surrogate, where rounding of weights
and activations to BF16 flips; weights one step old change it by 1.0 there, lost
moments by 0.43."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = ((1024, 2), (300, 3), (1500, 1))  # rows, epochs
LR = 1e-2

ORDER = """
#include <algorithm>
#include <numeric>
#include <random>
extern "C" void orders(int *out, int rows, int epochs, unsigned long long seed) {
  std::mt19937_64 gen(seed);
  for (int e = 0; e < epochs; e++, out += rows) {
    std::iota(out, out + rows, 0);
    std::shuffle(out, out + rows, gen);
  }
}
"""


@pytest.fixture(scope="module")
def orders(tmp_path_factory):
    d = tmp_path_factory.mktemp("orders")
    (d / "o.cpp").write_text(ORDER)
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-o", str(d / "o.so"), str(d / "o.cpp")])
    L = ctypes.CDLL(str(d / "o.so"))

    def f(rows, epochs, seed):
        out = np.zeros((epochs, rows), np.int32)
        L.orders(out.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), rows, epochs, ctypes.c_ulonglong(seed))
        return out
    return f


@pytest.mark.parametrize("dims, tol", [
    ([32, 256, 256, 256, 59], 0.17), ([40, 129, 31], 0.01), ([5, 17, 3], 0.001),
    ([256, 256, 256, 256, 256, 256, 256, 10], 0.4),  # the captured step
])
def test_calls_equal_host_replay(built, orders, dims, tol):
    rng = np.random.default_rng(7)
    x = rng.uniform(-1, 1, (1500, dims[0])).astype(np.float32)
    t = rng.uniform(0, 1, (1500, dims[-1])).astype(np.float32)
    t[:, -1] = t[:, -1] > 0.5
    net, rep = built.Mlp(dims, seed=3), built.Mlp(dims, seed=3)
    try:
        p0 = net.get_params()
        p, m, v, s = p0.copy(), np.zeros(p0.size), np.zeros(p0.size), 0
        for c, (rows, epochs) in enumerate(CALLS):
            net.train(x[:rows], t[:rows], epochs=epochs, lr=LR, seed=c + 5)
            for o in orders(rows, epochs, c + 5):
                for k in range(rows // 256):
                    q = o[256 * k:256 * k + 256]
                    rep.set_params(p)
                    g = rep.grad(x[q], t[q])[0].astype(np.float64)
                    m, v, s = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g, s + 1
                    p = (p - LR * (m / (1 - 0.9 ** s)) / (np.sqrt(v / (1 - 0.999 ** s)) + 1e-8)).astype(np.float32)
        got, want, o = net.get_params() - p0, p - p0, 0
        y = net.forward(x)  # the BF16 copies follow the parameters
        rep.set_params(net.get_params())
        np.testing.assert_array_equal(rep.forward(x), y)
    finally:
        net.close()
        rep.close()
    for a, b in zip(dims[:-1], dims[1:]):
        for n in (a * b, b):
            d = np.linalg.norm(got[o:o + n] - want[o:o + n]) / np.linalg.norm(want[o:o + n])
            assert d <= tol, (dims, o, d)
            o += n
