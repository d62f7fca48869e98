"""The inference kernel (k_forward) at the edges of its row tiles and widths.

Outputs against the CPU oracle (relative L2 below 1e-2, the bar of
test_gpu_mlp.py: a BF16 rounding may flip where FP32 and float64 sums differ),
and every row equal to the same row in a call of another size: neither the
tile height (16 or 64 rows), the chunk a row falls in nor the lane that runs it
may change a bit."""
import os
import sys
import threading

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle as mo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[32, 256, 256, 256, 59], [1, 2], [17, 3], [256, 16, 130, 129, 2], [40, 129, 31],
                                  [64] + [48] * 34 + [5]])
def test_rows_and_widths(built, dims):
    rng = np.random.default_rng(len(dims) + dims[0])
    net = built.Mlp(dims, seed=3)
    try:
        x = rng.uniform(-1, 1, (20001, dims[0])).astype(np.float32)
        y = net.forward(x)  # three chunks, 64-row tiles, ragged end
        if len(dims) < 10:
            ref, _ = mo.forward(net.get_params(), dims, x[:500].astype(np.float64))
            assert np.linalg.norm(y[:500] - ref) <= 1e-2 * np.linalg.norm(ref)
        for rows in (1, 15, 16, 17, 63, 65, 2368, 2369, 8191, 8192, 8193):
            for lo in (0, 20001 - rows):
                np.testing.assert_array_equal(net.forward(x[lo:lo + rows]), y[lo:lo + rows])
        assert net.forward(x[:0]).shape == (0, dims[-1])
    finally:
        net.close()


def test_networks_on_threads_share_lanes(built):
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (30000, 32)).astype(np.float32)
    nets = [built.Mlp([32, 256, 256, 59 + k], seed=k + 1) for k in range(4)]
    want = [n.forward(x) for n in nets]
    got = [None] * 4

    def work(k):
        for _ in range(5):
            got[k] = nets[k].forward(x)

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)
    for n in nets:
        n.close()
