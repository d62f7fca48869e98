"""The GEMM check entry with more row tiles than twice the SMs (one column tile
a row tile, which nothing else of the framework launches), a ragged last tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m, n, k", [(40001, 256, 256), (37889, 64, 48)])
def test_many_rows_equal_few(built, m, n, k):
    rng = np.random.default_rng(m)
    a = (rng.normal(0, 1, (m, k)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    b = (rng.normal(0, 1, (n, k)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    bias = rng.normal(0, 1, n).astype(np.float32)
    c = built.mlp_gemm(a, b, bias, relu=True)
    # every accumulator sums the same products in the same order
    for lo, hi in ((0, 300), (m - 257, m)):
        np.testing.assert_array_equal(built.mlp_gemm(a[lo:hi], b, bias, relu=True), c[lo:hi])
