"""device_ms of the surrogate's calls is time the device spent on kernels: it
cannot exceed the call's wall time, however many lanes of a large inference
overlap."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_forward_of_overlapping_lanes(built):
    # narrow and deep: a chunk's kernel takes far longer than its transfers, so
    # the lanes' kernels wait for each other
    dims = [16] * 401
    dims[-1] = 4
    net = built.Mlp(dims, seed=2)
    try:
        x = np.random.default_rng(0).uniform(-1, 1, (8192 * 18, 16)).astype(np.float32)
        net.forward(x)
        for _ in range(3):
            t = time.perf_counter()
            _, ms = net.forward(x, with_time=True)
            wall = 1e3 * (time.perf_counter() - t)
            assert ms <= wall, (ms, wall)
        _, one = net.forward(x[:8192], with_time=True)
        # 18 chunks of the same work, at most two at a time on the SMs
        assert 0.5 * 18 * one <= ms <= 1.5 * 18 * one, (ms, one)
    finally:
        net.close()


def test_training_without_the_hosts_part(built):
    # a small network on many rows: drawing an epoch's order of 2,000,000 rows
    # takes the host tens of ms; the first epoch's, which nothing hides, is not
    # in device_ms, so one epoch takes what each of four more adds
    rows = 2_000_000
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (rows, 1)).astype(np.float32)
    t = np.stack([x[:, 0], x[:, 0] > 0], 1).astype(np.float32)
    net = built.Mlp([1, 2], seed=2)
    try:
        net.train(x, t, epochs=1)
        one = net.train(x, t, epochs=1)[1]
        each = (net.train(x, t, epochs=5)[1] - one) / 4
        assert abs(one - each) <= 0.03 * each + 1.0, (one, each)
    finally:
        net.close()
