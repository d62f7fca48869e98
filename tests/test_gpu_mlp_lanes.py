"""The page-locked and device buffers that inference keeps between calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_of_growing_size_share_a_lane(built):
    # 14.3 to 16.8 MB a call: at most two sizes of lane (16 and 18 MB), not one
    # for each of the twelve calls (six kept: 90 MB)
    import torch
    net = built.Mlp([256, 256], seed=1)
    try:
        x = np.zeros((8192, 256), np.float32)
        net.forward(x[:16])
        free = torch.cuda.mem_get_info()[0]
        for rows in np.linspace(7000, 8192, 12).astype(int):
            net.forward(x[:rows])
        assert free - torch.cuda.mem_get_info()[0] <= 48 << 20
    finally:
        net.close()


def test_a_first_call_of_a_few_chunks_makes_one_lane(built):
    # five chunks: one lane of 18 MB, not five (a lane takes as long to make as
    # three chunks to run); later calls make more
    import torch
    net = built.Mlp([256, 256], seed=1)
    try:
        x = np.zeros((8192 * 5, 256), np.float32)
        net.grad(x[:16], x[:16])
        free = torch.cuda.mem_get_info()[0]
        net.forward(x)
        assert free - torch.cuda.mem_get_info()[0] <= 40 << 20
        for _ in range(12):
            net.forward(x)
        assert free - torch.cuda.mem_get_info()[0] >= 60 << 20
    finally:
        net.close()


def test_a_lane_that_cannot_be_made_is_done_without(built):
    # room for three or four more lanes of 4 MB where the call wants five
    import torch
    net = built.Mlp([64, 2], seed=1)
    fill = None
    try:
        x = np.random.default_rng(0).uniform(-1, 1, (8192 * 100, 64)).astype(np.float32)
        want = net.forward(x[:8192])
        free = torch.cuda.mem_get_info()[0]
        fill = torch.empty((free - (14 << 20)) // 2097152 * 2097152, dtype=torch.uint8, device="cuda")
        y = net.forward(x)
        np.testing.assert_array_equal(y[:8192], want)
        np.testing.assert_array_equal(net.forward(x[-8192:]), y[-8192:])
    finally:
        del fill
        torch.cuda.empty_cache()
        net.close()
