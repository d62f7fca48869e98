"""The FP64 interval kernel (blocks of 512 threads, one post to a warp in the
pull) against the FP64 tile kernels (256 threads), bit for bit: blocks with less
than a warp of posts, with one post more than its warps, with tiles of 64 and,
past 64 posts, of 128, and a second tile; batches of 10 steps and cut ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, degree", [(9, 3), (2517, 60), (9473, 40), (19203, 30)])
def test_fp64_interval_equals_tiles(built, n, degree):
    from flysim_b200 import netgen, network
    na = network.connectome_net(netgen.connectome_fast(n=n, regions=2, mean_degree=degree, seed=9))
    runs = []
    for tiles in (False, True):
        e = built.Engine(na.desc, "fp64", chunk_steps=100, interval_kernel=not tiles, tile_kernels=tiles)
        try:
            assert e.layout()["kernel"] == ("tiles" if tiles else "interval")
            e.reset(2)
            e.set_injection(0, n // 2, 1.0, 0.3)
            e.set_act(0, n // 2, 0, built.ACT["INJ"])
            sp = []
            for k in (1, 99, 137):
                sp += e.step(k)[0]
            runs.append((sp, e.state()[0].copy()))
        finally:
            e.close()
    (a, va), (b, vb) = runs
    assert sum(x.size for x in a) > 0
    for t, (x, y) in enumerate(zip(a, b)):
        np.testing.assert_array_equal(x, y, err_msg="step %d" % t)
    assert np.array_equal(va.view(np.uint8), vb.view(np.uint8))
