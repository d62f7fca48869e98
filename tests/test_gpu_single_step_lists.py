"""The single-step kernel's spike lists: regions of two spikes a block, read by
polling, a few more per block read in place and bursts block by block, in blocks
with helper warps (at most 256 posts) and without.  Every network here spikes in
bursts (a drive that hits a whole range of neurons at once), and every value is
compared bit for bit with the interval kernel's, which has no such lists."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, burst, plast", [
    (6, 6, None),          # two blocks, fewer posts than a warp
    (1009, 40, None),      # some blocks with 3-8 spikes a step
    (1009, 1009, None),    # every neuron of a block at once
    (20011, 3000, None),   # full blocks next to empty ones
    (20011, 20011, "tm"),
    (45007, 45007, None),  # more than 256 posts a block: no helper warps
])
def test_bursts_equal_interval_kernel(built, n, burst, plast):
    from flysim_b200 import netgen, network
    na = network.connectome_net(netgen.connectome_fast(n=n, regions=max(2, n // 345), mean_degree=min(60, n // 2), seed=4),
                                with_delays=False, tm=plast == "tm")
    runs = []
    for interval in (False, True):
        e = built.Engine(na.desc, "fp32", chunk_steps=150, interval_kernel=interval)
        try:
            assert e.layout()["single_step"] == (not interval)
            sp = []
            for seed in (3, 4):  # the second run's tags go on where the first's ended
                e.reset(seed)
                e.set_injection(0, burst, 30.0, 0.0)  # spikes of the whole range in one step
                e.set_act(0, burst, 0, built.ACT["INJ"])
                for k in (1, 1, 120, 201):
                    sp += e.step(k)[0]
            runs.append((sp, e.state()[0].copy(), e.spike_counts()))
        finally:
            e.close()
    (a, va, ca), (b, vb, cb) = runs
    assert max(x.size for x in b) >= min(burst, 6)
    for t, (x, y) in enumerate(zip(a, b)):
        np.testing.assert_array_equal(x, y, err_msg="step %d" % t)
    assert np.array_equal(va.view(np.uint32), vb.view(np.uint32))
    np.testing.assert_array_equal(ca, cb)
