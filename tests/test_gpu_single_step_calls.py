"""Calls of one step on the single-step kernel, with blocks of very different
work: a launch of one step exchanges no spike lists, and a light block must not
store its neurons' new NMDA state while a heavy one still reads the old.  Every
value bit for bit that of the interval kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uneven(hubs, per_hub, n, seed):
    """n neurons, the first `hubs` with per_hub inputs each, the others with
    one or two; drives strong enough that most neurons fire."""
    from flysim_b200 import netgen, network
    rng = np.random.default_rng(seed)
    pre = [rng.choice(n, per_hub, replace=False) for _ in range(hubs)] + [rng.integers(0, n, 2) for _ in range(hubs, n)]
    post = [np.full(p.size, i) for i, p in enumerate(pre)]
    key = np.unique(np.concatenate(pre).astype(np.int64) * n + np.concatenate(post))
    pre, post = (key // n).astype(np.uint32), (key % n).astype(np.uint32)
    c = netgen.connectome_fast(n=n, regions=2, mean_degree=4, seed=seed)
    c.excit[:] = True
    c.pre, c.post = pre, post
    c.weight = rng.uniform(0.02, 0.2, pre.size).astype(np.float32)
    c.delay_ms = np.zeros(pre.size, np.uint16)
    c.freq_ext = np.full(n, 6000.0, np.float32)
    return network.connectome_net(c, with_delays=False)


@pytest.mark.parametrize("hubs, per_hub, n", [(8, 3000, 6000), (3, 800, 1001), (40, 900, 30000)])
def test_one_step_calls_on_uneven_blocks(built, hubs, per_hub, n):
    na = _uneven(hubs, per_hub, n, seed=hubs)
    runs = []
    for interval in (False, True):
        e = built.Engine(na.desc, "fp32", chunk_steps=100, interval_kernel=interval)
        try:
            assert e.layout()["single_step"] == (not interval)
            e.reset(5)
            sp, v = [], []
            for _ in range(300):
                sp.append(e.step(1)[0][0])
                v.append(e.state()[0].copy())
            sp += e.step(101)[0]  # a chunk's remainder of one step
            v.append(e.state()[0].copy())
            runs.append((sp, np.array(v), e.spike_counts()))
        finally:
            e.close()
    (a, va, ca), (b, vb, cb) = runs
    assert sum(x.size for x in b) > 0
    for t, (x, y) in enumerate(zip(a, b)):
        np.testing.assert_array_equal(x, y, err_msg="step %d" % t)
    assert np.array_equal(va.view(np.uint32), vb.view(np.uint32))
    np.testing.assert_array_equal(ca, cb)
