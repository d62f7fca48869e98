"""The LTP kernel's NMDA pull takes twelve rows of eight edges of a post at once
and the next posts' first rows meanwhile.  With learning rates of 0 no weight
changes, so its runs equal the single-step kernel's (whose sums are its own) bit
for bit, whatever the in-degrees: none to a few, around twelve rows, several
rounds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, degree", [(5, 2), (301, 3), (1203, 137), (1999, 420)])
def test_ltp_kernel_without_learning_equals_single_step(built, n, degree):
    from flysim_b200 import netgen, network
    c = netgen.connectome_fast(n=n, regions=2, mean_degree=degree, seed=6)
    runs = []
    for ltp in (None, dict(tLP=20.0, SpiLPDy=1.0, PosISI=0.0, NegISI=0.0)):
        na = network.connectome_net(c, with_delays=False, ltp=ltp)
        e = built.Engine(na.desc, "fp32", chunk_steps=100)
        try:
            assert e.layout()["kernel"] == ("ltp" if ltp else "single_step")
            e.reset(8)
            e.set_injection(0, n, 1.0, 0.3)
            e.set_act(0, n, 0, built.ACT["INJ"])
            sp = []
            for k in (1, 99, 150):
                sp += e.step(k)[0]
            runs.append((sp, e.state()[0].copy()))
        finally:
            e.close()
    (a, va), (b, vb) = runs
    assert sum(x.size for x in a) > 0
    for t, (x, y) in enumerate(zip(a, b)):
        np.testing.assert_array_equal(x, y, err_msg="step %d" % t)
    assert np.array_equal(va.view(np.uint32), vb.view(np.uint32))
