"""Receptors no neuron uses are left out of a step (Params::live), batches of
steps are spread over tiles of 64, 128 or 256 posts, and networks without
delays keep no history of s.  None of it may show: every run here is compared
bit for bit with one whose receptors all count as used (one neuron has a drive
of 1e-30 on each but AMPA, where every neuron has its own; it hits with a chance
of 2^-24 a draw at most; and an injection of 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALL = ("AMPA", "GABA", "ACH", "GCL", "NMDA", "INJ")


def _scenario(fb, e, seed=6):
    """Spikes and the membrane after calls of uneven length between which a
    drive comes on, goes off, and an injection starts."""
    e.reset(seed)
    sp = []
    sp += e.step(37)[0]
    e.set_drive(5, 900, fb.FS_ACH, 0.06)
    e.set_drive(5, 900, fb.FS_AMPA, 0.5)
    sp += e.step(50)[0]
    e.set_drive(5, 900, fb.FS_ACH, 0.0)
    e.set_injection(100, 400, 1.0, 0.3)
    e.set_act(100, 400, 0, fb.ACT["INJ"])
    sp += e.step(1)[0]
    ck = e.checkpoint()
    sp += e.step(93)[0]
    return sp, e.state()[0].copy(), ck


def _same(a, b):
    assert len(a[0]) == len(b[0])
    for t, (x, y) in enumerate(zip(a[0], b[0])):
        np.testing.assert_array_equal(x, y, err_msg="step %d" % t)
    assert np.array_equal(a[1].view(np.uint8), b[1].view(np.uint8))


@pytest.mark.parametrize("mode, n, delays, kernel", [
    ("fp32", 5003, True, "interval"),    # tiles of 128 posts
    ("fp32", 45001, True, "interval"),   # of 256
    ("fp32", 5003, False, "interval"),   # s read from the neurons, no history
    ("fp32", 5003, True, "tiles"),
    ("fp32", 76001, False, "tiles"),     # (beyond the single-step kernel)
    ("fp64", 3001, True, "interval"),    # of 64
    ("fp64", 20011, True, "interval"),   # of 128
    ("fp64", 3001, False, "tiles"),
    ("fp32", 3001, False, "ltp"),
    ("fp64", 3001, False, "ltp"),
])
def test_dead_receptors_do_not_show(built, mode, n, delays, kernel):
    from flysim_b200 import netgen, network
    ltp = dict(tLP=20.0, SpiLPDy=1.0, PosISI=2e-4, NegISI=-1e-4) if kernel == "ltp" else None
    na = network.connectome_net(netgen.connectome_fast(n=n, regions=20, seed=3), with_delays=delays, ltp=ltp)
    opt = dict(chunk_steps=64)
    if kernel != "ltp":
        opt.update(interval_kernel=kernel == "interval", tile_kernels=kernel == "tiles")
    runs = []
    for everything in (False, True):
        e = built.Engine(na.desc, mode, **opt)
        try:
            assert e.layout()["kernel"] == kernel
            if everything:
                for r in (r for r in range(built.FS_NREC) if r != built.FS_AMPA):
                    e.set_drive(7, 1, r, 1e-30)
                e.set_injection(7, 1, 0.0, 0.0)
                for k in ALL:
                    e.set_act(7, 1, 0, built.ACT[k])
            runs.append(_scenario(built, e))
        finally:
            e.close()
    assert sum(x.size for x in runs[0][0]) > 50
    _same(*runs)
    # a new handle goes on from the checkpoint; without delays the interval
    # kernel, or the tiles, from the other's (or the single-step kernel's) too
    others = [opt]
    if not delays and kernel != "ltp":
        others = [dict(chunk_steps=64, interval_kernel=i, tile_kernels=t) for i, t in
                  ((True, False), (False, True)) + (((False, False),) if mode == "fp32" else ())]
    for o in others:
        e = built.Engine(na.desc, mode, **o)
        try:
            e.reset(1)
            e.restore(runs[0][2])
            _same((runs[0][0][88:], runs[0][1]), (e.step(93)[0], e.state()[0].copy()))
        finally:
            e.close()
