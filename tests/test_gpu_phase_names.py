"""Every counter that a persistent kernel's phase clock counts has a name in the
benchmark's phase line."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["single_step", "interval", "ltp"])
def test_counters_have_names(built, kernel):
    sys.path.insert(0, ROOT)
    import bench
    from flysim_b200 import netgen, network
    ltp = dict(tLP=20.0, SpiLPDy=1.0, PosISI=2e-4, NegISI=-1e-4) if kernel == "ltp" else None
    na = network.connectome_net(netgen.connectome_fast(n=2000, regions=5, mean_degree=50, seed=2),
                                with_delays=kernel == "interval", ltp=ltp)
    e = built.Engine(na.desc, "fp32", chunk_steps=100)
    try:
        assert e.layout()["kernel"] == kernel
        e.reset(1)
        e.phase_clock(True)
        e.run(100)
        e.sync()
        used = set(np.flatnonzero(e.phase_times().sum(0)).tolist())
        line = bench.phase_line(e, 100)
    finally:
        e.close()
    assert used == set(bench.PHASES[kernel]), used
    assert len(line) == len(used) and all(v["max"] > 0 for v in line.values())
