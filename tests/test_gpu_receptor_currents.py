"""Per-receptor currents (want_Irep) of receptors that no synapse and no drive
uses: 0 * (Vrev - V), a zero with the sign of the driving force, which the
IsynSeparatedSum files print ("-0"); in every production kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp32", "fp64"])
@pytest.mark.parametrize("kind", ["default", "interval", "tiles", "ltp", "delays"])
def test_unused_receptors_give_signed_zeros(built, mode, kind):
    from flysim_b200 import netgen, network
    c = netgen.connectome_fast(n=600, regions=2, mean_degree=30, seed=2)
    ltp = dict(tLP=20.0, SpiLPDy=1.0, PosISI=2e-4, NegISI=-1e-4) if kind == "ltp" else None
    na = network.connectome_net(c, with_delays=kind == "delays", ltp=ltp)
    # Vrev 0 mV (ACh) lies above, Vrev -90 mV (GluCl) below every potential the
    # current is formed at (a spike's V = 0 falls in the refractory steps)
    e = built.Engine(na.desc, mode, chunk_steps=100, interval_kernel=kind == "interval", tile_kernels=kind == "tiles")
    try:
        e.reset(3)
        _, V, I, _ = e.step(60, want_V=True, want_Irep=True, want_nstate=True)
    finally:
        e.close()
    assert V.min() > -90.0
    for r, neg in ((built.FS_ACH, False), (built.FS_GCL, True)):
        assert np.all(I[:, r] == 0.0)
        assert np.all(np.signbit(I[:, r]) == neg), "receptor %d" % r
    assert np.any(I[:, built.FS_AMPA] != 0.0)
