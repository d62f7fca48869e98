"""The interval and tile kernels over the lengths of a batch and in-degrees where
their pull, history and loads branch: smallest delays of 1 to 20 steps (batches of
one step, of up to eight, of more, cut at sixteen), posts with none to several
rounds of NMDA edges, neurons that project onto no NMDA receptor.

Potentials and spikes against the float64 restatement (2e-3 mV, the FP32 bar of
test_gpu_production.py; the targets stay below threshold), and the same bits
however the steps are split into calls."""
import numpy as np
import pytest

import prod_model

pytestmark = pytest.mark.gpu

DEG = (0, 1, 2, 9, 10, 11, 30, 31, 39, 40, 41, 64, 65, 79, 80, 81, 90)


def _net(fb, dmin, seed):
    """90 sources that project onto NMDA (and AMPA) receptors, 30 that project
    onto AMPA only, 190 targets."""
    from flysim_b200 import network
    rng = np.random.default_rng(seed)
    n_nm, n_src, n = 90, 120, 310
    f = network.neuron_fields(n, 0.1, receptors={
        fb.FS_AMPA: dict(Tau=2.0, Vrev=0.0, FExt=0.0), fb.FS_NMDA: dict(Tau=100.0, TauXT=2.0, Vrev=0.0, FExt=0.0)})
    f["act"][:n_src] |= fb.ACT["INJ"]
    f["inj_mean"][:n_src] = rng.uniform(0.8, 2.0, n_src)
    pre, post, rec, g = [], [], [], []
    for i in range(n_src, n):
        k = DEG[i % len(DEG)]
        a = rng.choice(n_nm, k, replace=False)
        b = rng.choice(n_src, 5, replace=False)
        pre += [a, b]
        post += [np.full(k + 5, i)]
        rec += [np.full(k, fb.FS_NMDA), np.full(5, fb.FS_AMPA)]
        g += [rng.uniform(0.5, 1.5, k) * (4.0 / max(k, 4)), rng.uniform(0.02, 0.1, 5)]
    pre = np.concatenate(pre)
    d = dmin + rng.integers(0, 30, pre.size)
    d[0] = dmin
    return network.desc_from_arrays(n, 0.1, f, pre.astype(np.uint32), np.concatenate(post).astype(np.uint32),
                                    np.concatenate(rec).astype(np.uint8), np.concatenate(g).astype(np.float32),
                                    d.astype(np.uint16))


@pytest.mark.parametrize("tiles", [False, True])
@pytest.mark.parametrize("dmin", [1, 2, 3, 5, 8, 9, 12, 13, 16, 20])
def test_batches_match_restatement_and_any_split(built, dmin, tiles):
    na = _net(built, dmin, dmin)
    steps = 400
    ref_sp, ref_V = prod_model.simulate(na, steps)
    assert sum(x.size for x in ref_sp) > 200 and all(np.all(x < 120) for x in ref_sp)
    runs = []
    for split in ((steps,), (1,) * 45 + (3, 7, 50, 2, 11, 17, 65, 200)):
        assert sum(split) == steps
        e = built.Engine(na.desc, "fp32", chunk_steps=1000, tile_kernels=tiles)
        try:
            assert e.layout()["kernel"] == ("tiles" if tiles else "interval") and e.layout()["interval"] == dmin
            e.reset(1)
            sp, V = [], []
            for k in split:
                a, b = e.step(k, want_V=True)
                sp += a
                V.append(b.copy())
            runs.append((sp, np.concatenate(V)))
        finally:
            e.close()
    for t in range(steps):
        np.testing.assert_array_equal(runs[0][0][t], ref_sp[t], err_msg="spikes at step %d" % t)
        np.testing.assert_array_equal(runs[1][0][t], ref_sp[t], err_msg="spikes at step %d, split" % t)
    assert np.abs(runs[0][1].astype(np.float64) - ref_V).max() < 2e-3
    assert np.array_equal(runs[0][1].view(np.uint32), runs[1][1].view(np.uint32))
    moved = np.ptp(ref_V[:, 120:], axis=0)
    assert (moved > 0.01).mean() > 0.9  # (nearly all targets felt their input)
