"""Compat kernel (k_compat) at the edges of its tiles against the CPU oracle:
more neurons than the resident blocks hold at 64 a tile (neurons loaded and
stored every step), a post whose records alone overflow a pass of shared
memory, ragged tiles and a few neurons.  Every value equals the oracle's (the
mode's bar is bit equality)."""
import ctypes as C

import numpy as np
import pytest

from conftest import OracleEngine
from flysim_b200 import ACT, DEFAULT_ACT, FS_AMPA, FS_GABA, FS_NMDA, FS_NREC, network

pytestmark = pytest.mark.gpu


def _net(fb, n, degree, seed, hub=0, gap=False, plastic=0):
    rng = np.random.default_rng(seed)
    pre = np.repeat(np.arange(n), degree)
    post = rng.integers(0, n, pre.size)
    if hub:
        pre = np.concatenate([pre, rng.integers(0, n, hub)])
        post = np.concatenate([post, np.full(hub, n // 2)])
    rec = rng.choice([FS_AMPA, FS_GABA, FS_NMDA], pre.size).astype(np.uint8)
    g = rng.uniform(0.01, 0.4, pre.size).astype(np.float32)
    act = DEFAULT_ACT | plastic
    f = network.neuron_fields(n, 0.1, act=act, receptors={
        FS_AMPA: dict(Tau=2.0, FExt=rng.uniform(2000, 5000, n)), FS_GABA: dict(Tau=5.0, Vrev=-70.0),
        FS_NMDA: dict(Tau=100.0, TauXT=2.0)})
    if plastic & ACT["STD"]:
        f["stp_pv"][:] = 0.3
        f["stp_dfD"][:] = np.exp(np.float32(-0.1 / 200))
        f["stp_efD"][:] = 1 - f["stp_dfD"]
    na = network.desc_from_arrays(n, 0.1, f, pre, post, rec, g, act_ctr=act)
    lay, u32, f32 = fb.CompatLayout(), C.POINTER(C.c_uint32), C.POINTER(C.c_float)
    keep = [lay]

    def ptr(a, ty, ct):
        keep.append(np.ascontiguousarray(a, ty))
        return keep[-1].ctypes.data_as(ct)

    for r in range(FS_NREC):
        e = np.flatnonzero(rec == r)
        e = e[np.argsort(post[e], kind="stable")]
        R = lay.rec[r]
        R.n_recs = e.size
        R.rec_pre, R.rec_post = ptr(pre[e], np.uint32, u32), ptr(post[e], np.uint32, u32)
        R.rec_g = ptr(g[e], np.float32, f32)
        R.rec_rowptr = ptr(np.concatenate([[0], np.cumsum(np.bincount(post[e], minlength=n))]), np.uint32, u32)
    if gap:
        a = rng.integers(0, n, 2 * n)
        row = np.concatenate([[0], np.cumsum(rng.multinomial(2 * n, np.full(n, 1.0 / n)))])
        lay.gap_rowptr, lay.gap_other = ptr(row, np.uint32, u32), ptr(a, np.uint32, u32)
        lay.gap_g = ptr(rng.uniform(0, 0.002, 2 * n), np.float32, f32)
    na.desc.compat = C.pointer(lay)
    na._keep += keep
    return na


@pytest.mark.parametrize("n,degree,hub,gap,plastic,calls", [
    (31009, 6, 0, True, 0, (70, 75)),               # two tiles a block
    (1000, 20, 16000, False, 0, (60, 61)),          # a hub: several passes
    (37, 9, 0, True, ACT["STD"], (1, 2, 150)),      # fewer neurons than a warp pair, odd call lengths
    (9001, 30, 0, False, ACT["STD"], (80,)),
])
def test_tiles_equal_oracle(built, oracle, n, degree, hub, gap, plastic, calls):
    na = _net(built, n, degree, 3, hub, gap, plastic)
    e, o = built.Engine(na.desc, "compat"), OracleEngine(built, oracle, C.pointer(na.desc))
    e.reset(7)
    o.reset(7)
    spikes = 0
    try:
        for k in calls:
            sp_g, _ = e.step(k)
            sp_o = o.step(k)
            for a, b in zip(sp_g, sp_o):
                np.testing.assert_array_equal(a, b)
                spikes += a.size
            V, cnt, ns = e.state()
            G, isyn = e.syn_state()
            oV, ocnt, ons, oG, oisyn = o.state()
            assert V.tobytes() == oV.tobytes() and G.tobytes() == np.asarray(oG).reshape(G.shape).tobytes()
            assert isyn.tobytes() == oisyn.tobytes()
            np.testing.assert_array_equal(cnt, ocnt)
            np.testing.assert_array_equal(ns, ons)
        assert spikes > 0
    finally:
        e.close()
