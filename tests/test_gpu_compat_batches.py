"""Steps that the reference-order engine runs at once: calls with per-step outputs,
which lie in device memory for the whole batch, are cut at 64 M random draws."""
import numpy as np
import pytest

from conftest import model_for

pytestmark = pytest.mark.gpu


def test_calls_with_outputs_are_cut(built):
    m = model_for(built, "two_pop")  # five draws a neuron and step
    runs = []
    for want_V in (False, True):
        e = built.Engine(m.desc(), "compat", chunk_steps=1 << 20)  # (a reset keeps the group gates)
        try:
            steps = (64 << 20) // (5 * e.n) + 100
            e.reset(m.seed())
            sp, V = e.step(steps, want_V=want_V, spike_cap=1 << 22)
            runs.append((sp, V, e.state()[0].copy(), e.stats()["launches"]))
        finally:
            e.close()
    m.close()
    (a, _, va, la), (b, V, vb, lb) = runs
    assert lb == 2 * la  # two batches instead of one
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
    np.testing.assert_array_equal(va, vb)
    np.testing.assert_array_equal(V[-1], vb)
