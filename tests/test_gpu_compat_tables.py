"""The exception tables of the reference-order engine: one hashed copy a device,
whatever the number of handles, given back with the last."""
import threading

import numpy as np
import pytest

from conftest import model_for

pytestmark = pytest.mark.gpu


def test_handles_share_the_tables(built):
    import torch
    m = model_for(built, "two_pop")
    first = built.Engine(m.desc(), "compat", chunk_steps=10)
    free = torch.cuda.mem_get_info()[0]
    more = [built.Engine(m.desc(), "compat", chunk_steps=10) for _ in range(24)]
    try:
        # a copy each took 24 x 8 MB and more
        assert free - torch.cuda.mem_get_info()[0] <= 24 * (4 << 20)
        want = None
        first.close()  # the others keep them
        for e in (more[0], more[-1]):
            e.reset(m.seed())
            got = [x.tolist() for x in e.step(300)[0]]
            want = want or got
            assert got == want and sum(map(len, got)) > 0
    finally:
        for e in [first] + more:
            e.close()
        m.close()


def test_handles_made_and_closed_on_threads(built):
    m = model_for(built, "two_pop")
    out = [None] * 6

    def work(k):
        for _ in range(3):
            e = built.Engine(m.desc(), "compat", chunk_steps=10)
            e.reset(m.seed())
            out[k] = np.concatenate(e.step(120)[0])
            e.close()

    th = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    m.close()
    for o in out:
        np.testing.assert_array_equal(o, out[0])
