"""The expf exception table against the device's filter.

The compat kernels look a result up only when the double exp lies within
2^21 units (of 2^29 per float ulp) of a float rounding boundary; every table
entry must therefore lie well inside that band.  The double exp here and the
device's each err by at most 1 double ulp, i.e. one unit."""
import os

import numpy as np


def test_every_expf_exception_passes_the_filter(built):
    d = np.fromfile(os.path.join(os.path.dirname(built.LIB_PATH), "expf_glibc.bin"), np.uint32)
    x = d[2:2 + int(d[1])].view(np.float32).astype(np.float64)
    bits = np.exp(x).view(np.uint64)
    off = np.abs((bits & np.uint64((1 << 29) - 1)).astype(np.int64) - (1 << 28))
    assert x.size > 0 and int(off.max()) + 2 <= 1 << 21
