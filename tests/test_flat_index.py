"""The 32-bit reciprocal division of flat (entity, level) indices (FastDiv in
csrc/device_common.cuh): its formula against exact division for every level
count the library takes, at the indices where a wrong multiplier shows first
(around multiples of the divisor up to 2^31)."""
import os
import re

import numpy as np

from conftest import ROOT


def test_formula_is_exact_below_two_to_31():
    src = open(os.path.join(ROOT, "fesom-c_b200", "csrc", "device_common.cuh")).read()
    body = re.search(r"struct FastDiv \{(.*?)\n\};", src, re.S).group(1)
    # the formula restated below is the one in the source
    assert "while ((1ull << b) < d) ++b;" in body and "(1ull << (31 + b)) / d + 1" in body and "s = b - 1;" in body
    assert "__umulhi(n, m) >> s" in body
    rng = np.random.default_rng(1)
    top = 2**31 - 1
    for d in range(2, 129):
        b = 1
        while (1 << b) < d:
            b += 1
        m = (1 << (31 + b)) // d + 1
        assert m < 2**32
        q = np.concatenate([np.arange(0, 1000), rng.integers(0, top // d + 1, 2000), np.arange(top // d - 1000, top // d + 1)])
        n = (q[:, None] * d + np.array([-1, 0, 1, d - 1])).ravel()
        n = n[(n >= 0) & (n <= top)].astype(np.uint64)
        got = ((n * np.uint64(m)) >> np.uint64(32)) >> np.uint64(b - 1)
        assert np.array_equal(got, n // np.uint64(d)), d
