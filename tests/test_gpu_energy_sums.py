"""The energy's compensated sums (block trees, then a tree over the blocks)
against exactly rounded sums, from one entity to several per thread, ragged
last blocks included.  Tolerance: every term is rounded as in the kernel, and
a compensated sum is within two roundings of the exact one, so the three sums
and the two operations on them stay within 8 ulp."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,e", [(3, 1), (255, 257), (20000, 1), (151553, 303107), (400001, 400003)])
def test_sums(built, n, e):
    import torch
    from fesomc import abi
    rng = np.random.default_rng(n + e)
    en = rng.integers(1, n + 1, (e, 4)).astype(np.int32)
    w = rng.random((e, 4))
    eta, depth, area = rng.standard_normal(n), 30.0 * rng.random(n), 1e4 * rng.random(n)
    u, ea = rng.standard_normal((e, 2)), 1e4 * rng.random(e)
    h = np.zeros(e)
    for k in range(4):
        h = h + w[:, k] * np.maximum(1.0, depth[en[:, k] - 1] + eta[en[:, k] - 1])
    pe = math.fsum(0.5 * 9.8 * area * (eta * eta))
    ke = math.fsum(0.5 * h * ea * (u[:, 0] * u[:, 0] + u[:, 1] * u[:, 1]))
    want = (pe + ke) / math.fsum(area)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (eta, depth, area, en, w, u, ea)]
    torch.cuda.synchronize()
    out = C.c_double()
    lib = abi.load()
    rc = lib.fesomc_energy_device(n, e, 1.0, *[t.data_ptr() for t in dev], None, C.byref(out))
    assert rc == 0
    assert abs(out.value - want) <= 8 * np.finfo(float).eps * want
