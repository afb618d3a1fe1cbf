"""The FP32 network on tiles of 64 and of 128 rows: a column's outputs have
the same bits whatever else is in the batch, below and above the batch size
from which the tiles are taller (4,608 columns for the hidden layers), at
ragged last tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsigma", [5, 21, 32])
def test_forward_does_not_depend_on_the_batch(built, nsigma):
    from fesomc import closure
    rng = np.random.default_rng(nsigma)
    c = closure.Closure(nsigma)
    try:
        c.params((0.06 * rng.standard_normal(c.nparams)).astype(np.float32))
        X = rng.standard_normal((8192, c.n_in)).astype(np.float32)
        whole = c.forward(X)
        for n in (1, 63, 64, 65, 127, 129, 1000, 4608, 4609, 4737):
            assert np.array_equal(c.forward(X[:n]), whole[:n]), n
    finally:
        c.close()
