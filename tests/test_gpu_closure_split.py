"""The network's gradients where the weight gradients' split of the batch and
the tiles have their edges: one sample, a full part, a sample more or less, a
second part, the largest batch; the fewest and the most levels.  Against the
CPU restatement in double, with the tolerances of the other gradient tests
(relative 1e-3 per array, 1e-5 on the loss)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsigma,batch", [(21, 1), (5, 255), (21, 256), (21, 257), (32, 513), (11, 8192)])
def test_gradients_at_the_splits(built, nsigma, batch):
    import pyoracle
    from fesomc import abi, closure
    rng = np.random.default_rng(nsigma * batch)
    c = closure.Closure(nsigma)
    try:
        p = (0.06 * rng.standard_normal(c.nparams)).astype(np.float32)
        c.params(p)
        X = rng.standard_normal((batch, c.n_in)).astype(np.float32)
        T = rng.standard_normal((batch, c.n_out)).astype(np.float32)
        loss, g = c.grad(X, T)
        lo, go = pyoracle.mlp_grad(abi, nsigma, p, X, T)
        assert abs(loss - lo) <= 1e-5 * lo
        dims, o = [c.n_in, 256, 256, 256, c.n_out], 0
        for l in range(4):
            for n in (dims[l + 1] * dims[l], dims[l + 1]):
                a, b = g[o:o + n].astype(np.float64), go[o:o + n]
                assert np.linalg.norm(a - b) <= 1e-3 * np.linalg.norm(b), (l, n)
                o += n
    finally:
        c.close()
