"""Kernel forms that are chosen by size give a mesh the same bits on its own
and as a member of a pack whose total lies on the other side of the choice,
in both precision forms: the sub-cycle's early-start kernels (2 blocks per
SM), d3_end's tiles of 16 and 32 columns (4,736 nodes) and, at 21 levels,
the vertical diffusion's register tiles (37,888 nodes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _member(i, nx, ny, nsigma, fp32):
    from fesomc import cases
    return cases.estuary_case("m%d" % i, nx, ny, 300.0, nsigma, 2.0, 25.0, stress=(0.02 * i, 0.05), seed=100 + i,
                              fp32_form=fp32)


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("sizes,nsigma", [([(40, 30), (90, 45), (61, 33)], 11), ([(30, 20), (250, 150), (33, 21)], 21)])
def test_member_alone_and_packed(built, sizes, nsigma, fp32):
    from fesomc import ensemble, model
    members = [_member(i, nx, ny, nsigma, fp32) for i, (nx, ny) in enumerate(sizes)]
    ens = ensemble.PackedEnsemble(members)
    try:
        _, status = ens.run(4)
        assert status == [0] * len(members)
        packed = [ens.member_state(i) for i in range(len(members))]
    finally:
        ens.close()
    for i, c in enumerate(members):
        one = ensemble.Ensemble([c])
        try:
            one.run(4)
            alone = one.models[0].state()
        finally:
            one.close()
        for f in ("eta_n", "U_n_2D", "U_n", "V_n", "TF", "SF", "bt", "snu", "Kv", "Av", "Wvel"):
            assert np.array_equal(packed[i][f], alone[f]), (i, f)
