"""Kernel forms of meshes with few layers on large grids against the oracle,
bit for bit, and against the forms of small grids: a member alone (small) and
in a pack whose total lies beyond every choice by size, in both precision
forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("eta_n", "U_n_2D", "U_n", "V_n", "TF", "SF", "T_old", "S_old", "bt", "snu", "Kv", "Ri", "tke_dissip", "Av", "Wvel")


# 48,461 nodes, about 63 k elements: not a multiple of the tiles' 64 columns
@pytest.mark.parametrize("nsigma,kw", [(n, {}) for n in range(5, 12)] + [(11, {"fic_point": 0}), (6, {"fic_point": 2})])
def test_large_grid_bit_exact(built, nsigma, kw):
    import pyoracle
    from fesomc import abi, cases, model

    def case_of(lib):
        return cases.estuary_case("e", 300, 160, 300.0, nsigma, 2.0, 25.0, stress=(0.0, 0.05), lib=lib, **kw)

    g = model.GpuModel(case_of(None))
    o = pyoracle.Oracle(case_of(pyoracle.MeshLib(abi)), abi, cases)
    try:
        assert g.case.mesh.N == 48461
        g.step(2)
        o.step(2)
        sg, so = g.state(), o.state()
        for f in FIELDS:
            assert np.array_equal(sg[f], so[f]), f
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("nsigma", [5, 8, 11])
def test_member_alone_and_packed(built, nsigma, fp32):
    from fesomc import cases, ensemble
    members = [cases.estuary_case("m%d" % i, nx, ny, 300.0, nsigma, 2.0, 25.0, stress=(0.02 * i, 0.05), seed=100 + i,
                                  fp32_form=fp32) for i, (nx, ny) in enumerate([(30, 20), (310, 160), (33, 21)])]
    ens = ensemble.PackedEnsemble(members)
    try:
        _, status = ens.run(3)
        assert status == [0] * len(members)
        packed = [ens.member_state(i) for i in range(len(members))]
    finally:
        ens.close()
    for i, c in enumerate(members):
        if i == 1:
            continue
        one = ensemble.Ensemble([c])
        try:
            one.run(3)
            alone = one.models[0].state()
        finally:
            one.close()
        for f in FIELDS:
            assert np.array_equal(packed[i][f], alone[f]), (i, f)
