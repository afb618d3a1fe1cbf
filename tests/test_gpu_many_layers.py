"""Kernel forms of meshes with many layers against the oracle, bit for bit:
the implicit viscosity's tiles of 32, 16 and 8 columns on both sides of their
choices (54 and 55, 105 and 106 layers) with whole and ragged last tiles, and the column
kernels' entities per block, which change with the level count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(case_of, steps):
    import pyoracle
    from fesomc import abi, cases, model
    g = model.GpuModel(case_of(None))
    o = pyoracle.Oracle(case_of(pyoracle.MeshLib(abi)), abi, cases)
    try:
        g.step(steps)
        o.step(steps)
        sg, so = g.state(), o.state()
        for f in ("eta_n", "U_n_2D", "U_n", "V_n", "U_n_filt", "TF", "SF", "bt", "snu", "Kv", "Ri", "tke_dissip", "Av", "Wvel",
                  "rho_c", "hpressure", "Bar_pr_2D"):
            assert np.array_equal(sg[f], so[f]), f
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("nx,ny,nsigma,kw", [(12, 11, 55, {}), (12, 11, 56, {}), (19, 13, 91, {"fic_point": 0}),
                                             (21, 12, 106, {}), (21, 12, 107, {"fic_point": 2}), (33, 17, 127, {})])
def test_implicit_viscosity_tiles(built, nx, ny, nsigma, kw):
    from fesomc import cases
    _compare(lambda lib: cases.estuary_case("e", nx, ny, 300.0, nsigma, 2.0, 25.0, stress=(0.0, 0.05), lib=lib, **kw), 3)


@pytest.mark.parametrize("nsigma", [18, 25, 28, 45, 54, 55, 70, 84, 97, 101, 106, 108, 120, 121])
def test_columns_per_block(built, nsigma):
    from fesomc import cases
    _compare(lambda lib: cases.estuary_case("e", 13, 11, 300.0, nsigma, 2.0, 25.0, stress=(0.0, 0.05), lib=lib), 3)
