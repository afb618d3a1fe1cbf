"""The forms of d3_end, which the launch-shape knob "d3end_arrays" or the
mesh's sizes choose: in the FP32 form the same bits under every number, over
the level counts at the edges of the forms, on meshes that are no multiple of
their blocks; in FP64 against the oracle on both sides of the choices by
shared memory (48 and 49 levels: 32 or 16 columns above 4,736 nodes; 62 and
63: tiles or one thread per column)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(nx, ny, nsigma, fp32, shapes, steps=3):
    from fesomc import autotune, cases, model
    g = model.GpuModel(cases.estuary_case("e", nx, ny, 300.0, nsigma, 2.0, 25.0, stress=(0.0, 0.05), fp32_form=fp32))
    try:
        autotune.apply(g, shapes)
        assert g.step(steps) == 0
        return g.state(), g.status()
    finally:
        g.close()


@pytest.mark.parametrize("nx,ny,nsigma", [(9, 9, 5), (40, 16, 11), (23, 14, 16), (71, 68, 21), (33, 21, 31), (25, 17, 40),
                                          (25, 17, 41), (21, 13, 62), (12, 11, 127)])
def test_fp32_forms_give_the_same_bits(built, nx, ny, nsigma):
    want, status = _run(nx, ny, nsigma, 1, {"d3end_arrays": 1})
    for form in (2, 3, 4, 5, 6):
        got, st = _run(nx, ny, nsigma, 1, {"d3end_arrays": form})
        assert st == status
        for k, v in want.items():
            if not k.startswith("_"):
                assert np.array_equal(got[k], v), (form, k)


@pytest.mark.parametrize("nx,ny,nsigma", [(71, 68, 48), (71, 68, 49), (71, 68, 62), (12, 11, 62), (12, 11, 63), (71, 68, 63)])
def test_fp64_sides_of_the_choices(built, nx, ny, nsigma):
    import pyoracle
    from fesomc import abi, cases, model

    def case_of(lib):
        return cases.estuary_case("e", nx, ny, 300.0, nsigma, 2.0, 25.0, stress=(0.0, 0.05), lib=lib)

    g = model.GpuModel(case_of(None))
    o = pyoracle.Oracle(case_of(pyoracle.MeshLib(abi)), abi, cases)
    try:
        g.step(3)
        o.step(3)
        sg, so = g.state(), o.state()
        for f in ("bt", "snu", "Kv", "Ri", "tke_dissip", "Av", "U_n", "V_n", "TF", "SF", "eta_n"):
            assert np.array_equal(sg[f], so[f]), f
    finally:
        g.close()
        o.close()
