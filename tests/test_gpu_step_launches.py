"""The step's launch rules against the oracle, bit for bit: meshes whose
grids lie on both sides of the size up to which kernels are started early
(programmatic dependent launch), in eager and captured steps; and sub-cycles
of one, two, three and ten external steps, whose AB3 velocities alternate
between two buffers and whose elevation is rotated by the next sub-step or,
after the last, by the jacobian kernel."""
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
        for f in ("eta_n", "eta_n_1", "eta_n_2", "U_n_2D", "U_n_1", "U_n_2", "U_filt_2D", "U_n", "V_n", "TF", "SF",
                  "bt", "snu", "Kv", "Av", "Wvel", "mask_wd", "mask_wd_node"):
            assert np.array_equal(sg[f], so[f]), f
    finally:
        g.close()
        o.close()


# elements per 256-thread block of the 2D kernels, times 2 blocks per SM on
# 148 SMs: 75,776 threads; the level kernels cross it at a few thousand
# elements
@pytest.mark.parametrize("nx,ny", [(9, 9), (100, 57), (310, 180)])
def test_early_launch_sizes(built, nx, ny):
    from fesomc import cases
    _compare(lambda lib: cases.estuary_case("e", nx, ny, 300.0, 11, 2.0, 25.0, stress=(0.0, 0.05), lib=lib), 3)


@pytest.mark.parametrize("sub", [1, 2, 3])
def test_sub_cycle_lengths(built, sub):
    from fesomc import cases

    def case_of(lib):
        return cases.estuary_case("e", 23, 14, 300.0, 11, 2.0, 25.0, stress=(0.0, 0.05), lib=lib, dt=2.0 * sub)

    assert case_of(None).params.Mt == sub
    _compare(case_of, 4)


# d3_end on tiles of columns: ragged last tiles of 16 and 32 columns, the
# smallest level count, and the level counts on both sides of the switches
# from 32 to 16 columns (47 interfaces, FP64) and to one thread per column (61)
@pytest.mark.parametrize("nx,ny,nsigma", [(9, 9, 5), (70, 69, 11), (71, 68, 47), (71, 68, 48), (12, 11, 61), (12, 11, 62)])
def test_d3end_tiles(built, nx, ny, nsigma):
    from fesomc import cases
    _compare(lambda lib: cases.estuary_case("e", nx, ny, 300.0, nsigma, 2.0, 25.0, stress=(0.0, 0.05), lib=lib), 3)


# the column solvers on tiles of 32 columns: the smallest and largest layer
# counts, ragged last tiles, more layers than threads of a batch, and the
# element counts around one wave of the viscosity's tiles at 30 layers
# (148 SMs x 4 tiles x 32 = 18,944), with the river's salinity source and,
# in the third variant, the atmospheric sources
@pytest.mark.parametrize("nx,ny,nsigma,atm", [(9, 9, 5, False), (13, 11, 127, False), (25, 17, 33, True),
                                              (160, 89, 31, False), (160, 92, 31, False), (60, 40, 21, False)])
def test_column_solver_tiles(built, nx, ny, nsigma, atm):
    from fesomc import cases
    kw = {"atm": {"qns": -80.0, "qsr": 120.0, "emp": 1e-7, "mslp": 101000.0}} if atm else {}
    _compare(lambda lib: cases.estuary_case("e", nx, ny, 300.0, nsigma, 2.0, 25.0, stress=(0.0, 0.05), lib=lib, **kw), 3)


# biharmonic_2D's first edge pass runs inside adv2d_edge, or on its own
# without the 2D advection; with biharmonic_viscosity the two operators share
# the mesh's coefficients
@pytest.mark.parametrize("params", [{"bih_2D": 1, "mom_adv_2D": 0}, {"bih_2D": 1}, {"bih_3D": 1},
                                    {"bih_2D": 1, "bih_3D": 1, "mom_adv_2D": 0}])
@pytest.mark.parametrize("nx,ny", [(7, 6), (23, 14)])
def test_biharmonic_passes(built, params, nx, ny):
    from fesomc import cases
    _compare(lambda lib: cases.estuary_case("e", nx, ny, 300.0, 11, 2.0, 25.0, stress=(0.0, 0.05), Abh0=1e4, lib=lib,
                                            **params), 4)
