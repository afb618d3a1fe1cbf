"""The column kernels' blocks against the oracle, bit for bit: entities per
block from one to the most, level counts whose blocks are not whole warps,
ragged last blocks, and a mesh with a node of more edges than a block's
staging holds (the edge lists are then read where they are used)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("eta_n", "U_n_2D", "U_n", "V_n", "U_n_filt", "V_n_filt", "TF", "SF", "bt", "snu", "Kv", "Av", "Wvel", "hpressure",
          "Bar_pr_2D")


def _compare(case_of, steps, columns):
    import pyoracle
    from fesomc import abi, autotune, cases, model
    g = model.GpuModel(case_of(None))
    o = pyoracle.Oracle(case_of(pyoracle.MeshLib(abi)), abi, cases)
    try:
        if columns:
            autotune.apply(g, {"columns": columns})
        g.step(steps)
        o.step(steps)
        sg, so = g.state(), o.state()
        for f in FIELDS:
            assert np.array_equal(sg[f], so[f]), f
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("nsigma,columns", [(5, 0), (11, 1), (11, 32), (21, 0), (21, 3), (38, 0), (127, 0)])
def test_block_sizes(built, nsigma, columns):
    from fesomc import cases
    _compare(lambda lib: cases.estuary_case("e", 19, 13, 300.0, nsigma, 2.0, 25.0, stress=(0.0, 0.05), lib=lib), 3, columns)


def _fan(lib, spokes=12):
    """A closed basin: a node with `spokes` edges in a ring of triangles and a
    ring of quads, a temperature front across it."""
    from fesomc import abi, cases
    ang = 2.0 * math.pi * np.arange(spokes) / spokes
    ring = np.stack([np.cos(ang), np.sin(ang)], axis=1)
    xy = np.concatenate([[[0.0, 0.0]], 1000.0 * ring, 2000.0 * ring])
    index = np.array([0] * (1 + spokes) + [1] * spokes, dtype=np.int32)
    a = 2 + np.arange(spokes)                       # inner ring, 1-based
    b = 2 + (np.arange(spokes) + 1) % spokes
    tri = np.stack([np.ones(spokes, dtype=int), b, a, np.ones(spokes, dtype=int)], axis=1)
    quad = np.stack([a, b, b + spokes, a + spokes], axis=1)
    elems = np.concatenate([quad, tri]).astype(np.int32)
    mesh = cases.HostMesh(xy, index, elems, np.full(len(xy), 20.0), cartesian=True, nsigma=11, coriolis_on=True, lib=lib)
    lib = lib if lib is not None else abi.load()
    p = cases.default_params(dt=4.0, dt_2D=2.0, tracer_adv=abi.TRACER_MUSCL, salinity_on=1)
    p.scale_area = mesh.scale_area
    p.density_0 = 1000.0 + lib.fesomc_host_density_jm(12.0, 30.0, 0.0, 1000.0)
    x = mesh.coord_nod2D[:, 0]
    TF = np.repeat(np.where(x < 0.0, 10.0, 14.0)[:, None], mesh.L, axis=1)
    st = cases.initial_state(mesh, p, TF, np.full_like(TF, 30.0), wet_dry_on=False)
    ze, zn = np.zeros(mesh.E), np.zeros(mesh.N)
    return cases.Case("fan", mesh, p, st, lambda step, t: {"taux": ze + 0.05, "tauy": ze, "windx": zn, "windy": zn})


@pytest.mark.parametrize("columns", [0, 1])
def test_node_with_many_edges(built, columns):
    _compare(_fan, 4, columns)
