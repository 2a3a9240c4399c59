"""The strip march of the open-boundary sweep and the ordinate-major fields
around it, at the sizes where the split can go wrong: grids of a few cells,
row counts that leave remainders in the strips and in a thread's rows, layer
counts that are and are not multiples of four, several CTAs per column, and
both transform paths on the same fields.

The march, the level schedule and the oracle form the same cell integrals in
FP32; a radiance is a chain of at most (planes) such steps whose weights sum
to at most one, so rounding differences grow at most linearly: 1e-5 relative
RMS covers 100 planes of 1e-7 each.
"""
import numpy as np
import pytest

from at3d_gb300.scenes import cloud_blob, cloud_field, polarized_blob

pytestmark = pytest.mark.gpu


def relrms(a, b):
    a = np.asarray(a, np.float64); b = np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2)) / max(np.sqrt(np.mean(b ** 2)), 1e-30))


@pytest.fixture(scope="module")
def rte_cls():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from at3d_gb300.solver import RTE
    return RTE


SCENES = {
    "3x3x3": lambda: cloud_blob(seed=1, nx=3, ny=3, nz=3, dx=0.05, dz=0.08, boundary="open"),
    "5x9x4": lambda: cloud_blob(seed=2, nx=5, ny=9, nz=4, dx=0.05, dz=0.08, boundary="open"),
    "17x6x13": lambda: cloud_field(seed=3, nx=17, ny=6, nz=13, nmu=8, nphi=16, nleg=64),
    "40x31x22": lambda: cloud_field(seed=4, nx=40, ny=31, nz=22, nmu=8, nphi=16, nleg=64),
    "9x70x8 nmu 12": lambda: cloud_field(seed=5, nx=9, ny=70, nz=8, nmu=12, nphi=24, nleg=64),
    "67x5x37": lambda: cloud_field(seed=6, nx=67, ny=5, nz=37, nmu=8, nphi=16, nleg=64),
    "11x13x9 polarized": lambda: polarized_blob(seed=7, nx=11, ny=13, nz=9, boundary="open"),
}


@pytest.mark.parametrize("scene", list(SCENES))
def test_march_matches_levels_and_oracle(rte_cls, scene):
    from oracle.oracle import Oracle
    pb = SCENES[scene]()
    r = rte_cls.from_problem(pb)
    marches = r.sizes["march"] == 3
    r.solve(2, verbose=False)
    a = r.export_state()
    r.set_sweep_mode("levels_only")
    assert r.sizes["march"] == 0
    r.solve(2, verbose=False)
    b = r.export_state()
    r.close()
    for k in ("radiance", "fluxes"):
        assert relrms(a[k], b[k]) < 1e-5, k
    assert marches or scene == "3x3x3"
    o = Oracle(pb, fp64=False)
    o.solve(2)
    c = o.export()
    assert np.array_equal(a["ns"], c["ns"]) and np.array_equal(a["nr"], c["nr"])
    assert relrms(a["radiance"], c["radiance"]) < 1e-4
    assert relrms(a["fluxes"], c["fluxes"]) < 1e-4


@pytest.mark.parametrize("scene", ["5x9x4", "17x6x13", "11x13x9 polarized"])
def test_cuda_core_transforms_on_ordinate_major_fields(rte_cls, scene):
    """Switching the transform arithmetic on one handle: the FP32 CUDA-core
    transforms work on transposed copies of the ordinate-major fields."""
    pb = SCENES[scene]()
    r = rte_cls.from_problem(pb)
    r.solve(2, verbose=False)
    a = r.export_state()
    r.set_transform_mode("fp32")
    r.solve(2, verbose=False)
    b = r.export_state()
    r.close()
    assert relrms(a["radiance"], b["radiance"]) < 1e-4
    assert relrms(a["fluxes"], b["fluxes"]) < 1e-5


PLANES = {  # planes beyond what the deepest staging holds, and rows beyond a thread per position
    "200x200x5": dict(nx=200, ny=200, nz=5),     # z class: one group of layers
    "246x246x6": dict(nx=246, ny=246, nz=6),     # z class: single planes
    "100x300x7": dict(nx=100, ny=300, nz=7),     # z class: positions along x
    "1010x4x64": dict(nx=1010, ny=4, nz=64),     # y class: single planes
    "5x6x600": dict(nx=5, ny=6, nz=600),         # x and y classes: more than 512 positions
}


@pytest.mark.parametrize("shape", list(PLANES))
def test_march_of_large_planes(rte_cls, shape):
    """Grids that march although their planes are large, with a column split
    over several CTAs, so that rows go from one to the next."""
    from oracle.oracle import Oracle
    pb = cloud_field(seed=8, nmu=6, nphi=12, nleg=128, boundary="open", **PLANES[shape])
    r = rte_cls.from_problem(pb)
    s = r.sizes
    assert s["march"] == 3
    assert shape == "5x6x600" or (s["march_cluster_down"] > 1 and s["march_cluster_up"] > 1)
    r.solve(2, verbose=False)
    a = r.export_state()
    r.set_sweep_mode("levels_only")
    r.solve(2, verbose=False)
    b = r.export_state()
    r.close()
    for k in ("radiance", "fluxes"):
        assert relrms(a[k], b[k]) < 1e-5, k
    o = Oracle(pb, fp64=False)
    o.solve(2)
    c = o.export()
    assert np.array_equal(a["ns"], c["ns"]) and np.array_equal(a["nr"], c["nr"])
    for k in ("radiance", "fluxes"):
        assert relrms(a[k], c[k]) < 1e-4, k
