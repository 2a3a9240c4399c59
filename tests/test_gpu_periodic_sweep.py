"""The reference-order walk of periodic grids at the sizes where its runs and
windows can go wrong: rows much shorter and longer than a warp, odd row
counts, grids of less than one window and of several, layers larger than the
values kept in shared memory.

The walk sums the reference's own terms in FP32 (in scan order); the states
of two FP32 solvers after 2 iterations agree to the 1e-4 relative RMS that the
path is held to, and the truncations exactly.
"""
import numpy as np
import pytest

from at3d_gb300.scenes import cloud_blob, cloud_field, polarized_blob

pytestmark = pytest.mark.gpu


def relrms(a, b):
    a = np.asarray(a, np.float64); b = np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2)) / max(np.sqrt(np.mean(b ** 2)), 1e-30))


SCENES = {
    "3x4x5": lambda: cloud_blob(seed=1, nx=3, ny=4, nz=5, dx=0.05, dz=0.08),
    "10x33x9": lambda: cloud_field(seed=2, nx=10, ny=33, nz=9, nmu=8, nphi=16, nleg=64, boundary="periodic"),
    "31x7x12": lambda: cloud_blob(seed=3, nx=31, ny=7, nz=12, dx=0.03, dz=0.05),
    "100x80x4": lambda: cloud_field(seed=5, nx=100, ny=80, nz=4, nmu=6, nphi=12, nleg=64, boundary="periodic"),
    "12x9x7 polarized": lambda: polarized_blob(seed=6, nx=12, ny=9, nz=7),
}


@pytest.mark.parametrize("scene", list(SCENES))
def test_periodic_walk_matches_oracle(scene):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from at3d_gb300.solver import RTE
    from oracle.oracle import Oracle
    pb = SCENES[scene]()
    r = RTE.from_problem(pb)
    r.solve(2, verbose=False)
    a = r.export_state()
    r.close()
    o = Oracle(pb, fp64=False)
    o.solve(2)
    b = o.export()
    assert np.array_equal(a["ns"], b["ns"]) and np.array_equal(a["nr"], b["nr"])
    for k in ("source", "radiance", "fluxes"):
        assert relrms(a[k], b[k]) < 1e-4, k
