"""Angular resolutions beyond the usual ones, against the oracle.

More than 1,344 ordinates: the columns' weights of the points that do not
scatter take more than the default 48 KB of shared memory.

The states of two FP32 solvers after 2 iterations agree to the 1e-4 relative
RMS that the path is held to, and the truncations exactly.
"""
import numpy as np
import pytest

from at3d_gb300.scenes import cloud_field

pytestmark = pytest.mark.gpu


def relrms(a, b):
    a = np.asarray(a, np.float64); b = np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2)) / max(np.sqrt(np.mean(b ** 2)), 1e-30))


def check_state(pb, mode=None):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from at3d_gb300.solver import RTE
    from oracle.oracle import Oracle
    r = RTE.from_problem(pb)
    if mode:
        r.set_transform_mode(mode)
    r.solve(2, verbose=False)
    a = r.export_state()
    r.close()
    o = Oracle(pb, fp64=False)
    o.solve(2)
    b = o.export()
    assert np.array_equal(a["ns"], b["ns"]) and np.array_equal(a["nr"], b["nr"])
    for k in ("source", "radiance", "fluxes"):
        assert relrms(a[k], b[k]) < 1e-4, k


@pytest.mark.parametrize("boundary", ["open", "periodic"])
def test_sparse_field_beyond_1344_ordinates(boundary):
    pb = cloud_field(seed=31, nx=10, ny=9, nz=7, nmu=32, nphi=64, nleg=128, fraction=0.3, boundary=boundary)
    check_state(pb)
