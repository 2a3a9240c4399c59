"""Angular resolutions beyond the usual ones, against the oracle.

More than 1,344 ordinates: the columns' weights of the points that do not
scatter take more than the default 48 KB of shared memory.

More than 32 azimuthal modes (34 azimuths and up): more than a lane each in the
factorised transforms, which take the FP32 mode, rows of harmonics that are not
a multiple of four (NMU 18, NPHI 34: 322 terms) and grids of less than 128
points.

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


@pytest.mark.parametrize("nmu,nphi,shape,mode", [
    (16, 32, (9, 8, 7), "fp32"),    # 31 modes: one lane each
    (17, 34, (9, 8, 7), "fp32"),    # 33: one mode past a warp
    (18, 34, (9, 8, 7), None),      # by the rows' length, ordinates to harmonics on the tensor cores
    (18, 36, (9, 8, 7), "fp32"),
    (32, 64, (9, 8, 7), "fp32"),    # 63, the most there are
    (20, 40, (4, 5, 5), None),      # by the number of points
])
@pytest.mark.parametrize("boundary", ["open", "periodic"])
def test_more_than_32_azimuthal_modes(nmu, nphi, shape, mode, boundary):
    nx, ny, nz = shape
    check_state(cloud_field(seed=nmu + nphi, nx=nx, ny=ny, nz=nz, nmu=nmu, nphi=nphi, nleg=128, fraction=0.4,
                            boundary=boundary), mode)
