"""The row kernels of the source step (source function, truncations, series
acceleration, packed rows) at the row lengths where their split can go wrong:
fewer terms than lanes, lengths that leave lanes and passes partly empty, the
largest they take and the first they leave to the general kernels, with and
without points that do not scatter, scalar and I, Q, U.

Truncations are whole numbers and equal the oracle's; the fields are those of
two FP32 solvers after 3 iterations, held to the path's 1e-4 relative RMS.
"""
import numpy as np
import pytest

from at3d_gb300.scenes import cloud_blob, cloud_field, polarized_blob

pytestmark = pytest.mark.gpu


def relrms(a, b):
    a = np.asarray(a, np.float64); b = np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2)) / max(np.sqrt(np.mean(b ** 2)), 1e-30))


@pytest.mark.parametrize("kind,nmu", [("field", 4), ("field", 6), ("field", 10), ("field", 12), ("field", 14), ("field", 18),
                                      ("blob", 8), ("polarized", 6), ("polarized", 10), ("polarized", 12)])
def test_source_rows_match_oracle(kind, nmu):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from at3d_gb300.solver import RTE
    from oracle.oracle import Oracle
    kw = dict(seed=nmu, nx=11, ny=9, nz=10, boundary="open", nmu=nmu, nphi=2 * nmu)
    pb = (cloud_field(nleg=64, **kw) if kind == "field" else cloud_blob(**kw) if kind == "blob" else polarized_blob(**kw))
    r = RTE.from_problem(pb)
    r.solve(3, verbose=False)
    a = r.export_state()
    r.close()
    o = Oracle(pb, fp64=False)
    o.solve(3)
    b = o.export()
    assert np.array_equal(a["ns"], b["ns"]) and np.array_equal(a["nr"], b["nr"])
    for k in ("source", "radiance", "fluxes"):
        assert relrms(a[k], b[k]) < 1e-4, k
