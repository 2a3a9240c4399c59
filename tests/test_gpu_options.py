"""Solver options and media that take their own branches of the kernels, each
against the oracle: traces that stop once little is transmitted (TRANSMIN below
one: general traces, and the walk in the reference's order), no series
acceleration, every radiance term kept, the truncation fixed after some
iterations, and more phase functions than the 32 that a ray keeps values of.

States after 4 iterations of two FP32 solvers agree to the 1e-4 relative RMS
that the path is held to, and the truncations exactly; so do the renders.
"""
import numpy as np
import pytest

from at3d_gb300.scenes import cloud_blob, cloud_field, polarized_blob

pytestmark = pytest.mark.gpu


def relrms(a, b):
    a = np.asarray(a, np.float64); b = np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2)) / max(np.sqrt(np.mean(b ** 2)), 1e-30))


SCENES = {
    "field": lambda bc: cloud_field(seed=51, nx=12, ny=9, nz=8, nmu=8, nphi=16, nleg=64, boundary=bc),
    "blob": lambda bc: cloud_blob(seed=52, nx=9, ny=11, nz=7, boundary=bc),
    "polarized": lambda bc: polarized_blob(seed=53, nx=8, ny=9, nz=7, boundary=bc),
}
OPTIONS = {
    "transmin 0.9": dict(transmin=0.9),
    "transmin 0.3": dict(transmin=0.3),
    "no acceleration": dict(acceleration_flag=False),
    "high order": dict(high_order_radiance=True),
    "fixed truncation": dict(iterfixsh=2),
    "fixed truncation, high order": dict(iterfixsh=2, high_order_radiance=True),
}


def solve_both(pb, iters=4):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from at3d_gb300.solver import RTE
    from oracle.oracle import Oracle
    r = RTE.from_problem(pb)
    r.solve(iters, verbose=False)
    o = Oracle(pb, fp64=False)
    o.solve(iters)
    return r, o


@pytest.mark.parametrize("option", list(OPTIONS))
@pytest.mark.parametrize("boundary", ["open", "periodic"])
@pytest.mark.parametrize("scene", list(SCENES))
def test_options_match_oracle(scene, boundary, option):
    pb = SCENES[scene](boundary)
    for k, v in OPTIONS[option].items():
        setattr(pb.params, k, v)
    r, o = solve_both(pb)
    a, b = r.export_state(), o.export()
    r.close()
    assert np.array_equal(a["ns"], b["ns"]) and np.array_equal(a["nr"], b["nr"])
    for k in ("source", "radiance", "fluxes"):
        assert relrms(a[k], b[k]) < 1e-4, k


@pytest.mark.parametrize("transmin", [0.999, 0.5, 0.0])
def test_transmin_of_a_column(transmin):
    """One dimension, where the reference stops at the first point whatever TRANSMIN is."""
    pb = cloud_blob(seed=55, nx=1, ny=1, nz=9)
    pb.params.transmin = transmin
    r, o = solve_both(pb)
    a, b = r.export_state(), o.export()
    r.close()
    assert np.array_equal(a["ns"], b["ns"]) and np.array_equal(a["nr"], b["nr"])
    for k in ("source", "radiance", "fluxes"):
        assert relrms(a[k], b[k]) < 1e-4, k


@pytest.mark.parametrize("boundary", ["open", "periodic"])
@pytest.mark.parametrize("num_stokes", [1, 3])
@pytest.mark.parametrize("numphase", [32, 33, 45])
def test_render_of_many_phase_functions(numphase, num_stokes, boundary):
    """Phase functions spread over the points, more of them than a ray keeps
    the single-scatter values of, and just as many."""
    pb = (polarized_blob if num_stokes == 3 else cloud_blob)(seed=54, nx=8, ny=9, nz=7, boundary=boundary)
    s = pb.species[0]
    n = numphase - 1  # the other species' is the last
    rng = np.random.default_rng(numphase)
    leg = np.asarray(s.legcoef, np.float32)
    fade = (1.0 - 0.005 * np.arange(n))[:, None] ** np.arange(leg.shape[-1])[None, :]
    s.legcoef = (leg[None] * (fade[:, None] if num_stokes == 3 else fade)).astype(np.float32)
    s.table_index = rng.integers(1, n + 1, (1,) + pb.shape).astype(np.int32)
    s.phase_weights = np.ones((1,) + pb.shape, np.float32)
    r, o = solve_both(pb, 3)
    n = 40
    nx, ny, _ = pb.shape
    rays = ((rng.uniform(0.1, 0.9, n) * nx * pb.delx).astype(np.float32), (rng.uniform(0.1, 0.9, n) * ny * pb.dely).astype(np.float32),
            np.full(n, float(pb.zlevels[-1]), np.float32), rng.uniform(0.3, 1.0, n), rng.uniform(0.0, 6.0, n))
    assert relrms(r.render(*rays), o.render(*rays, nthreads=4)) < 1e-4
    r.close()
