"""Rays on the lanes of a warp (render and Levis adjoint) at the counts and
mixtures where their split can go wrong: fewer rays than a warp or a block
takes, one more than a block, blocks of one direction and of many, rays that
start inside the medium and look up or down, rays of weight zero, rows of
harmonics that are not a multiple of four; and the ordinate-to-harmonic
transform with such rows; and a grid with more lines than fit on the chip.

Compared with the FP64 oracle on the state of 3 iterations (I, Q, U: the FP32
one), to the 1e-4 relative RMS that the solve, the render and the gradient
are held to.
"""
import numpy as np
import pytest

from at3d_gb300.scenes import cloud_blob, cloud_field, polarized_blob

pytestmark = pytest.mark.gpu


def relrms(a, b):
    a = np.asarray(a, np.float64); b = np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2)) / max(np.sqrt(np.mean(b ** 2)), 1e-300))


SCENES = {
    "blob open": lambda: cloud_blob(seed=11, nx=10, ny=13, nz=9, boundary="open"),
    "blob periodic 8x6": lambda: cloud_blob(seed=12, nx=9, ny=8, nz=11, nmu=8, nphi=6),
    "field open 10x10": lambda: cloud_field(seed=13, nx=12, ny=9, nz=8, nmu=10, nphi=10, nleg=64, boundary="open"),
    "polarized open": lambda: polarized_blob(seed=14, nx=9, ny=10, nz=8, boundary="open"),
}


def some_rays(pb, n, mixed):
    """n rays from inside the domain (both ways) and from its top (down the view), of one direction or of many."""
    rng = np.random.default_rng(n)
    nx, ny, _ = pb.shape
    top = float(pb.zlevels[-1])
    inside = rng.random(n) < 0.5
    x = rng.uniform(0.05, 0.9, n) * nx * pb.delx
    y = rng.uniform(0.05, 0.9, n) * ny * pb.dely
    z = np.where(inside, rng.uniform(0.1, 0.9, n) * top, top)
    mu = rng.uniform(0.2, 1.0, n) * np.where(inside & (rng.random(n) < 0.5), -1.0, 1.0)
    phi = rng.uniform(0.0, 2 * np.pi, n)
    if not mixed:
        mu[:], phi[:] = 0.7, 0.4
    return x.astype(np.float32), y.astype(np.float32), z.astype(np.float32), mu, phi


@pytest.fixture(scope="module", params=list(SCENES))
def solved(request):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from at3d_gb300.solver import RTE
    from oracle.oracle import Oracle
    pb = SCENES[request.param]()
    r = RTE.from_problem(pb)
    r.solve(3, verbose=False)
    o = Oracle(pb, fp64=pb.num_stokes == 1)
    o.solve(3)
    yield pb, r, o
    r.close()


def test_state_of_odd_rows(solved):
    pb, r, o = solved
    a, b = r.export_state(), o.export()
    for k in ("source", "radiance", "fluxes"):
        assert relrms(a[k], b[k]) < 1e-4, k


@pytest.mark.parametrize("n,mixed", [(1, True), (3, True), (5, False), (16, True), (17, False), (17, True), (131, True)])
def test_render_lanes(solved, n, mixed):
    pb, r, o = solved
    rays = some_rays(pb, n, mixed)
    assert relrms(r.render(*rays), o.render(*rays, nthreads=4)) < 1e-4


@pytest.mark.parametrize("n,mixed", [(1, True), (15, False), (17, True), (130, True)])
def test_adjoint_lanes(solved, n, mixed):
    pb, r, o = solved
    if pb.num_stokes > 1:
        pytest.skip("the gradient is of I")
    rays = some_rays(pb, n, mixed)
    w = np.random.default_rng(n + 1).standard_normal(n)
    w[::5] = 0.0
    if n == 1:
        w[:] = 1.0
    ga = r.levis_adjoint(rays, w)
    gb = o.levis_adjoint(0, rays, w, nthreads=4).reshape(ga.shape)
    for d in range(2):
        assert relrms(ga[..., d], gb[..., d]) < 1e-4, d


def test_render_of_a_grid_of_many_lines():
    """57,000 cells along x: the rays read the grid's lines from memory.  The
    rays stay near its start, where positions in FP32 are as fine as elsewhere."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from at3d_gb300.solver import RTE
    from oracle.oracle import Oracle
    pb = cloud_field(seed=15, nx=57000, ny=2, nz=3, nmu=4, nphi=8, nleg=128, boundary="open")
    near = cloud_field(seed=16, nx=20, ny=2, nz=3, nmu=4, nphi=8, nleg=128, boundary="open")
    pb.species[0].extinction[:20] = near.species[0].extinction
    r = RTE.from_problem(pb)
    r.solve(1, verbose=False)
    o = Oracle(pb, fp64=True)
    o.solve(1)
    rays = list(some_rays(near, 33, True))
    assert relrms(r.render(*rays), o.render(*rays, nthreads=4)) < 1e-4
    r.close()
