"""What a handle has done before, and has under way, does not change what comes after.

Modes changed on a handle that has already solved: the calls that follow
equal those of a handle that had the mode from the start (to the 1e-6 relative
RMS of sums in another order; the transform arithmetics themselves differ by
1e-5 and more).  A solve that starts while images of the last one are being
rendered on the caller's streams leaves those images as they are."""
import numpy as np
import pytest

from at3d_gb300.scenes import cloud_blob, cloud_field

pytestmark = pytest.mark.gpu


def relrms(a, b):
    a = np.asarray(a, np.float64); b = np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2)) / max(np.sqrt(np.mean(b ** 2)), 1e-300))


@pytest.fixture(scope="module")
def rte_cls():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from at3d_gb300.solver import RTE
    return RTE


SCENES = {
    "open": lambda: cloud_field(seed=71, nx=11, ny=9, nz=8, nmu=8, nphi=16, nleg=64, boundary="open"),
    "periodic": lambda: cloud_blob(seed=72, nx=9, ny=8, nz=7),
}


def solved(r, iters=3):
    r.solve(iters, verbose=False)
    return r.export_state()["radiance"]


@pytest.mark.parametrize("scene", list(SCENES))
def test_transform_mode_after_a_captured_iteration(rte_cls, scene):
    """An iteration replayed from a graph is captured again for another transform arithmetic."""
    pb = SCENES[scene]()
    r = rte_cls.from_problem(pb)
    r.set_sweep_mode("graph")
    got = {}
    for mode in ("tf32", "fp32", "tf32x3"):
        r.set_transform_mode(mode)
        got[mode] = solved(r)
    r.close()
    for mode, a in got.items():
        r = rte_cls.from_problem(pb)
        r.set_transform_mode(mode)
        b = solved(r)
        r.close()
        assert relrms(a, b) < 1e-6, mode
    assert relrms(got["tf32"], got["fp32"]) > 1e-5


def test_solve_while_images_render(rte_cls):
    import torch
    from at3d_gb300.scenes import orthographic_views
    pb = cloud_field(seed=73, nx=48, ny=48, nz=24, nmu=8, nphi=16, nleg=64, boundary="open")
    r = rte_cls.from_problem(pb)
    r.solve(4, verbose=False)
    rays = [torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float32 if i < 3 else torch.float64).cuda()
            for i, v in enumerate(orthographic_views(pb, 96, 96))]
    n = rays[0].numel()

    def render(stream):
        out = torch.zeros(n, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        r.render_device(*(v.data_ptr() for v in rays), out.data_ptr(), n, stream.cuda_stream)
        return out

    streams = [torch.cuda.Stream() for _ in range(2)] + [torch.cuda.default_stream()]
    want = render(streams[0])
    torch.cuda.synchronize()
    want = want.cpu().numpy()
    for _ in range(3):
        for s in streams:
            r.solve(4, verbose=False)
            got = render(s)
            r.solve(1, verbose=False)  # resets the solution while the image is on its way
            torch.cuda.synchronize()
            assert relrms(got.cpu().numpy(), want) < 1e-6
    r.close()


@pytest.mark.parametrize("transforms", ["tf32x3", "fp32"])
@pytest.mark.parametrize("kind", ["field", "blob", "polarized", "RPV surface"])
def test_level_schedule_and_back(rte_cls, kind, transforms):
    """The plane march switched off and on between calls: the fields' layout
    turns, and the radiances at the surface and the top go along (to the 1e-5
    relative RMS of the march against the levels)."""
    from at3d_gb300.scenes import polarized_blob
    kw = dict(seed=74, nx=11, ny=10, nz=9, boundary="open")
    pb = polarized_blob(**kw) if kind == "polarized" else cloud_blob(**kw) if kind == "blob" else cloud_field(nmu=8, nphi=16, nleg=64, **kw)
    pb.skyrad = 0.05
    if kind == "RPV surface":
        pb.surface_brdf, pb.surface_params, pb.surface_delx, pb.surface_dely = "R", np.tile(np.float32([0.1, 0.8, -0.1]), (2, 2, 1)), 1.0, 1.0
    rng = np.random.default_rng(9)
    n = 20
    rays = ((rng.uniform(0.1, 0.9, n) * 11 * pb.delx).astype(np.float32), (rng.uniform(0.1, 0.9, n) * 10 * pb.dely).astype(np.float32),
            np.full(n, float(pb.zlevels[-1]), np.float32), rng.uniform(0.3, 1.0, n), rng.uniform(0.0, 6.0, n))
    r, q = rte_cls.from_problem(pb), rte_cls.from_problem(pb)
    for h in (r, q):
        h.set_transform_mode(transforms)
        h.solve(2, verbose=False)
    image = r.render(*rays)
    for step, mode in enumerate(("levels_only", "persistent", "levels_only", "graph")):
        r.set_sweep_mode(mode)
        assert r.sizes["march"] == (0 if mode == "levels_only" else 3)
        assert relrms(r.render(*rays), image) < 1e-6  # the surface's radiances are where they were
        for h in (r, q):
            h.solve(3 + step, init_solution=False, verbose=False)
        a, b = r.export_state(), q.export_state()
        for k in ("radiance", "fluxes"):
            assert relrms(a[k], b[k]) < 1e-5, (k, mode)
        image = r.render(*rays)
        assert relrms(image, q.render(*rays)) < 1e-5
    r.close()
    q.close()
