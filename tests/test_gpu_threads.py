"""Handles used from several host threads at once: what they share (a grid's
device tables, the kernels' launch attributes) must not let one thread's call
change another's.  Results equal those of the same calls made one after
another, to the 1e-6 relative RMS of sums in another order."""
import threading

import numpy as np
import pytest

from at3d_gb300.scenes import cloud_field, polarized_blob

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


def run_threads(calls):
    """Runs the calls at once, one thread each; returns their results, or raises the first error."""
    out, errors, start = [None] * len(calls), [], threading.Barrier(len(calls))

    def work(i):
        try:
            start.wait()
            out[i] = calls[i]()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
    return out


@pytest.mark.parametrize("shape", [(21, 19, 11), (9, 30, 14)])
def test_handles_of_one_grid_created_at_once(rte_cls, shape):
    """The first handles on a grid, created and solved by several threads: each
    starts with the grid's tables complete, whoever built them."""
    nx, ny, nz = shape

    def solve(w, seed):
        pb = cloud_field(seed=seed, wavelength_index=w, nx=nx, ny=ny, nz=nz, nmu=8, nphi=16, nleg=64, boundary="open")
        r = rte_cls.from_problem(pb)
        r.solve(3, verbose=False)
        state = r.export_state()
        r.close()
        return state

    calls = [lambda w=w: solve(w, 40 + w) for w in range(4)]
    together = run_threads(calls)
    for a, call in zip(together, calls):
        b = call()
        assert np.array_equal(a["ns"], b["ns"])
        for k in ("radiance", "fluxes"):
            assert relrms(a[k], b[k]) < 1e-6, k


@pytest.mark.parametrize("kind", ["render", "render polarized", "gradient", "fp32 transforms"])
def test_calls_of_different_size_at_once(rte_cls, kind):
    """Renders, gradients and FP32 transforms need shared memory by their number
    of terms and rays, less or more than the default limit; threads that launch
    the same kernels with different needs must each get theirs, call after call."""
    rng = np.random.default_rng(5)
    handles, calls = [], []
    for nmu, nphi, nrays, ncalls in ((32, 32, 2500, 1000), (4, 8, 2, 2500), (32, 32, 3, 1500), (4, 8, 2, 2500)):
        kw = dict(seed=nmu, nx=7, ny=6, nz=6, nmu=nmu, nphi=nphi, boundary="open")
        pb = polarized_blob(**kw) if kind == "render polarized" else cloud_field(nleg=128, **kw)
        nx, ny, _ = pb.shape
        q = ((rng.uniform(0.1, 0.9, nrays) * nx * pb.delx).astype(np.float32),
             (rng.uniform(0.1, 0.9, nrays) * ny * pb.dely).astype(np.float32),
             np.full(nrays, float(pb.zlevels[-1]), np.float32), rng.uniform(0.5, 1.0, nrays), rng.uniform(0.0, 6.0, nrays))
        w = np.ones(nrays)
        r = rte_cls.from_problem(pb)
        if kind == "fp32 transforms":
            r.set_transform_mode("fp32")
            ncalls //= 25
        r.solve(1, verbose=False)
        handles.append(r)

        def call(r=r, q=q, w=w):
            if kind == "fp32 transforms":
                r.solve(2, verbose=False)
                return r.export_state()["fluxes"]
            return r.levis_adjoint(q, w) if kind == "gradient" else r.render(*q)

        def repeat(call=call, n=ncalls):
            first = call()
            return first, max(relrms(call(), first) for _ in range(n))
        calls.append((call, repeat))
    alone = [call() for call, _ in calls]
    for a, (first, spread) in zip(alone, run_threads([repeat for _, repeat in calls])):
        assert relrms(first, a) < 1e-6 and spread < 1e-6
    for r in handles:
        r.close()
