"""Handles used from several host threads at once: what they share (a grid's
device tables, the kernels' launch attributes) must not let one thread's call
change another's.  Results equal those of the same calls made one after
another, to the 1e-6 relative RMS of sums in another order."""
import threading

import numpy as np
import pytest

from at3d_gb300.scenes import cloud_field

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
