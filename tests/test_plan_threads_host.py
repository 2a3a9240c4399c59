"""The planner's host threads: where no more can be started, their share of the
work runs in the caller's, and no error leaves a thread (which would end the
process)."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import resource, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from at3d_gb300.scenes import cloud_blob
from at3d_gb300.solver import HostPlan
pb = cloud_blob(nx=32, ny=32, nz=24)
want = HostPlan(pb).sizes
# the grid is planned (and kept); the next plan's threads ask for 1 GB of stack each
size = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (size + (600 << 20), resource.RLIM_INFINITY))
pb.species[0].extinction = np.asarray(pb.species[0].extinction) * np.float32(1.5)
assert HostPlan(pb).sizes == want
print("planned")
"""


def test_plan_without_threads():
    import resource

    def stack():
        hard = resource.getrlimit(resource.RLIMIT_STACK)[1]
        want = 1 << 30
        resource.setrlimit(resource.RLIMIT_STACK, (want if hard == resource.RLIM_INFINITY else min(want, hard), hard))

    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, preexec_fn=stack, timeout=300)
    assert r.returncode == 0 and "planned" in r.stdout, r.stderr[-2000:]
