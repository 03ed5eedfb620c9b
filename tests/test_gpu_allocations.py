"""How often a new context's set-up and a new trainer's first pass allocate device memory: 23 and 20 times before
the set-up kept each node's place in its row and the diagonal, and the trainer two samples in flight. Large
allocations take 0.1 to 0.3 ms each, more than most kernels here. (Counted by torch's profiler in a process of
its own: a second session in one process may lose events.)"""
import json
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

CODE = """
import importlib, json, sys
import numpy as np, torch
from torch.profiler import ProfilerActivity, profile
pkg = importlib.import_module("mpi-cst-fem-solver_b200")
m, D, kept = pkg.plate.quarter_plate(40, 80), pkg.constitutive_matrix(1.0, 0.3), []

def set_up():
    ctx = pkg.Context()
    K = pkg.build_stiffness_pattern(m, ctx=ctx)
    pkg.assemble_stiffness(m, D, 1.0, K)
    pkg.apply_dirichlet(pkg.plate.symmetry_dirichlet(m), K, np.zeros(m.num_dofs))
    pkg.CgJacobiSolver().setup(K)
    kept.append(K)

set_up()
f = set_up
if sys.argv[1] == "trainer":
    K, w = kept[0], pkg.learned.load_weights(mode="cycle")
    pkg.learned.setup(K, w, pkg.learned.node_material(D, m.num_nodes))
    E = torch.from_numpy(np.random.default_rng(0).standard_normal((3, m.num_dofs))).cuda()
    R = torch.stack([K.multiply(e.contiguous()) for e in E])
    first, second = pkg.learned.Trainer(w), pkg.learned.Trainer(w)
    first.accumulate_cycle(K, R, E)  # (builds the hierarchy)
    f = lambda: second.accumulate_cycle(K, R, E)
torch.cuda.synchronize()
with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
    f()
    torch.cuda.synchronize()
print(json.dumps({e.key: e.count for e in p.key_averages() if e.key.startswith("cuda")}))
"""


@pytest.mark.parametrize("what,most", [("context", 23), ("trainer", 20)])
def test_allocations(pkg, gpu_lib, what, most):
    r = subprocess.run([sys.executable, "-c", CODE, what], capture_output=True, text=True, cwd=REPO, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    calls = json.loads(r.stdout.strip().splitlines()[-1])
    if "cudaLaunchKernel" not in calls:
        pytest.skip("the profiler records no calls of the runtime here")
    assert 0 < calls.get("cudaMalloc", 0) <= most, calls
