"""How often a new context's set-up and a new trainer's first pass allocate device memory: 23 and 20 times before
the set-up kept each node's place in its row and the diagonal, and the trainer two samples in flight. Large
allocations take 0.1 to 0.3 ms each, more than most kernels here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _allocations(f):
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    calls = {e.key: e.count for e in p.key_averages()}
    if not any(k.startswith("cudaLaunchKernel") for k in calls):
        pytest.skip("the profiler records no calls of the runtime here")
    return calls.get("cudaMalloc", 0)


def test_allocations(pkg, gpu_lib):
    import torch
    m = pkg.plate.quarter_plate(40, 80)
    D = pkg.constitutive_matrix(1.0, 0.3)
    kept = []

    def set_up():
        ctx = pkg.Context()
        K = pkg.build_stiffness_pattern(m, ctx=ctx)
        pkg.assemble_stiffness(m, D, 1.0, K)
        b = np.zeros(m.num_dofs)
        pkg.apply_dirichlet(pkg.plate.symmetry_dirichlet(m), K, b)
        pkg.CgJacobiSolver().setup(K)
        kept.append(K)

    set_up()
    assert 0 < _allocations(set_up) <= 23
    K = kept[0]
    w = pkg.learned.load_weights(mode="cycle")
    pkg.learned.setup(K, w, pkg.learned.node_material(D, m.num_nodes))
    E = torch.from_numpy(np.random.default_rng(0).standard_normal((3, m.num_dofs))).cuda()
    R = torch.stack([K.multiply(e.contiguous()) for e in E])
    first, second = pkg.learned.Trainer(w), pkg.learned.Trainer(w)
    first.accumulate_cycle(K, R, E)  # (builds the hierarchy)
    assert 0 < _allocations(lambda: second.accumulate_cycle(K, R, E)) <= 20
    for t in (first, second):
        t.close()
    for k in kept:
        k.ctx.close()
