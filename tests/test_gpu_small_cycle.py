"""The learned cycle on matrices that are their own coarsest level (at most 200 DOFs, where the cycle's
fixed part is the dense solve) and on ones just above: solve and training step.

Bars: the solve stops at a true residual of 1e-10; with condition numbers below 1e5 the solution is within
1e-5 of the dense one. A sample's loss and gradient are finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [(3, 4), (7, 6), (11, 8), (12, 8), (31, 40)])
def test_cycle_on_small_systems(pkg, gpu_lib, kind):
    import torch
    mesh = pkg.plate.quarter_plate(*kind)
    D = pkg.constitutive_matrix(1.0, 0.3)
    K = pkg.build_stiffness_pattern(mesh)
    pkg.assemble_stiffness(mesh, D, 1.0, K)
    fixed = pkg.plate.symmetry_dirichlet(mesh)[0]
    b = np.zeros(mesh.num_dofs)
    pkg.apply_dirichlet((fixed, np.zeros(fixed.size)), K, b)
    opts = pkg.SolverOptions(rtol=1e-10, max_iter=1000, preconditioner="learned_mg", true_residual_stop=True)
    s = pkg.CgJacobiSolver(opts)
    s.setup(K)
    params = pkg.learned.load_weights(mode="cycle")
    pkg.learned.setup(K, params, pkg.learned.node_material(D, mesh.num_nodes))
    rp, cols, vals = K.download()
    n = mesh.num_dofs
    Kd = np.zeros((n, n))
    Kd[np.repeat(np.arange(n), np.diff(rp)), cols] = vals
    r = np.random.default_rng(n).standard_normal(n)
    e = np.linalg.solve(Kd, r)
    x = np.zeros(n)
    stats = s.solve(r, x)
    assert stats.converged
    assert np.linalg.norm(x - e) < 1e-5 * np.linalg.norm(e)
    tr = pkg.learned.Trainer(params)
    loss = tr.accumulate_cycle(K, torch.from_numpy(r[None]).cuda(), torch.from_numpy(e[None]).cuda())
    grads = tr.params(grads=True)[1]
    assert np.isfinite(loss[0])
    assert np.all(np.isfinite(grads))
