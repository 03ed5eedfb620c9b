"""A limit on the waits between blocks holds for every solve of a mesh, small ones in the automatic launch mode
too, and takes no solve of a caller's CSR matrix down."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,n_t", [(20, 40), (40, 80), (100, 200)])
@pytest.mark.parametrize("launch", ["auto", "persistent"])
def test_mesh_solve_times_out(pkg, gpu_lib, launch, n_r, n_t):
    m = pkg.plate.quarter_plate(n_r, n_t)
    K = pkg.build_stiffness_pattern(m)
    pkg.assemble_stiffness(m, pkg.constitutive_matrix(1.0, 0.3), 1.0, K)
    b = np.zeros(m.num_dofs)
    pkg.add_traction(K, m.boundary_edges["right"], 1.0, 1.0, 0.0, b)
    pkg.apply_dirichlet(pkg.plate.symmetry_dirichlet(m), K, b)
    s = pkg.CgJacobiSolver(pkg.SolverOptions(launch=launch))
    s.setup(K)
    x = np.zeros(m.num_dofs)
    K.ctx.set_wait_limits(barrier_polls=0)
    with pytest.raises(pkg.CstgError) as ei:
        s.solve(b, x)
    assert ei.value.code == pkg.native.ERR_TIMEOUT
    K.ctx.set_wait_limits()
    assert s.solve(b, x).converged
    K.ctx.close()


@pytest.mark.parametrize("n", [4097, 40001])
def test_csr_solve_has_no_wait(pkg, gpu_lib, n):
    i = np.arange(n)
    cols = np.stack([i - 1, i, i + 1], axis=1)
    vals = np.stack([np.full(n, -1.0), np.full(n, 2.01), np.full(n, -1.0)], axis=1)
    ok = (cols >= 0) & (cols < n)
    rp = np.concatenate([[0], np.cumsum(ok.sum(axis=1))])
    K = pkg.GpuCsrMatrix.from_csr(rp, cols[ok], vals[ok])
    b = np.random.default_rng(n).standard_normal(n)
    x = [np.zeros(n), np.zeros(n)]
    s = pkg.CgJacobiSolver(pkg.SolverOptions(launch="graph"))
    s.setup(K)
    assert s.solve(b, x[0]).converged
    s = pkg.CgJacobiSolver(pkg.SolverOptions())
    s.setup(K)
    K.ctx.set_wait_limits(barrier_polls=0)
    assert s.solve(b, x[1]).converged
    assert np.array_equal(x[0], x[1])
    K.ctx.close()
