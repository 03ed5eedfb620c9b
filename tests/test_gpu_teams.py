"""The persistent solve's teams of blocks against the per-phase kernels (launch="graph"), at the sizes
where the choice between them turns and where a block's share is ragged.

Both run the same recurrence and differ in the order of their sums only, so the bar is the one of
every solve here: converged under the same rule, iterations within 2 % (at least 2), displacements
within relative 1e-8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_TOL = 1e-8


def _plate(pkg, n_r, n_t, numbering="ray"):
    m = pkg.plate.quarter_plate(n_r, n_t)
    dofs, vals = pkg.plate.symmetry_dirichlet(m)
    edges = m.boundary_edges["right"]
    if numbering == "random":
        new = np.random.default_rng(n_r).permutation(m.num_nodes).astype(np.int32)
        xy = np.empty((m.num_nodes, 2))
        xy[new] = m.xy.reshape(-1, 2)
        m = pkg.plate.Mesh(xy=xy.reshape(-1), triangles=new[m.triangles], boundary_edges={})
        edges = new[edges]
        dofs = (2 * new[dofs // 2] + dofs % 2).astype(np.int32)
    K = pkg.build_stiffness_pattern(m)
    pkg.assemble_stiffness(m, pkg.constitutive_matrix(1.0, 0.3), 1.0, K)
    b = np.zeros(m.num_dofs)
    pkg.add_traction(K, np.ascontiguousarray(edges), 1.0, 1.0, 0.0, b)
    pkg.apply_dirichlet((dofs, vals), K, b)
    return K, b


def _both(pkg, K, b, launches=("graph", "auto"), **kw):
    out = []
    for launch in launches:
        s = pkg.CgJacobiSolver(pkg.SolverOptions(max_iter=200000, launch=launch, record_history=True, **kw))
        s.setup(K)
        x = np.zeros(b.size)
        out.append((s.solve(b, x), x))
    (sg, xg), rest = out[0], out[1:]
    for st, x in rest:
        assert st.converged and sg.converged, (st.message, sg.message)
        assert abs(st.iterations - sg.iterations) <= max(2, 0.02 * sg.iterations)
        assert np.linalg.norm(x - xg) <= REL_TOL * np.linalg.norm(xg)
        assert len(st.residual_history) == st.iterations + 1
    K.ctx.close()
    return [o[0] for o in out]


# one ray; a cluster's last and a grid team's first sizes; a block's threads and lanes just full and not;
# the last resident and the first streamed sizes; narrow groups of rows
@pytest.mark.parametrize("precision,n_r,n_t", [
    ("fp64", 1, 2), ("mixed", 1, 2), ("fp64", 16, 32), ("mixed", 54, 108), ("fp64", 55, 110), ("mixed", 137, 274),
    ("fp64", 241, 482), ("fp64", 245, 490), ("mixed", 270, 540), ("mixed", 276, 552), ("fp64", 480, 960)])
def test_mesh_teams(pkg, gpu_lib, precision, n_r, n_t):
    _both(pkg, *_plate(pkg, n_r, n_t), ("graph", "auto", "persistent"), precision=precision)


@pytest.mark.parametrize("precision,n_r,n_t", [("fp64", 40, 80), ("fp64", 180, 360), ("mixed", 180, 360),
                                                ("fp64", 300, 600), ("mixed", 300, 600)])
def test_numbering_without_locality(pkg, gpu_lib, precision, n_r, n_t):
    """Large halos; at 300 x 600 they do not fit, and the per-phase kernels take the solve."""
    _both(pkg, *_plate(pkg, n_r, n_t, "random"), precision=precision)


@pytest.mark.parametrize("n_r,n_t", [(40, 80), (300, 600)])
def test_precision_switch(pkg, gpu_lib, n_r, n_t):
    """An rtol below the FP32 operator's floor: a resident team goes on with the FP64 rows itself, a
    streaming one leaves the iteration to the per-phase kernels."""
    stats = _both(pkg, *_plate(pkg, n_r, n_t), precision="mixed", rtol=1e-12)
    assert "then FP64" in stats[-1].message, [st.message for st in stats]


def _csr(pkg, rp, cols, vals):
    n = len(rp) - 1
    b = np.random.default_rng(n).standard_normal(n)
    return pkg.GpuCsrMatrix.from_csr(rp, cols, vals), b


@pytest.mark.parametrize("n", [1, 2, 33, 4097, 12000, 12001, 40001])
def test_csr_teams(pkg, gpu_lib, n):
    """Tridiagonal rows (2, -1 and a small shift: SPD), every size a ragged share of some block."""
    i = np.arange(n)
    cols = np.stack([i - 1, i, i + 1], axis=1)
    vals = np.stack([np.full(n, -1.0), np.full(n, 2.01), np.full(n, -1.0)], axis=1)
    ok = (cols >= 0) & (cols < n)
    rp = np.concatenate([[0], np.cumsum(ok.sum(axis=1))])
    _both(pkg, *_csr(pkg, rp, cols[ok], vals[ok]))


def test_csr_with_a_long_row(pkg, gpu_lib):
    """An arrow matrix (its first row is full) stays on the per-phase kernels."""
    n = 3000
    rp = np.concatenate([[0, n], n + 2 * np.arange(1, n)])
    cols = np.concatenate([np.arange(n), np.stack([np.zeros(n - 1, int), np.arange(1, n)], axis=1).reshape(-1)])
    vals = np.concatenate([[2.0], np.full(n - 1, 0.01), np.tile([0.01, 1.0], n - 1)])
    _both(pkg, *_csr(pkg, rp, cols, vals))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n_cases,config", [(1, (1, 256)), (1, (4, 512)), (2, (1, 512)), (2, (2, 256)), (3, (1, 512)),
                                            (3, (16, 256)), (4, (1, 512)), (4, (2, 512)), (4, (8, 256))])
def test_batch_shapes(pkg, gpu_lib, precision, n_cases, config):
    """Batches whose largest plate's direction vectors fit a block and batches whose do not, against the
    single solve of every plate and case."""
    cases = dict(list(pkg.plate.LOAD_CASES.items())[:n_cases])
    specs = [pkg.plate.PlateSpec(n_r=n, n_theta=2 * n, a=1.0, E=1.0, nu=0.3, plane_strain=False)
             for n in (3, 24, 40, 61, 84)]
    batch = pkg.build_batch(specs, cases=cases)
    solver = pkg.BatchSolver(pkg.SolverOptions(precision=precision, max_iter=200000))
    solver.setup(batch)
    sol = solver.solve(config=config)
    assert sol.converged.all() and (sol.true_rel_residual <= 1e-10).all()
    solver.close()
    for s, spec in enumerate(specs):
        m = pkg.plate.quarter_plate(spec.n_r, spec.n_theta)
        K = pkg.build_stiffness_pattern(m)
        for q, parts in enumerate(cases.values()):
            pkg.assemble_stiffness(m, pkg.constitutive_matrix(1.0, 0.3), 1.0, K)
            b = np.zeros(m.num_dofs)
            for group, tx, ty in parts:
                pkg.add_traction(K, m.boundary_edges[group], 1.0, tx, ty, b)
            pkg.apply_dirichlet(pkg.plate.symmetry_dirichlet(m), K, b)
            one = pkg.CgJacobiSolver(pkg.SolverOptions(precision=precision, max_iter=200000, true_residual_stop=True))
            one.setup(K)
            x = np.zeros(b.size)
            st = one.solve(b, x)
            assert st.converged
            assert abs(sol.iterations[s, q] - st.iterations) <= max(2, 0.02 * st.iterations)
            assert np.linalg.norm(sol.x[q, batch.dof_range(s)] - x) <= REL_TOL * np.linalg.norm(x)
        K.ctx.close()
