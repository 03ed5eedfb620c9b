"""Batches whose rows of one warp differ in length: every plate's nodes numbered at random, so rows of 3 to 7
blocks meet in a group of 32, with a ragged last group. Against the same batch in its own numbering.

Bar: both stop at an FP64 true residual of 1e-10; with condition numbers below 1e5 the solutions agree to
1e-5 (the rounding differs with the numbering)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _renumbered(batch, seed):
    """The batch with every plate's nodes numbered at random, and new[old node]."""
    rng = np.random.default_rng(seed)
    o = batch.node_offsets
    new = np.concatenate([o[s] + rng.permutation(o[s + 1] - o[s]) for s in range(batch.n_plates)]).astype(np.int32)
    dof = np.stack([2 * new, 2 * new + 1], 1).reshape(-1)
    xy = np.empty_like(batch.mesh.xy)
    xy[dof] = batch.mesh.xy
    loads = np.empty_like(batch.loads)
    loads[:, dof] = batch.loads
    d, v = batch.dirichlet
    at = np.argsort(dof[d])
    mesh = dataclasses.replace(batch.mesh, xy=xy, triangles=new[batch.mesh.triangles], boundary_edges={})
    return dataclasses.replace(batch, mesh=mesh, loads=loads,
                               dirichlet=(dof[d][at].astype(np.int32), np.asarray(v)[at])), dof


@pytest.mark.parametrize("precision,n_cases,config", [("mixed", 4, (2, 512)), ("mixed", 3, (1, 256)),
                                                      ("mixed", 1, (4, 512)), ("fp64", 2, (2, 512))])
def test_rows_of_mixed_lengths(pkg, gpu_lib, precision, n_cases, config):
    cases = dict(list(pkg.plate.LOAD_CASES.items())[:n_cases])
    specs = [pkg.plate.PlateSpec(n_r=n, n_theta=m, a=1.0, E=1.0, nu=0.3, plane_strain=False)
             for n, m in ((1, 2), (4, 6), (9, 14), (13, 22), (20, 30))]
    batch = pkg.build_batch(specs, cases=cases)
    other, dof = _renumbered(batch, 3)
    x = []
    for b in (batch, other):
        solver = pkg.BatchSolver(pkg.SolverOptions(precision=precision, max_iter=200000))
        solver.setup(b)
        sol = solver.solve(config=config)
        assert sol.converged.all() and (sol.true_rel_residual <= 1e-10).all()
        x.append(np.asarray(sol.x))
        solver.close()
    back = x[1][:, dof]
    for s in range(batch.n_plates):
        for q in range(n_cases):
            a, c = x[0][q, batch.dof_range(s)], back[q, batch.dof_range(s)]
            assert np.linalg.norm(a - c) <= 1e-5 * np.linalg.norm(a)
