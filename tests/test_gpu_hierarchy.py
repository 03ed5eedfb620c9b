"""The multigrid set-up where its kernels' groups are ragged: rows of more output blocks than lanes, few
rows, aggregates and levels of odd sizes, coarsest levels above and below the register inverse's size.

Bars: a V(2,2) cycle that interpolates the rigid modes is positive and takes well under 100 iterations; two
set-ups give the same bits."""
import numpy as np
import pytest

from test_gpu_setup import _wheels

pytestmark = pytest.mark.gpu


def _system(pkg, kind):
    if kind[0] == "wheels":  # rows of 4 to 31 blocks; every hub and one node of its rim held
        xy, tri, hub = _wheels(kind[1:], 5)
        mesh = pkg.plate.Mesh(xy=xy, triangles=tri, boundary_edges={})
        t = tri.reshape(-1, 3)
        rim = [next(int(v) for v in t[np.argmax((t == h).any(axis=1))] if v != h) for h in hub]
        held = np.concatenate([hub, rim])
        fixed = np.unique(np.concatenate([2 * held, 2 * held + 1])).astype(np.int32)
    else:
        mesh = pkg.plate.quarter_plate(*kind)
        fixed = pkg.plate.symmetry_dirichlet(mesh)[0]
    K = pkg.build_stiffness_pattern(mesh)
    pkg.assemble_stiffness(mesh, pkg.constitutive_matrix(1.0, 0.3), 1.0, K)
    b = np.zeros(mesh.num_dofs)
    pkg.apply_dirichlet((fixed, np.zeros(fixed.size)), K, b)
    s = pkg.CgJacobiSolver(pkg.SolverOptions(rtol=1e-10, max_iter=500, preconditioner="amg"))
    s.setup(K)
    return mesh, K, s


@pytest.mark.parametrize("kind", [(9, 12), (10, 10), (14, 22), (33, 34), (61, 90), (128, 130),
                                  ("wheels",) + (5, 8, 9, 16, 17, 20, 30) * 6])
def test_hierarchy_at_ragged_sizes(pkg, gpu_lib, kind):
    import torch
    out = []
    for _ in range(2):
        mesh, K, s = _system(pkg, kind)
        n = mesh.num_dofs
        rng = np.random.default_rng(n)
        r = torch.from_numpy(rng.standard_normal((2, n))).cuda()
        z = torch.stack([pkg.amg_apply(K, r[i].contiguous(), torch.empty_like(r[i])) for i in range(2)])
        x = np.zeros(n)
        st = s.solve(rng.standard_normal(n), x)
        out.append((z.cpu().numpy(), x))
        assert st.converged and st.iterations < 100
        assert float(z[0] @ r[0]) > 0 and float(z[1] @ r[1]) > 0
        K.ctx.close()
    assert all(np.array_equal(u, v) for u, v in zip(*out))
