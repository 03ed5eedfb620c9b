"""Pattern, assembly, elimination and Jacobi diagonal at the neighbourhood sizes where a kernel changes its
way: wheels of k triangles around one node (k + 1 blocks in its row), against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _wheels(spokes, copies):
    """`copies` wheels of every spoke count, side by side, in a shuffled numbering."""
    xy, tri, hub = [], [], []
    rng = np.random.default_rng(len(spokes))
    for c in range(copies):
        for k in spokes:
            base = len(xy)
            t = 2 * np.pi * (np.arange(k) + 0.2 * rng.random(k)) / k
            hub.append(base)
            xy += [(3.0 * len(hub), 0.1)] + [(3.0 * len(hub) + np.cos(a), 0.1 + np.sin(a)) for a in t]
            tri += [(base, base + 1 + i, base + 1 + (i + 1) % k) for i in range(k)]
    new = rng.permutation(len(xy)).astype(np.int32)
    out = np.empty((len(xy), 2))
    out[new] = xy
    return out.reshape(-1), new[np.array(tri, dtype=np.int32)].reshape(-1), new[hub]


@pytest.mark.parametrize("spokes,copies", [((3, 4, 5, 6, 7), 60), ((7, 8), 20), ((8, 9, 15), 9), ((15, 16, 17), 5),
                                           ((62, 3), 1)])
def test_wheels_vs_oracle(pkg, gpu_lib, oracle, spokes, copies):
    xy, tri, hub = _wheels(spokes, copies)
    mesh = pkg.plate.Mesh(xy=xy, triangles=tri, boundary_edges={})
    D = pkg.constitutive_matrix(2.1, 0.27, 1)
    K = pkg.build_stiffness_pattern(mesh)
    pkg.assemble_stiffness(mesh, D, 0.7, K)
    rp, cols, vals = K.download()
    rp_o, cols_o = oracle.build_stiffness_pattern(mesh.num_nodes, tri)
    vals_o = oracle.assemble_stiffness(xy, tri, D, 0.7, rp_o, cols_o)
    assert np.array_equal(rp, rp_o) and np.array_equal(cols, cols_o)
    assert np.array_equal(vals.view(np.int64), vals_o.view(np.int64))
    # some hubs and rim nodes prescribed, with nonzero values
    rng = np.random.default_rng(1)
    fixed = np.unique(np.concatenate([2 * hub[::2], 2 * hub[1::2] + 1,
                                      rng.integers(0, mesh.num_dofs, 5)])).astype(np.int32)
    ubar = rng.standard_normal(fixed.size)
    b = rng.standard_normal(mesh.num_dofs)
    b_o = b.copy()
    pkg.apply_dirichlet((fixed, ubar), K, b)
    oracle.apply_dirichlet(rp_o, cols_o, vals_o, fixed, ubar, b_o)
    assert np.array_equal(K.download()[2].view(np.int64), vals_o.view(np.int64))
    assert np.array_equal(b.view(np.int64), b_o.view(np.int64))
    # the Jacobi diagonal: one step from r = b is D^-1 b up to a factor
    s = pkg.CgJacobiSolver(pkg.SolverOptions(max_iter=1, launch="graph"))
    s.setup(K)
    s.solve(b)
    diag = np.array([vals_o[rp_o[i] + np.searchsorted(cols_o[rp_o[i]:rp_o[i + 1]], i)] for i in range(b.size)])
    z = b / diag
    alpha = (b @ z) / (z @ oracle.multiply(rp_o, cols_o, vals_o, z))
    assert np.linalg.norm(s.x - alpha * z) <= 1e-12 * np.linalg.norm(s.x)
    K.ctx.close()
