"""Training gradients at the sizes where the backward kernels' tiles, lanes and partial sums are ragged,
against the FP64 oracle; and several samples, which overlap, against the same samples one by one.

Bars: the ones of the gradient test (BF16 activations on both sides): loss 1e-3, every block of the
gradient within relative 5e-2. A sum over samples: FP32 additions in another order, 1e-5."""
import numpy as np
import pytest

from test_gpu_learned import _bf16_params, _rel
from test_gpu_setup import _wheels
from test_oracle_mpnn import node_graph

pytestmark = pytest.mark.gpu

BLOCKS = [0, 576, 576 + 8256, 576 + 2 * 8256, 576 + 3 * 8256, 25474]


def _system(pkg, mesh, fixed):
    D = pkg.constitutive_matrix(1.0, 0.3)
    K = pkg.build_stiffness_pattern(mesh)
    pkg.assemble_stiffness(mesh, D, 1.0, K)
    b = np.zeros(mesh.num_dofs)
    pkg.apply_dirichlet((fixed, np.zeros(fixed.size)), K, b)
    pkg.CgJacobiSolver().setup(K)
    return K, pkg.learned.node_material(D, mesh.num_nodes)


def _mesh(pkg, kind):
    if kind == "wheels":  # rows of 4 to 21 blocks, several pieces, each held at its rim
        xy, tri, hub = _wheels((3, 7, 8, 9, 20), 3)
        held = np.setdiff1d(np.arange(xy.size // 2, dtype=np.int32), hub)
        return pkg.plate.Mesh(xy=xy, triangles=tri, boundary_edges={}), np.sort(np.concatenate([2 * held, 2 * held + 1]))
    m = pkg.plate.quarter_plate(*kind)
    return m, pkg.plate.symmetry_dirichlet(m)[0]


@pytest.mark.parametrize("kind", [(1, 2), (7, 6), (6, 8), (8, 6), (12, 8), (8, 14), (15, 38), "wheels"])
def test_gradients_at_ragged_sizes(pkg, oracle, gpu_lib, kind):
    import torch
    mesh, fixed = _mesh(pkg, kind)
    K, mat = _system(pkg, mesh, fixed)
    p, q = _bf16_params(oracle, pkg, seed=9)
    pkg.learned.setup(K, p, mat)
    rp, cols, vals = K.download()
    n = mesh.num_dofs
    Kd = np.zeros((n, n))
    Kd[np.repeat(np.arange(n), np.diff(rp)), cols] = vals
    r = np.random.default_rng(n).standard_normal(n)
    e = np.linalg.solve(Kd, r)
    invd = 1.0 / np.diag(Kd)
    tr = pkg.learned.Trainer(p)
    loss = tr.accumulate(K, torch.from_numpy(r[None]).cuda(), torch.from_numpy(e[None]).cuda())
    g = tr.params(grads=True)[1]
    node_ptr, nbr = node_graph(rp, cols)
    X, s = oracle.mp_features(r, invd, mesh.xy, mat.astype(np.float64))
    Y, cache = oracle.mp_forward(node_ptr, nbr, X, q, q=True)
    L, dY = oracle.mp_loss(rp, cols, vals, r, e, invd, s, Y)
    g_ref = oracle.mp_backward(node_ptr, nbr, X, q, cache, dY, q=True)
    assert abs(loss[0] - L) < 1e-3 * max(1.0, abs(L))
    for a, c in zip(BLOCKS[:-1], BLOCKS[1:]):
        assert _rel(g[a:c], g_ref[a:c]) < 5e-2, (a, c)
    tr.close()
    K.ctx.close()


@pytest.mark.parametrize("mode", ["accumulate", "accumulate_cycle"])
@pytest.mark.parametrize("samples", [1, 2, 5])
def test_samples_together_and_one_by_one(pkg, oracle, gpu_lib, mode, samples):
    import torch
    mesh = pkg.plate.quarter_plate(20, 40)
    K, mat = _system(pkg, mesh, pkg.plate.symmetry_dirichlet(mesh)[0])
    p, _ = _bf16_params(oracle, pkg, seed=3)
    pkg.learned.setup(K, p, mat)
    E = torch.from_numpy(np.random.default_rng(2).standard_normal((samples, mesh.num_dofs))).cuda()
    R = torch.stack([K.multiply(e.contiguous()) for e in E])
    tr = pkg.learned.Trainer(p)
    losses = getattr(tr, mode)(K, R, E)
    g = tr.params(grads=True)[1]
    one, total = [], np.zeros(g.size)
    for k in range(samples):
        tr.zero_grad()
        one.append(getattr(tr, mode)(K, R[k:k + 1], E[k:k + 1])[0])
        total += tr.params(grads=True)[1]
    assert np.array_equal(losses, np.array(one))
    assert np.linalg.norm(g - total) <= 1e-5 * np.linalg.norm(total)
    tr.close()
    K.ctx.close()
