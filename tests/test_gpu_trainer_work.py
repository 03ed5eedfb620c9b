"""The trainer's work arrays: their bytes a node on either side of the size up to which two samples are in flight;
the gradients above it; and the same bits from the smaller arrays that a full GPU leaves room for."""
import numpy as np
import pytest

from test_gpu_backward import BLOCKS, _system
from test_gpu_learned import _bf16_params, _rel
from test_oracle_mpnn import node_graph

pytestmark = pytest.mark.gpu

PARTIAL_SUMS = 4 * 148 * (64 * 128 + 64) * 4


def _samples(K, mesh, count):
    import torch
    E = torch.from_numpy(np.random.default_rng(5).standard_normal((count, mesh.num_dofs))).cuda()
    return torch.stack([K.multiply(e.contiguous()) for e in E]), E


@pytest.mark.parametrize("n_r,n_t,samples,per_node", [(128, 256, 2, 4440), (400, 500, 2, 3136)])
def test_bytes(pkg, oracle, gpu_lib, n_r, n_t, samples, per_node):
    import torch
    mesh = pkg.plate.quarter_plate(n_r, n_t)
    K, mat = _system(pkg, mesh, pkg.plate.symmetry_dirichlet(mesh)[0])
    p, _ = _bf16_params(oracle, pkg, seed=3)
    pkg.learned.setup(K, p, mat)
    R, E = _samples(K, mesh, samples)
    taken = []
    for _ in range(2):  # (the first pass loads the kernels)
        tr = pkg.learned.Trainer(p)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        tr.accumulate(K, R, E)
        taken.append(free - torch.cuda.mem_get_info()[0])
        tr.close()
    assert taken[1] <= per_node * mesh.num_nodes + PARTIAL_SUMS + (8 << 20), taken  # (2 MB pages and small arrays)
    K.ctx.close()


@pytest.mark.parametrize("n_r,n_t", [(128, 256), (400, 500)])
def test_same_bits_on_a_full_gpu(pkg, oracle, gpu_lib, n_r, n_t):
    import torch
    mesh = pkg.plate.quarter_plate(n_r, n_t)
    K, mat = _system(pkg, mesh, pkg.plate.symmetry_dirichlet(mesh)[0])
    p, _ = _bf16_params(oracle, pkg, seed=3)
    pkg.learned.setup(K, p, mat)
    R, E = _samples(K, mesh, 3)
    torch.cuda.empty_cache()

    def train():
        tr = pkg.learned.Trainer(p)
        free = torch.cuda.mem_get_info()[0]
        losses = tr.accumulate(K, R, E)
        taken = free - torch.cuda.mem_get_info()[0]
        again = tr.accumulate(K, R, E)
        assert np.array_equal(losses, again)
        grads = tr.params(grads=True)[1]
        tr.close()
        return losses, grads, taken

    losses, grads, taken = train()
    lean = 2368 * mesh.num_nodes + PARTIAL_SUMS + (8 << 20)
    assert lean < taken
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (lean + taken) // 2, dtype=torch.uint8, device="cuda")
    losses_f, grads_f, taken_f = train()
    del filler
    torch.cuda.empty_cache()
    assert taken_f <= lean
    assert np.array_equal(losses, losses_f) and np.array_equal(grads, grads_f)
    K.ctx.close()


def test_gradients_above_the_limit(pkg, oracle, gpu_lib):
    mesh = pkg.plate.quarter_plate(400, 500)
    assert mesh.num_nodes > 200000
    K, mat = _system(pkg, mesh, pkg.plate.symmetry_dirichlet(mesh)[0])
    p, q = _bf16_params(oracle, pkg, seed=9)
    pkg.learned.setup(K, p, mat)
    R, E = _samples(K, mesh, 2)
    tr = pkg.learned.Trainer(p)
    both = tr.accumulate(K, R, E)
    g2 = tr.params(grads=True)[1]
    tr.zero_grad()
    assert tr.accumulate(K, R[1:], E[1:])[0] == both[1]
    g1 = tr.params(grads=True)[1]
    tr.zero_grad()
    loss = tr.accumulate(K, R[:1], E[:1])
    g = tr.params(grads=True)[1]
    assert loss[0] == both[0] and _rel(g2, g + g1) < 1e-5
    rp, cols, vals = K.download()
    r, e = R[0].cpu().numpy(), E[0].cpu().numpy()
    rows = np.repeat(np.arange(mesh.num_dofs), np.diff(rp))
    invd = 1.0 / vals[rows == cols]
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
