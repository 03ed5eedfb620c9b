"""The message-passing layer's gather plan where its forms meet: nodes with seven neighbours (a seventh
place per node), neighbours in the tile's own rows only, own rows between two runs, tiles whose other
rows are just more or fewer than a stage holds. The plan kernel and the row kernel sum the same neighbours
in the same order: the outputs have the same bits."""
import numpy as np
import pytest

from test_gpu_learned import _bf16_params
from test_gpu_setup import _wheels

pytestmark = pytest.mark.gpu


def _mesh(pkg, kind):
    if isinstance(kind, str):  # wheels of seven spokes, rims held (a lone one, a ragged last tile)
        xy, tri, hub = _wheels((7,) * int(kind), 3)
        held = np.setdiff1d(np.arange(xy.size // 2, dtype=np.int32), hub)
        return pkg.plate.Mesh(xy=xy, triangles=tri, boundary_edges={}), np.sort(np.concatenate([2 * held, 2 * held + 1]))
    n_r, n_t, window = kind
    m = pkg.plate.quarter_plate(n_r, n_t)
    fixed = pkg.plate.symmetry_dirichlet(m)[0]
    if window:  # the halves of every window swapped: a tile's neighbours lie further apart
        N = m.num_nodes
        n = np.arange(N)
        w = n // window * window
        perm = np.where(w + window <= N, w + (n - w + window // 2) % window, n)
        xy = np.empty((N, 2))
        xy[perm] = np.asarray(m.xy).reshape(-1, 2)
        tri = perm[np.asarray(m.triangles).reshape(-1, 3)].astype(np.int32)
        fixed = np.sort(2 * perm[fixed // 2] + fixed % 2).astype(np.int32)
        m = pkg.plate.Mesh(xy=xy.reshape(-1), triangles=tri.reshape(-1), boundary_edges={})
    return m, fixed


@pytest.mark.parametrize("kind", ["1", "16", "40", (9, 12, 0), (20, 126, 0), (20, 128, 0), (30, 254, 0),
                                  (30, 254, 64), (30, 254, 200), (30, 278, 280)])
def test_plan_and_rows_give_the_same_bits(pkg, oracle, gpu_lib, monkeypatch, kind):
    import torch
    D = pkg.constitutive_matrix(1.0, 0.3)
    mesh, fixed = _mesh(pkg, kind)
    p, _ = _bf16_params(oracle, pkg, seed=8)
    r = torch.from_numpy(np.random.default_rng(5).standard_normal(mesh.num_dofs)).cuda()
    out = []
    for rows in (False, True):
        if rows:
            monkeypatch.setenv("CSTG_MP_GATHER", "rows")
        else:
            monkeypatch.delenv("CSTG_MP_GATHER", raising=False)
        K = pkg.build_stiffness_pattern(mesh)
        pkg.assemble_stiffness(mesh, D, 1.0, K)
        b = np.zeros(mesh.num_dofs)
        pkg.apply_dirichlet((fixed, np.zeros(fixed.size)), K, b)
        pkg.CgJacobiSolver().setup(K)
        pkg.learned.setup(K, p, pkg.learned.node_material(D, mesh.num_nodes))
        out.append(pkg.learned.apply(K, r).cpu().numpy())
        K.ctx.close()
    assert np.array_equal(out[0], out[1])
