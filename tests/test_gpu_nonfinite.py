"""Elements that are not finite (a material matrix with an infinity or a NaN, a triangle so thin that its
strain matrix overflows): the assembled matrix holds the infinities and NaNs of the oracle in their places,
and the Jacobi set-up refuses what the oracle's diagonal refuses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    nan = np.isnan(b)
    return np.array_equal(np.isnan(a), nan) and np.array_equal(a[~nan].view(np.int64), b[~nan].view(np.int64))


def _check(pkg, oracle, xy, tri, D):
    mesh = pkg.plate.Mesh(xy=xy, triangles=tri, boundary_edges={})
    K = pkg.build_stiffness_pattern(mesh)
    rp, cols = oracle.build_stiffness_pattern(mesh.num_nodes, tri)
    with np.errstate(all="ignore"):
        vals = oracle.assemble_stiffness(xy, tri, D, 0.7, rp, cols)
    pkg.assemble_stiffness(mesh, D, 0.7, K)
    assert _same(K.download()[2], vals)
    diag = np.array([vals[rp[i] + np.searchsorted(cols[rp[i]:rp[i + 1]], i)] for i in range(rp.size - 1)])
    bad = ~(diag > 0.0)
    s = pkg.CgJacobiSolver()
    if bad.any():
        with pytest.raises(pkg.CstgError) as ei:
            s.setup(K)
        assert ei.value.code == pkg.native.ERR_NONPOSITIVE_DIAGONAL
        assert f"row {np.flatnonzero(bad)[0]}" in str(ei.value)
    else:
        s.setup(K)
    K.ctx.close()
    return bool(bad.any())


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e308])
def test_material(pkg, gpu_lib, oracle, value):
    m = pkg.plate.quarter_plate(3, 6)
    refused = []
    for k in range(9):
        D = np.array(pkg.constitutive_matrix(1.0, 0.3), dtype=np.float64).reshape(3, 3).copy()
        D.reshape(-1)[k] = value
        refused.append(_check(pkg, oracle, m.xy, np.ascontiguousarray(m.triangles).reshape(-1), D))
    if not np.isfinite(value):
        assert refused[0] and refused[1]  # D00 and D01 among them


@pytest.mark.parametrize("h", [1e-310, 1e-308, 1e-160])
def test_thin_triangles(pkg, gpu_lib, oracle, h):
    """One thin triangle beside an ordinary one, and a hub of ten (its rows are summed in place)."""
    xy = np.array([0.0, 0.0, 1.0, 0.0, 0.5, 1.0, 0.5, -h])
    tri = np.array([0, 1, 2, 0, 3, 1], dtype=np.int32)
    D = np.array(pkg.constitutive_matrix(1.0, 0.3), dtype=np.float64).reshape(3, 3)
    _check(pkg, oracle, xy, tri, D)
    t = 2.0 * np.pi * np.arange(10) / 10
    ring = np.stack([np.cos(t), np.sin(t)], axis=1)
    ring[1] = ring[0] + (0.0, h)
    xy = np.concatenate([[0.0, 0.0], ring.reshape(-1)])
    tri = np.array([(0, 1 + i, 1 + (i + 1) % 10) for i in range(10)], dtype=np.int32).reshape(-1)
    _check(pkg, oracle, xy, tri, D)
