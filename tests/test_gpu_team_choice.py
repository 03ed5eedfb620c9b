"""Which team of blocks solves a system, as the library reports it: a team whose blocks' shares do not fit
declines, and the next one takes the solve. The sizes on either side of each limit follow from what a block
keeps in its shared memory (231,424 bytes): FP64 in shared memory 320 bytes a node of an O-grid and 20 a
halo node (224 x 448 fits with room for 126 more halo nodes, 226 x 452 lacks 71), mixed 223 and 20 (268 x 536
fits with 80, 270 x 540 lacks 81). Numbered at random, 300 x 600 has 63 (FP64) and 415 (mixed) to spare in narrow
groups of rows, and 330 x 660 lacks more than 1,300. Their values are compared at convergence."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_teams import _both, _plate

pytestmark = pytest.mark.gpu

TEAMS = ["cluster", "resident", "stream", "narrow", "grid"]


def _teams(K):
    """The teams that the last solve was launched on, in order."""
    got, count = (C.c_int * 8)(), C.c_int(0)
    K.ctx.check(K.ctx.L.cstg_solve_teams(K.ctx.h, got, 8, C.byref(count)))
    return [TEAMS[t] for t in got[:count.value]]


def _check(pkg, K, b, want, **kw):
    s = pkg.CgJacobiSolver(pkg.SolverOptions(**kw))
    s.setup(K)
    s.solve(b)
    assert _teams(K) == want
    K.ctx.close()


@pytest.mark.parametrize("precision,n_r,n_t,want", [
    ("fp64", 54, 108, ["cluster"]), ("fp64", 55, 110, ["resident"]), ("fp64", 224, 448, ["resident"]),
    ("fp64", 226, 452, ["resident", "stream"]), ("fp64", 232, 464, ["stream"]), ("fp64", 590, 1770, ["narrow"]),
    ("mixed", 54, 108, ["cluster"]), ("mixed", 55, 110, ["resident"]), ("mixed", 268, 536, ["resident"]),
    ("mixed", 270, 540, ["resident", "stream"]), ("mixed", 276, 552, ["stream"]), ("mixed", 565, 1766, ["narrow"])])
def test_mesh(pkg, gpu_lib, precision, n_r, n_t, want):
    _check(pkg, *_plate(pkg, n_r, n_t), want, precision=precision, max_iter=200)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_small_mesh_without_the_cluster(pkg, gpu_lib, precision):
    _check(pkg, *_plate(pkg, 40, 80), ["resident"], launch="persistent", precision=precision, max_iter=200)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_r,n_t,want", [(300, 600, ["stream", "narrow"]), (330, 660, ["stream", "narrow", "grid"])])
def test_numbering_without_locality(pkg, gpu_lib, precision, n_r, n_t, want):
    _check(pkg, *_plate(pkg, n_r, n_t, "random"), want, precision=precision, max_iter=200)


def test_streamed_solve_after_its_switch(pkg, gpu_lib):
    _check(pkg, *_plate(pkg, 300, 600), ["stream", "grid"], precision="mixed", rtol=1e-12, max_iter=200000)


@pytest.mark.parametrize("n,want", [(12000, ["cluster"]), (12001, ["resident"])])
def test_csr(pkg, gpu_lib, n, want):
    i = np.arange(n)
    cols = np.stack([i - 1, i, i + 1], axis=1)
    vals = np.stack([np.full(n, -1.0), np.full(n, 2.01), np.full(n, -1.0)], axis=1)
    ok = (cols >= 0) & (cols < n)
    rp = np.concatenate([[0], np.cumsum(ok.sum(axis=1))])
    _check(pkg, pkg.GpuCsrMatrix.from_csr(rp, cols[ok], vals[ok]), np.random.default_rng(n).standard_normal(n), want)


def test_csr_with_a_long_row(pkg, gpu_lib):
    n = 3000
    rp = np.concatenate([[0, n], n + 2 * np.arange(1, n)])
    cols = np.concatenate([np.arange(n), np.stack([np.zeros(n - 1, int), np.arange(1, n)], axis=1).reshape(-1)])
    vals = np.concatenate([[2.0], np.full(n - 1, 0.01), np.tile([0.01, 1.0], n - 1)])
    _check(pkg, pkg.GpuCsrMatrix.from_csr(rp, cols, vals), np.random.default_rng(n).standard_normal(n), [])


@pytest.mark.parametrize("precision,n_r,n_t,numbering", [
    ("fp64", 224, 448, "ray"), ("fp64", 226, 452, "ray"), ("mixed", 268, 536, "ray"), ("mixed", 270, 540, "ray"),
    ("fp64", 590, 1770, "ray"), ("fp64", 330, 660, "random"), ("mixed", 330, 660, "random")])
def test_values_at_the_limits(pkg, gpu_lib, precision, n_r, n_t, numbering):
    """Against the captured kernels, to the bars of test_gpu_teams.py."""
    _both(pkg, *_plate(pkg, n_r, n_t, numbering), precision=precision)
