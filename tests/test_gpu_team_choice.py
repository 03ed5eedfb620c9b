"""Which team of blocks solves a system, read from the kernels that ran: a team whose blocks' shares do not fit
declines, and the next one takes the solve. The sizes on either side of each limit follow from what a block
keeps in its shared memory (231,424 bytes): FP64 in shared memory 320 bytes a node of an O-grid and 20 a
halo node (224 x 448 fits with room for 126 more halo nodes, 226 x 452 lacks 71), mixed 223 and 20 (268 x 536
fits with 80, 270 x 540 lacks 81). Numbered at random, 300 x 600 has 63 (FP64) and 415 (mixed) to spare in narrow
groups of rows, and 330 x 660 lacks more than 1,300. Their values are compared at convergence."""
import re

import numpy as np
import pytest

from test_gpu_teams import _both, _plate

pytestmark = pytest.mark.gpu

TEAMS = {("true", "true", 256): "cluster", ("false", "true", 256): "resident", ("0", 384): "stream", ("0", 256): "narrow",
         ("1", 1): "stream", ("1", 2): "narrow"}


def _teams(f):
    """The teams launched by f, in order."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    kernels = sorted((e.time_range.start, e.name) for e in p.events() if "k_" in e.name and "cstg" in e.name)
    if not kernels:
        pytest.skip("the profiler records no kernels here")
    out = []
    for _, name in kernels:
        if "k_pcg_grid" in name:
            out.append("grid")
        m = re.search(r"k_pcg_persistent<([^>]*)>", name)
        if m:
            op, cluster, resident, lanes, threads = (re.sub(r"\(\w+\)", "", a).strip() for a in m[1].split(","))
            op, cluster, resident = op[-1], {"1": "true", "0": "false"}.get(cluster, cluster), \
                {"1": "true", "0": "false"}.get(resident, resident)
            key = (cluster, resident, int(threads)) if resident == "true" else (op, int(threads) if op == "0" else int(lanes))
            out.append(TEAMS[key])
    return out


def _check(pkg, K, b, want, **kw):
    s = pkg.CgJacobiSolver(pkg.SolverOptions(**kw))
    s.setup(K)
    assert _teams(lambda: s.solve(b)) == want
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
