"""The count of kernel launches with several threads at work: a thread's captured launches are its own."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plate(pkg, ctx=None):
    m = pkg.plate.quarter_plate(12, 24)
    K = pkg.build_stiffness_pattern(m, ctx=ctx)
    pkg.assemble_stiffness(m, pkg.constitutive_matrix(1.0, 0.3), 1.0, K)
    b = np.zeros(m.num_dofs)
    pkg.add_traction(K, m.boundary_edges["right"], 1.0, 1.0, 0.0, b)
    pkg.apply_dirichlet(pkg.plate.symmetry_dirichlet(m), K, b)
    pkg.CgJacobiSolver().setup(K)
    return m, K, b


def _batch(pkg, batch):
    s = pkg.BatchSolver(pkg.SolverOptions(precision="mixed"))
    s.setup(batch, device_rhs=True)
    for _ in range(4):  # captures, then replays
        assert s.solve(device=True).converged.all()
    s.close()


def _cycles(pkg):
    _, K, b = _plate(pkg)
    s = pkg.CgJacobiSolver(pkg.SolverOptions(preconditioner="amg", true_residual_stop=True))
    s.setup(K)
    for _ in range(3):
        assert s.solve(b, np.zeros_like(b)).converged
    K.ctx.close()


def test_threads_count_apart(pkg, gpu_lib):
    count = lambda: gpu_lib.cstg_kernel_launches()
    specs = [pkg.plate.PlateSpec(n_r=n, n_theta=2 * n, a=1.0, E=1.0, nu=0.3, plane_strain=False) for n in (6, 8, 10)]
    batch = pkg.build_batch(specs)
    m, K, _ = _plate(pkg)
    x = np.ones(m.num_dofs)
    works = [lambda: _batch(pkg, batch), lambda: _cycles(pkg)]
    each = []
    for w in works:
        w()
        before = count()
        w()
        each.append(count() - before)
    before = count()
    K.multiply(x)
    product = count() - before
    rounds, products, stop = 12, [0], threading.Event()

    def other():
        while not stop.is_set():
            K.multiply(x)
            products[0] += 1

    before = count()
    t = threading.Thread(target=other)
    t.start()
    try:
        for _ in range(rounds):
            for w in works:
                w()
    finally:
        stop.set()
        t.join()
    assert products[0] > 100
    assert count() - before == rounds * sum(each) + products[0] * product
    K.ctx.close()
