"""Timeouts in the middle of the network's pipeline: with a few polls a wait (2 us each) its roles stop at any tile.
Every application ends in time, with the right values or the timeout's status, and the next one with the
default limits gives the same bits as before."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,n_t", [(120, 240), (300, 700)])
def test_stops_in_the_middle(pkg, gpu_lib, n_r, n_t):
    import torch
    m = pkg.plate.quarter_plate(n_r, n_t)
    D = pkg.constitutive_matrix(1.0, 0.3)
    K = pkg.build_stiffness_pattern(m)
    pkg.assemble_stiffness(m, D, 1.0, K)
    b = np.zeros(m.num_dofs)
    pkg.apply_dirichlet(pkg.plate.symmetry_dirichlet(m), K, b)
    pkg.CgJacobiSolver().setup(K)
    pkg.learned.setup(K, pkg.learned.load_weights(), pkg.learned.node_material(D, m.num_nodes))
    r = torch.from_numpy(np.random.default_rng(0).standard_normal(m.num_dofs)).cuda()
    z = pkg.learned.apply(K, r).cpu().numpy()
    for polls in (1, 2, 3, 4, 6, 9, 14, 30):
        K.ctx.set_wait_limits(mma_polls=polls)
        t = time.perf_counter()
        try:
            assert np.array_equal(pkg.learned.apply(K, r).cpu().numpy(), z)
        except pkg.CstgError as e:
            assert e.code == pkg.native.ERR_TIMEOUT
        assert time.perf_counter() - t < 2.0
        K.ctx.set_wait_limits()
        assert np.array_equal(pkg.learned.apply(K, r).cpu().numpy(), z)
    K.ctx.close()
