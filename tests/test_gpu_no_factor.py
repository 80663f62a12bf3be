"""sparse_max_bodies 0: every scene on PCG, with no factor and no shared memory for
one, from a handle, from a batch and from the allocation-free entry point.  The same
bits from all three, and within the repository's bar of 1e-9 of the factor's results on
these settled piles (both solve the linear systems to rounding; three iterations)."""
import ctypes as C

import numpy as np
import pytest

from primal_dual_contacts_miror_b200 import abi, scenes
from test_zz_no_alloc import DeviceScene, _bind

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 150])
def test_pcg_without_a_factor(n):
    import torch

    from primal_dual_contacts_miror_b200 import lib

    s = scenes.settled_pile(n, np.random.default_rng(n), vel_noise=0.002)
    kw = dict(max_iter=3)
    cfg = abi.default_config(sparse_max_bodies=0, **kw)
    solver = lib.Solver(cfg)
    one = solver.solve(s)
    assert one[3]["factor_blocks"] == 0 and one[3]["pcg_iters"] > 0
    b = solver.batch_solve(abi.HostBatch([s, s], 0.01, (0, 0, -9.81)))
    dev = DeviceScene(s)
    out, res = dev.outputs()
    L = _bind(lib.load())
    g = (C.c_double * 3)(0.0, 0.0, -9.81)
    assert L.pdc_solve_noalloc(C.byref(cfg), 0.01, g, C.byref(dev.bodies), C.byref(dev.contacts), C.byref(res), None,
                               None) == abi.PDC_OK
    torch.cuda.synchronize()
    ref = lib.Solver(abi.default_config(**kw)).solve(s)
    assert ref[3]["factor_blocks"] > 0 or n == 1
    for k in range(3):
        m = len(one[k])
        assert np.array_equal(one[k], b[k][:m]) and np.array_equal(one[k], b[k][m:])
        assert np.array_equal(one[k], out[k].cpu().numpy())
        assert np.abs(one[k] - ref[k]).max() <= 1e-9 * max(np.abs(ref[k]).max(), 0.0981 if k < 2 else 0.0)
