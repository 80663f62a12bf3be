"""The direct branch where PCG stands in for the factor: states of the reference's
funnel scene (1,607 bodies; golden/funnel_states.npz, from trajectories of this
library) whose Newton systems are soft enough that stopping the PCG at a residual of
1e-13 |b| leaves velocities 7.6e-6 to 9.3e-6 away from the oracle's LDL^T.  The
oracle moves by 2e-7 there when its contacts are permuted; the bar is the one that the
scene's other checkpoints have, 1e-6."""
import os

import numpy as np
import pytest

import oracle_lib
from primal_dual_contacts_miror_b200 import abi
from test_gpu_reference_scenes import load

pytestmark = pytest.mark.gpu
STATES = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "funnel_states.npz")


@pytest.mark.parametrize("step", [150, 186])
def test_pcg_is_as_close_as_a_factor(step):
    from primal_dual_contacts_miror_b200 import lib

    sc, sim, cfg = load("funnel")
    dt, g = sim["timestep"], tuple(sim["gravity"])
    d = np.load(STATES)
    w = lib.World(abi.ShapeBatch([sc], dt, g), cfg=cfg, contacts_per_body=16)
    w.set_state(*(np.ascontiguousarray(d[f"{step}/{k}"]) for k in ("pos", "quat", "vel", "ang")))
    w.sync()
    hs = w.host_scene(0)
    w.close()
    dv, da, _, st = lib.Solver(cfg).solve(hs, dt=dt, gravity=g)
    odv, oda, _, ost = oracle_lib.solve(hs, dt=dt, gravity=g, cfg=cfg, nthreads=0)
    assert st["pcg_iters"] > 0 and st["factor_blocks"] == 0
    assert st["status"] == 0 and ost["status"] == 0 and st["newton_iters"] == ost["newton_iters"]
    v, ov = np.concatenate([dv, da], 1), np.concatenate([odv, oda], 1)
    assert np.abs(v - ov).max() / max(np.abs(ov).max(), 9.81 * dt) < 1e-6
