"""The block teams' sparse factor at the edges of its layouts: factors that just
fit and just miss the shared memory of a block (200 blocks of 6x6 with 256
threads, 80 with 128, two of them scratch), short and long update lists, warp
teams, and a contact graph whose lists outgrow their room.  Three Newton
iterations against the oracle's LDL^T: the linear systems are solved to about
2^-53 times their condition (up to 1e6 in these scenes), and three iterations
do not yet amplify that, so the repository's bar of 1e-9 holds with room."""
import numpy as np
import pytest

import mmd_ref
import oracle_lib
from primal_dual_contacts_miror_b200 import abi, scenes

pytestmark = pytest.mark.gpu


def rel(a, b, floor=1e-300):
    return np.abs(a - b).max() / max(np.abs(b).max(), floor) if a.size else 0.0


def clump(n, rng):
    """n spheres that nearly all touch one another: a graph so dense that its
    factor has n (n - 1) / 2 blocks."""
    sb = scenes.SceneBuilder()
    g = sb.add_ground()
    ids = [sb.add_body(tuple(rng.uniform(-1, 1, 3)), float(rng.uniform(1, 2)), (0.1, 0.1, 0.1),
                       vel=tuple(rng.uniform(-0.1, 0.1, 3))) for _ in range(n)]
    for i in range(n):
        for j in range(i + 1, n):
            if (i + j) % 3 == 0 or j == i + 1:
                nrm = rng.normal(size=3)
                sb.add_contact(ids[i], ids[j], tuple(rng.uniform(-1, 1, 3)), tuple(nrm / np.linalg.norm(nrm)))
    sb.add_contact(g, ids[0], (0.0, 0.0, -1.0), (0.0, 0.0, 1.0))
    return sb.build()


def build(kind, n):
    rng = np.random.default_rng(17 + (sum(n) if isinstance(n, tuple) else n))
    if kind == "pile":
        return scenes.settled_pile(n, rng, vel_noise=0.01)
    if kind == "crate":
        return scenes.packed_lattice(*n, rng)
    return clump(n, rng)


CASES = [("pile", n) for n in (1, 2, 31, 32, 33, 43, 44, 45, 110, 111, 112, 113, 240)] + \
        [("crate", d) for d in ((2, 2, 2), (3, 3, 2), (3, 3, 3), (4, 4, 2), (4, 4, 3), (6, 6, 4))] + \
        [("clump", n) for n in (12, 18, 19, 60, 190)]


@pytest.mark.parametrize("threads", [256, 128])
@pytest.mark.parametrize("kind,n", CASES)
def test_factor_layouts(kind, n, threads):
    from primal_dual_contacts_miror_b200 import lib

    s = build(kind, n)
    cfg = abi.default_config(max_iter=3, cta_threads=threads, grid_min_bodies=0)
    dv, da, lf, st = lib.Solver(cfg).solve(s)
    odv, oda, olf, ost = oracle_lib.solve(s, cfg=cfg)
    assert st["newton_iters"] == ost["newton_iters"]
    assert st["factor_blocks"] == mmd_ref.factor_blocks_strict(mmd_ref.active_graph(s.body, s.is_static))
    assert rel(lf, olf) < 1e-9
    assert rel(np.concatenate([dv, da], 1), np.concatenate([odv, oda], 1), 0.0981) < 1e-9


def test_teams_of_one_batch_agree():
    """The same small scenes alone (a block each) and many at once (a warp
    each): the oracle's results from both."""
    from primal_dual_contacts_miror_b200 import lib

    cfg = abi.default_config(max_iter=3)
    few = scenes.pile_batch(8, seed=3, n_min=1, n_max=8)
    many = few * 300
    for sc in (few, many):
        b = abi.HostBatch(sc, 0.01, (0, 0, -9.81))
        dv, da, lf, st = lib.Solver(cfg).batch_solve(b)
        odv, oda, olf, ost = oracle_lib.batch_solve(abi.HostBatch(few, 0.01, (0, 0, -9.81)), cfg=cfg)
        k = len(olf)
        assert rel(lf[:k], olf) < 1e-9 and rel(lf[-k:], olf) < 1e-9
        o = np.concatenate([odv, oda], 1)
        v = np.concatenate([dv, da], 1)
        assert rel(v[:len(o)], o, 0.0981) < 1e-9 and rel(v[-len(o):], o, 0.0981) < 1e-9
