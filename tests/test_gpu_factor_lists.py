"""The block and warp teams' sparse factor where its update lists leave the room
behind the blocks (each product's partners are then found from the row patterns)
and where a scene is solved by a warp, on levels of short and of long lists; what
a case reaches is counted from the reference ordering.  Three Newton iterations
against the oracle's LDL^T at the repository's bar of 1e-9, as for the other
layouts of the factor: linear systems solved to about 2^-53 times their condition
(up to 1e6 here)."""
import numpy as np
import pytest

import mmd_ref
import oracle_lib
from primal_dual_contacts_miror_b200 import abi, scenes

NODES = 256                                  # of a factor
BLOCK_TEAM, WARP_TEAM = 32640, 64 * 63 // 2  # off-diagonal blocks of a team's slot
SHORT = 4                                    # longest list of a level done row by row


def graph_scene(n, touch, seed):
    """n bodies at random positions, a contact at a random point of every pair that
    `touch` names, one contact with the ground."""
    rng = np.random.default_rng(seed)
    sb = scenes.SceneBuilder()
    g = sb.add_ground()
    ids = [sb.add_body(tuple(rng.uniform(-1, 1, 3)), float(rng.uniform(1, 2)), (0.1, 0.1, 0.1),
                       vel=tuple(rng.uniform(-0.1, 0.1, 3))) for _ in range(n)]
    for i in range(n):
        for j in range(i + 1, n):
            if touch(i, j):
                nrm = rng.normal(size=3)
                sb.add_contact(ids[i], ids[j], tuple(rng.uniform(-1, 1, 3)), tuple(nrm / np.linalg.norm(nrm)))
    sb.add_contact(g, ids[0], (0.0, 0.0, -1.0), (0.0, 0.0, 1.0))
    return sb.build()


def complete(n):
    return graph_scene(n, lambda i, j: True, n)


def thirds(n):
    return graph_scene(n, lambda i, j: (i + j) % 3 == 0 or j == i + 1, n)


def lists(scene, slot):
    """Blocks of the scene's factor (diagonal ones too), whether its update lists fit
    the slot when the blocks are there as well, and the longest list."""
    perm, pattern = mmd_ref.symbolic_strict(mmd_ref.active_graph(scene.body, scene.is_static))
    row = {v: set() for v in perm}
    for d in perm:
        for u in pattern[d]:
            row[u].add(d)
    lens = [len(row[k] & row[u]) for k in perm for u in (k, *pattern[k])]
    room = 288 * (slot + NODES - (len(lens) + 2))
    return len(lens), 4 * sum((n + 1) // 2 * 2 for n in lens) <= room, max(lens)


def rel(a, b, floor=1e-300):
    return np.abs(a - b).max() / max(np.abs(b).max(), floor) if a.size else 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [256, 128])
@pytest.mark.parametrize("kind,n", [(complete, 184), (complete, 190), (thirds, 255)])
def test_lists_beyond_their_room(kind, n, threads):
    from primal_dual_contacts_miror_b200 import lib

    s = kind(n)
    blocks, fits, _ = lists(s, BLOCK_TEAM)
    assert fits == (n == 184)
    cfg = abi.default_config(max_iter=3, cta_threads=threads, grid_min_bodies=0)
    dv, da, lf, st = lib.Solver(cfg).solve(s)
    odv, oda, olf, ost = oracle_lib.solve(s, cfg=cfg, nthreads=0)
    assert st["factor_blocks"] == blocks - n and st["newton_iters"] == ost["newton_iters"]
    assert rel(lf, olf) < 1e-9
    assert rel(np.concatenate([dv, da], 1), np.concatenate([odv, oda], 1), 0.0981) < 1e-9


@pytest.mark.gpu
def test_warp_teams():
    """A batch on warps and the same batch on thread blocks: the oracle's results from
    both.  Piles (short lists), crates (long ones), complete graphs (lists that do not
    fit a warp's slot, at the largest scene that a warp takes)."""
    from primal_dual_contacts_miror_b200 import lib

    rng = np.random.default_rng(3)
    few = [scenes.settled_pile(n, rng, vel_noise=0.01) for n in (1, 2, 7, 31, 33, 63)]
    few += [scenes.packed_lattice(*d, rng) for d in ((2, 2, 2), (3, 3, 3), (4, 4, 3), (7, 3, 3))]
    few += [complete(n) for n in (5, 40, 63)]
    info = [lists(s, WARP_TEAM) for s in few]
    assert any(fits and longest > SHORT for _, fits, longest in info)
    assert any(longest <= SHORT for _, _, longest in info) and not info[-1][1]
    b = abi.HostBatch(few * 3, 0.01, (0, 0, -9.81))
    odv, oda, olf, _ = oracle_lib.batch_solve(abi.HostBatch(few, 0.01, (0, 0, -9.81)),
                                              cfg=abi.default_config(max_iter=3))
    o = np.concatenate([odv, oda], 1)
    for team in (1, 0):
        cfg = abi.default_config(max_iter=3, warp_max_contacts=4096 * team, warp_max_bodies=64 * team)
        dv, da, lf, st = lib.Solver(cfg).batch_solve(b)
        assert [s["team"] for s in st] == [team] * len(st)
        assert [s["factor_blocks"] for s in st] == [i[0] - s.n_bodies + 1 for i, s in zip(info, few)] * 3
        v = np.concatenate([dv, da], 1)
        for k in range(3):
            b0, b1 = 0, 0
            for q, s in enumerate(few):  # scene by scene: each against its own largest value
                a0, a1 = b0, b1
                b0, b1 = b0 + s.n_bodies, b1 + s.n_contacts
                assert rel(lf[k * len(olf) + a1:k * len(olf) + b1], olf[a1:b1]) < 1e-9, (team, q)
                assert rel(v[k * len(o) + a0:k * len(o) + b0], o[a0:b0], 0.0981) < 1e-9, (team, q)


@pytest.mark.gpu
def test_warp_slots_hold_factors_of_64():
    """Device memory of a call with warp teams: a warp's slot has room for the blocks,
    descriptors and lists of 64 bodies, no more than 0.92 MB (it once held descriptors
    for every block of a 256-body factor, 1.23 MB); with 64 MB for everything else."""
    import torch

    from primal_dual_contacts_miror_b200 import lib

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    grid = 2 * sms  # blocks in flight, eight warps each
    b = abi.HostBatch([scenes.settled_pile(2, np.random.default_rng(0))] * grid, 0.01, (0, 0, -9.81))
    solver = lib.Solver(abi.default_config(warp_max_contacts=64, warp_max_bodies=64))
    free = torch.cuda.mem_get_info()[0]
    st = solver.batch_solve(b)[3]
    used = free - torch.cuda.mem_get_info()[0]
    assert all(s["team"] == 1 for s in st)
    assert used < grid * (10.1e6 + 8 * 0.92e6) + 64e6, used
