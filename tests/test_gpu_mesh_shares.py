"""Pairs of very different size in one mesh query: every pair gets blocks in
proportion to its triangle pairs, so a large one among many small ones costs little
more than alone, and the contacts are those of one query per pair, bit for bit."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def torus(around, tube, major=0.5, minor=0.1):
    a = np.arange(around)[:, None] * (2 * np.pi / around)
    t = np.arange(tube)[None, :] * (2 * np.pi / tube)
    r = major + minor * np.cos(t)
    verts = np.stack([r * np.cos(a), r * np.sin(a), minor * np.sin(t) + 0 * a], -1).reshape(-1, 3)
    i, j = (x.ravel() for x in np.meshgrid(np.arange(around), np.arange(tube), indexing="ij"))
    p = lambda x, y: (x % around) * tube + y % tube
    return verts, np.concatenate([np.stack([p(i, j), p(i + 1, j), p(i + 1, j + 1)], 1),
                                  np.stack([p(i, j), p(i + 1, j + 1), p(i, j + 1)], 1)])


def pairs(lib, around, tube, n, rng):
    v, f = torus(around, tube)
    a, b = lib.Mesh(v, f), lib.Mesh(1.001 * v, f)
    out = []
    for _ in range(n):
        q = np.array([0.0, 0.0, 0.1, 1.0]) + rng.normal(0, 0.02, 4)
        out.append((a, np.r_[0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0], b,
                    np.r_[0.05, 0.02, 0.03 + rng.uniform(0, 0.01), q / np.linalg.norm(q)]))
    return out


@pytest.mark.parametrize("order", ["large first", "large last", "large between"])
def test_large_pair_among_small_ones(order):
    from primal_dual_contacts_miror_b200 import lib

    rng = np.random.default_rng(7)
    large, small = pairs(lib, 200, 50, 1, rng), pairs(lib, 24, 10, 200, rng)
    at = {"large first": 0, "large last": 200, "large between": 77}[order]
    every = small[:at] + large + small[at:]

    def query(p):
        out = lib.mesh_contact_buffers(200 * len(p) + 4000)
        best = np.inf
        for _ in range(4):
            t = time.perf_counter()
            got = lib.mesh_contacts_pairs(p, out=out)
            best = min(best, time.perf_counter() - t)
        return best, np.array(got["counts"]), {k: out[k].copy() for k in ("pos", "normal", "depth", "frame", "arm")}

    t_large, _, _ = query(large)
    t_every, counts, rows = query(every)
    assert counts.min() > 0
    o = 0
    for k, p in enumerate(every):
        if k in (0, at - 1, at, at + 1, 100, 200):
            _, n, one = query([p])
            assert n[0] == counts[k]
            for f in rows:
                assert np.array_equal(rows[f][o:o + n[0]], one[f][:n[0]]), (k, f)
        o += counts[k]
    # 200 small pairs have 0.1 of the large one's triangle pairs: 1.1 to 1.5 times its
    # time as shared by size, 15 times with an equal share of blocks for every pair
    assert t_every < 4 * t_large, (t_every, t_large)
