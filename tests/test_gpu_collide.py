"""Contact generation at the edges of its kernels' tiles: the per-scene kernel
around its rounds of 128 threads and 512 bodies of shared memory, the sort-based
sweep around its tiles of 256 bodies, against the numpy restatement.  The two do
the same arithmetic on coordinates of order 1, a few hundred operations in 64
bits: 1e-12."""
import numpy as np
import pytest

import world_ref
from primal_dual_contacts_miror_b200 import abi, scenes

pytestmark = pytest.mark.gpu


def scene(n, seed):
    """n bodies: a plane, then boxes and spheres (every 7th static) in a volume
    that grows with n, so that the number of neighbours stays the same."""
    rng = np.random.default_rng(seed)
    sb = scenes.ShapeSceneBuilder()
    sb.add_plane((0.0, 0.0, 0.0), "+z")
    side = 0.35 * max(n, 1) ** (1 / 3)
    for k in range(1, n):
        pos = tuple(rng.uniform([-side, -side, 0.0], [side, side, 2 * side]))
        if k % 3:
            sb.add_box(tuple(rng.uniform(0.05, 0.2, 3)), pos, quat=tuple(scenes.random_quat(rng)), static=k % 7 == 0)
        else:
            sb.add_sphere(float(rng.uniform(0.05, 0.2)), pos)
    return sb.build()


def check(got, counts, shapes):
    o = 0
    for k, s in enumerate(shapes):
        ref = world_ref.npr.collide(s["type"], s["size"], s["pos"], s["quat"], s["is_static"])
        assert counts[k] == len(ref), (k, counts[k], len(ref))
        for q, c in enumerate(ref):
            assert tuple(got["body"][o + q]) == c["body"]
            np.testing.assert_allclose(got["pos"][o + q], c["pos"], atol=1e-12)
            np.testing.assert_allclose(got["frame"][o + q], c["frame"].reshape(-1), atol=1e-12)
            np.testing.assert_allclose(got["arm"][o + q], c["arm"], atol=1e-12)
            assert got["depth"][o + q] == pytest.approx(c["depth"], abs=1e-12)
        o += counts[k]


def collide(shapes, gmin, cpb=24):
    from primal_dual_contacts_miror_b200 import lib

    w = lib.World(abi.ShapeBatch(shapes, 0.01, (0, 0, -9.81)), cfg=abi.default_config(grid_min_bodies=gmin),
                  contacts_per_body=cpb)
    w.collide()
    counts, got = w.contacts()
    dropped = np.array(w.stats()[1])
    w.close()
    return counts, got, dropped


@pytest.mark.parametrize("large", [False, True])
@pytest.mark.parametrize("sizes", [(1, 2, 3, 16, 17, 32, 33), (129, 255), (256, 257, 100)])
def test_scene_sizes(sizes, large):
    shapes = [scene(n, 100 + n) for n in sizes]
    counts, got, _ = collide(shapes, 2 if large else 0)
    check(got, counts, shapes)


@pytest.mark.parametrize("sizes", [(511, 512, 513), (900, 256, 770)])
def test_paths_agree(sizes):
    """Bit for bit the same contacts from the per-scene kernel and the sort-based
    path, several large scenes of different sizes in one world."""
    shapes = [scene(n, 100 + n) for n in sizes]
    (ca, a, _), (cb, b, _) = collide(shapes, 0), collide(shapes, 2)
    assert np.array_equal(ca, cb) and ca.sum() > 300
    for k in ("body", "frame", "arm", "depth", "pos"):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("gmin", [0, 2])
def test_contacts_beyond_the_capacity_are_counted(gmin):
    """One contact per body (and the 16 that every scene gets) of room for a stack of
    boxes with four contacts per interface: the first contacts in order stay, the
    rest are counted as dropped."""
    sb = scenes.ShapeSceneBuilder()
    sb.add_plane((0.0, 0.0, 0.0), "+z")
    for k in range(40):
        sb.add_box((0.1, 0.1, 0.1), (0.0, 0.0, 0.0999 + 0.1998 * k))
    s = sb.build()
    full, every, none = collide([s], gmin, 8)
    cut, first, dropped = collide([s], gmin, 1)
    assert none[0] == 0 and full[0] == 160
    assert cut[0] == 41 + 16 and dropped[0] == full[0] - cut[0]
    for k in ("body", "frame", "arm", "depth", "pos"):
        assert np.array_equal(first[k][:57], every[k][:57]), k
