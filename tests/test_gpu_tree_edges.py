"""The hierarchy build at its launch edges: triangle counts around a tile of the level cuts and of a PLOC pass,
around the counts at which one block takes over the remaining levels and passes, and the smallest scenes, with
the smallest and the largest clusters. Object hierarchy and box tree equal the oracle's, bit for bit, and stay so
after a rebuild in place (rsh_scene_set_transforms)."""
import numpy as np
import pytest

import oracle
import rsh
from rsh import scenes

pytestmark = pytest.mark.gpu


def _check(sc, positions, cluster):
    lo, hi = sc.bounds()
    oh = oracle.ObjH(positions, cluster, lo, hi)
    order, tris, sph = oh.arrays()
    assert np.array_equal(sc.order(), order)
    levels = sc.levels()
    assert [len(l) for l in levels] == oh.levels()
    flat = np.concatenate([np.stack([l["c"][:, 0], l["c"][:, 1], l["c"][:, 2], l["radius"]], 1) for l in levels])
    assert flat.astype(np.float32).tobytes() == sph.tobytes()
    kids = oh.kids()
    for l in range(1, len(levels)):
        assert np.array_equal(np.append(levels[l]["first_child"], len(levels[l - 1])), kids[l])
    root, boxes, t = sc.box_tree()
    oroot, oboxes, ot = oh.box_tree()
    assert root == oroot and boxes.shape == oboxes.shape
    assert boxes[1:].tobytes() == oboxes[1:].tobytes() and t.tobytes() == ot.tobytes()


@pytest.mark.parametrize("cluster", [1, 6, 64])
@pytest.mark.parametrize("n", [1, 2, 7, 65, 255, 256, 257, 2047, 2048, 2049, 4095, 4097, 20_011])
def test_build_edges_bitexact(n, cluster):
    s = scenes.random_soup(max(n, 80) + 80, np.random.default_rng(n))
    pick = np.sort(np.random.default_rng(n + 1).permutation(s.tri_count)[:n])
    pos = np.ascontiguousarray(s.positions[pick])
    c = rsh.Context(rsh.default_config(cluster_size=cluster))
    sc = c.scene(pos, object_ids=(np.arange(n) % 3).astype(np.uint32))
    _check(sc, pos, cluster)
    for k in range(2):  # the second pose rebuilds over the first one's arrays
        m = np.tile(np.eye(4, dtype=np.float32), (3, 1, 1))
        m[1, :3, 3] = (0.25 + k, -0.5, 0.125)
        m[2, 0, 0] = -1.0
        sc.set_transforms(m)
        moved = sc.triangles()
        c.check_device_errors()
        _check(sc, moved, cluster)
    # identical triangles: every Morton code and every merged area ties
    same = c.scene(np.ascontiguousarray(np.repeat(pos[:1], n, axis=0)))
    _check(same, np.repeat(pos[:1], n, axis=0), cluster)
    c.check_device_errors()
    same.destroy()
    sc.destroy()
    c.destroy()
