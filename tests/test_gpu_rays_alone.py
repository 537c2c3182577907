"""Single rays from the root of the box tree (k_fused_rays on one segment), the plain path's form at
plain_ray_level >= 1: hit records and shadow flags equal brute force over every triangle, exactly, at the sizes
where a launch can go wrong -- fewer rays than a warp, one more or less than a work unit, empty slots among them,
trees of one level and of several, the largest clusters -- with shared and with sequential launch ends, sorted
and unsorted (RSH_FLAG_RAH)."""
import numpy as np
import pytest

import oracle
import rsh
from rsh import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, rsh.FLAG_SEQUENTIAL_RAYS, rsh.FLAG_RAH])
@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("tris,cluster,level", [(80, 64, 1), (80, 1, 15), (12_000, 6, 2), (12_000, 64, 4)])
def test_trace_rays_alone_vs_brute(tris, cluster, level, any_hit, flags):
    c = rsh.Context(rsh.default_config(cluster_size=cluster, plain_ray_level=level, flags=flags))
    s = scenes.random_soup(tris, np.random.default_rng(tris + cluster))
    sc = c.scene(s.positions, s.normals, s.material_ids, s.materials)
    rng = np.random.default_rng(11)
    for n in (1, 31, 63, 64, 65, 4097, 30_011):
        rays = scenes.surface_rays(s, n, rng)
        if any_hit:
            rays["tmax"] = rng.uniform(0.05, 15.0, n).astype(np.float32)
        rays["tmax"][5::7] = -1.0
        assert np.array_equal(c.trace(sc, rays, any_hit), oracle.brute(s.positions, rays, any_hit)), n
    rays["tmax"] = -1.0  # no ray at all
    out = c.trace(sc, rays, any_hit)
    assert np.all(out == (0 if any_hit else rsh.HIT_NONE))
    c.check_device_errors()
    sc.destroy()
    c.destroy()


def test_trace_rays_alone_empty_scene():
    c = rsh.Context(rsh.default_config())
    sc = c.scene(np.zeros((0, 3, 4), np.float32))
    s = scenes.random_soup(80, np.random.default_rng(1))
    rays = scenes.surface_rays(s, 100, np.random.default_rng(2))
    assert np.all(c.trace(sc, rays, True) == 0) and np.all(c.trace(sc, rays, False) == rsh.HIT_NONE)
    sc.destroy()
    c.destroy()


def test_frame_counts_ray_cluster_pairs(cornell):
    """A frame's (ray, cluster) pairs: every pair tests at least one and at most cluster_size triangles."""
    c = rsh.Context(rsh.default_config(flags=rsh.FLAG_SEQUENTIAL_RAYS))
    sc = c.scene(cornell.positions, cornell.normals, cornell.material_ids, cornell.materials)
    c.set_camera(rsh.camera_look_at(cornell.eye, cornell.target, cornell.up, cornell.fov, 64, 48))
    c.set_lights(cornell.lights)
    c.render(sc, 64, 48, 1)
    st = c.stats()
    assert st["candidates"] > 0 and st["tri_tests"] <= st["candidates"] * c.config.cluster_size
    assert st["overflow_passes"] == 0
    sc.destroy()
    c.destroy()
