"""Frames of many bounces: the statistics' counts of every bounce are those of the frame's own rays, whatever the depth,
in the rays-alone and in the packet form. (The counters are copied to pinned memory, 4 words a bounce, by a kernel in
the first form: the block has to hold them at 60 bounces, where they once met the statistics behind them, and past 252,
where they once met its end.)"""
import numpy as np
import pytest

import rsh
from rsh import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [dict(flags=rsh.FLAG_FUSED), dict(), dict(plain_ray_level=0)])
@pytest.mark.parametrize("depths", [(59, 60, 61), (3, 247, 248, 300, 3)])
def test_deep_frame_counts(depths, form):
    s = scenes.cornell()
    W, H, L = 12, 9, len(s.lights)
    c = rsh.Context(rsh.default_config(reflect_jitter=0.3, **form))
    sc = c.scene(s.positions, s.normals, s.material_ids, s.materials)
    c.set_camera(rsh.camera_look_at(s.eye, s.target, s.up, s.fov, W, H))
    c.set_lights(s.lights)
    for depth in depths:
        c.render(sc, W, H, depth)
        st = c.stats()
        want = [0, 0]
        for b in range(depth):
            for shadow in (0, 1):
                r = c.frame_rays(b, bool(shadow), W * H * (L if shadow else 1))
                want[shadow] += int((r["tmax"] > r["tmin"]).sum())
        assert [st["reflection_rays"], st["shadow_rays"]] == want and want[0] > 0
        assert st["node_tests"] > 0 and st["tri_tests"] > 0 and st["primary_rays"] == W * H
    c.check_device_errors()
    sc.destroy()
    c.destroy()
