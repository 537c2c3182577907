"""Frames back to back without a host synchronisation: a frame's kernels are chained, and every buffer they pass on is
written again by the next bounce and the next frame, so a kernel that read a value from before the last write would
show a ray, flag or hit of another frame. Two different frames in turn, in every form, equal each of them alone bit for
bit; sizes from less than a block to several waves."""
import numpy as np
import pytest

import rsh
from rsh import scenes

pytestmark = pytest.mark.gpu


def _records(c, W, H, depth, lights, rgba):
    n = W * H
    out = [rgba.numpy(), c.frame_hits(-1, n)]
    for b in range(depth):
        out += [c.frame_hits(b, n), c.frame_shadow(b, n * lights), c.frame_rays(b, False, n).view(np.uint8)]
    return out


@pytest.mark.parametrize("flags", [0, rsh.FLAG_FUSED, rsh.FLAG_FUSED | rsh.FLAG_SEQUENTIAL_RAYS,
                                   rsh.FLAG_FUSED | rsh.FLAG_SOFT_SHADOWS])
@pytest.mark.parametrize("W,H,depth", [(9, 7, 4), (64, 64, 4), (200, 121, 3), (640, 360, 2)])
def test_frames_in_turn(W, H, depth, flags):
    s = scenes.cornell()
    samples = 16 if flags & rsh.FLAG_SOFT_SHADOWS else 1
    frames = []
    for k in range(2):
        eye = np.array(s.eye) + np.array([0.3 * k, -0.2 * k, 0.1 * k])
        frames.append((rsh.camera_look_at(eye, s.target, s.up, s.fov + 7 * k, W, H), (s.lights * 2)[:2 - k]))
    c = rsh.Context(rsh.default_config(flags=flags, reflect_jitter=0.5))
    sc = c.scene(s.positions, s.normals, s.material_ids, s.materials)
    rgba = rsh.DeviceArray(W * H, np.uint32)

    def render(k):
        c.set_camera(frames[k][0])
        c.set_lights(frames[k][1])
        c.render(sc, W, H, depth, rgba)

    alone = []
    for k in range(2):
        render(k)
        rsh.check(rsh.lib().rsh_stream_synchronize(None), "sync")
        alone.append(_records(c, W, H, depth, len(frames[k][1]) * samples, rgba))
    assert not np.array_equal(alone[0][0], alone[1][0])
    for last in (0, 1):
        for _ in range(8):
            render(1 - last)
            render(last)
        got = _records(c, W, H, depth, len(frames[last][1]) * samples, rgba)
        assert all(np.array_equal(a, b) for a, b in zip(got, alone[last]))
    c.check_device_errors()
    sc.destroy()
    c.destroy()
