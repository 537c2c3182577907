"""The scratch that a context keeps for rebuilding moving scenes is part of what it says it has allocated, makes room
when the budget needs it, and goes with the scene."""
import ctypes as C

import numpy as np
import pytest

import rsh
from rsh import scenes

pytestmark = pytest.mark.gpu

SLACK = 64 << 20  # allocations come in pages of 2 MiB


def _free():
    f, t = C.c_uint64(), C.c_uint64()
    rsh.check(rsh.lib().rsh_device_memory(C.byref(f), C.byref(t)), "memory")
    return f.value


def _matrix(angle):
    m = np.eye(4, dtype=np.float32)
    m[0, 0] = m[2, 2] = np.cos(angle)
    m[0, 2], m[2, 0] = np.sin(angle), -np.sin(angle)
    return m.reshape(1, 16)


def test_kept_scratch_is_counted_and_given_back():
    T = 1_000_000
    s = scenes.random_soup(T, np.random.default_rng(3))
    L = rsh.lib()
    c = rsh.Context(rsh.default_config())
    empty = L.rsh_bytes_allocated(c.handle)
    f0 = _free()
    sc = c.scene(s.positions)
    up = L.rsh_bytes_allocated(c.handle)
    assert abs((f0 - _free()) - (up - empty)) < SLACK  # the scene's arrays are what is counted
    f1 = _free()
    sc.set_transforms(_matrix(0.1))
    sc.set_transforms(_matrix(0.2))
    moved = L.rsh_bytes_allocated(c.handle)
    rest_pose = 2 * 48 * T
    assert f1 - _free() < (moved - up) + rest_pose + SLACK
    sc.destroy()
    assert L.rsh_bytes_allocated(c.handle) < empty + (1 << 20)
    assert f0 - _free() < SLACK
    c.destroy()


def test_kept_scratch_makes_room_for_what_the_budget_has_to_hold():
    """A budget that holds the scene and the rays' buffers, but not the scratch beside them: every call that fits without
    it is served, before and after a rebuild, and the results are those of an unlimited context."""
    T, n = 200_000, 2_500_000  # more rays than are traced unsorted: the sort's buffers come from the budget
    s = scenes.random_soup(T, np.random.default_rng(5))
    rays = scenes.surface_rays(s, n, np.random.default_rng(6))
    free = rsh.Context(rsh.default_config())
    sc = free.scene(s.positions)
    sc.set_transforms(_matrix(0.3))
    want = free.trace(sc, rays, False)
    sc.destroy()
    L = rsh.lib()
    c = rsh.Context(rsh.default_config())
    sc = c.scene(s.positions)
    c.trace(sc, rays, False)
    need = L.rsh_bytes_allocated(c.handle)  # scene and buffers, nothing kept
    sc.destroy()
    c.destroy()
    c = rsh.Context(rsh.default_config(hbm_budget=need + (1 << 20)))
    sc = c.scene(s.positions)
    for angle in (0.1, 0.3):
        sc.set_transforms(_matrix(angle))
        got = c.trace(sc, rays, False)
        assert L.rsh_bytes_allocated(c.handle) <= need + (1 << 20)
    assert np.array_equal(got, want)
    sc2 = c.scene(scenes.random_soup(100, np.random.default_rng(7)).positions)  # a scene beside it
    sc2.destroy()
    sc.destroy()
    c.destroy()
    free.destroy()
