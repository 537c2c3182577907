"""rsh_batch_stats_get reports the last rsh_batch_trace, whatever plain traces came after it."""
import ctypes as C

import numpy as np
import pytest

import rsh
from rsh import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 2_100_000])  # in their own order; sorted
def test_plain_traces_leave_the_batch_statistics(n):
    c = rsh.Context(rsh.default_config())
    s = scenes.random_soup(12_000, np.random.default_rng(1))
    sc = c.scene(s.positions)
    rays = scenes.surface_rays(s, n, np.random.default_rng(2))
    rays["tmax"][::4] = -1.0
    c.trace(sc, rays, True, fused=True)
    want = int((rays["tmax"] > rays["tmin"]).sum())
    for _ in range(2):
        st = rsh.FrameStats()
        rsh.check(rsh.lib().rsh_batch_stats_get(c.handle, C.byref(st)), "stats")
        assert st.reflection_rays == st.chunks == want
        c.trace(sc, rays[:700], False)
    sc.destroy()
    c.destroy()
