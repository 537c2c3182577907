"""Ray sets past the limits of one sorted batch: more slots than a sort's 30-bit digit counts hold (a batched call traces
them in their own order) and more than 31 bits count (the plain path takes them in parts). Nearly all slots are empty;
the results of the rays at the ends and around the part borders equal brute force, and empty slots beside them get
theirs."""
import ctypes as C

import numpy as np
import pytest

import oracle
import rsh
from rsh import scenes

pytestmark = pytest.mark.gpu

N = (1 << 31) + 1000
M = (1 << 30) + 1010
NEED = 32 * N + 4 * N + (24 << 30)


def test_more_rays_than_a_sort_or_31_bits_hold():
    free, total = C.c_uint64(), C.c_uint64()
    rsh.check(rsh.lib().rsh_device_memory(C.byref(free), C.byref(total)), "memory")
    if free.value < NEED:
        pytest.skip("needs 102 GB of device memory")
    s = scenes.random_soup(12_000, np.random.default_rng(4))
    c = rsh.Context(rsh.default_config())
    sc = c.scene(s.positions, s.normals, s.material_ids, s.materials)
    rays = rsh.DeviceArray(N, rsh.RAY_DTYPE, zero=True)  # tmax = tmin: no ray
    out = rsh.DeviceArray(M, np.uint64)  # flags of N rays, then hits of M
    assert out.nbytes >= max(4 * N, 8 * M)
    rng = np.random.default_rng(5)
    marks = {}
    for at in (0, (1 << 29) - 1000, (1 << 30) - 1000, (1 << 30) + 10, 3 * (1 << 29) - 7, N - 1000):
        r = scenes.surface_rays(s, 990, rng)
        r["tmax"] = rng.uniform(0.5, 15.0, len(r)).astype(np.float32)
        r["tmax"][::5] = -1.0
        rsh.check(rsh.lib().rsh_memcpy_h2d(rays.ptr + 32 * at, r.ctypes.data, r.nbytes, None), "h2d")
        rsh.check(rsh.lib().rsh_stream_synchronize(None), "sync")
        marks[at] = r

    def check(n, any_hit, dtype, miss):
        c.check_device_errors()
        for at, r in marks.items():
            if at + 1000 > n:
                continue
            got = np.empty(1000, dtype)
            rsh.check(rsh.lib().rsh_memcpy_d2h(got.ctypes.data, out.ptr + got.itemsize * at, got.nbytes, None), "d2h")
            assert np.array_equal(got[:990], oracle.brute(s.positions, r, any_hit)), (n, at)
            assert np.all(got[990:] == miss), (n, at)

    out.fill_bytes(0x5A)
    rsh.check(rsh.lib().rsh_trace_rays(c.handle, sc.handle, rays.ptr, N, 1, None, out.ptr, None), "plain")
    check(N, True, np.uint32, 0)
    out.fill_bytes(0x5A)
    rsh.check(rsh.lib().rsh_trace_rays_fused(c.handle, sc.handle, rays.ptr, M, 0, out.ptr, None, None), "batched")
    check(M, False, np.uint64, rsh.HIT_NONE)
    sc.destroy()
    c.destroy()
