"""Serving scenes whose rays go alone beside scenes whose rays use packets: steps that hold only one kind, then both,
then the other, so that a request's stage is generated beside another mixture than the stage before it. Every record
equals the same request served by itself, and rsh_render_frame's."""
import ctypes as C

import numpy as np
import pytest

import rsh
from rsh import scenes
from test_gpu_server import _request

pytestmark = pytest.mark.gpu


def _serve(ctx, scs, reqs, step_rays=0, first=None):
    """Serves reqs; `first`: a long request that keeps the GPU busy while they are submitted."""
    L = rsh.lib()
    arr = (C.c_void_p * len(scs))(*[s.handle for s in scs])
    srv = C.c_void_p()
    rsh.check(L.rsh_server_create(ctx.handle, arr, len(scs), 4 << 30, 64, C.byref(srv)), "server")
    rsh.check(L.rsh_server_set_step_rays(srv, step_rays), "step rays")
    ids = []
    for r in ([first] if first else []) + reqs:
        i = C.c_uint64()
        rsh.check(L.rsh_server_submit(srv, C.byref(r), C.byref(i)), "submit")
        ids.append(i.value)
    if first:
        rsh.check(L.rsh_server_wait(srv, ids.pop(0), 120_000, None, None, None), "wait")
    outs = []
    for r, i in zip(reqs, ids):
        npix = r.width * r.height
        hits, flags = np.empty(npix * r.depth, np.uint64), np.empty(npix * r.light_count * r.depth, np.uint32)
        res = rsh.RequestResult()
        st = L.rsh_server_wait(srv, i, 120_000, C.byref(res), hits.ctypes.data, flags.ctypes.data)
        outs.append((st, hits, flags, res.rays))
    L.rsh_server_destroy(srv)
    return outs


@pytest.mark.parametrize("packets", [0, 1, 2])
def test_requests_beside_another_form(packets):
    """Scene `packets` is tuned to packets, the two others go alone. With 8000 rays a step, requests X, A, C (with the
    primary rays X 4096, A 1024, C 4096; bounces twice that) run as {X, A}, {X}, {A, C}, ...: A's first stage beside X,
    its second beside C."""
    ctx = rsh.Context(grid_bits=5, dir_log2=4, packet_size=8, cluster_size=8, reflect_jitter=1.0)
    sd = (scenes.cornell(), scenes.soup(n_spheres=300, extent=20.0), scenes.soup(n_spheres=60, extent=9.0))
    scs = [ctx.scene(s.positions, s.normals, s.material_ids, s.materials) for s in sd]
    scs[packets].set_tuning(ray_level=0)

    def req(si, size, depth):
        s = sd[si]
        return _request(si, rsh.camera_look_at(s.eye, s.target, s.up, s.fov, size, size), size, size, depth, s.lights[:1])

    big = req(0, 2048, 1)
    x, a, c = [k for k in range(3) if k != packets] + [packets]  # X and A alone, C with packets
    orders = [[req(x, 64, 1), req(a, 32, 4), req(c, 64, 3)],
              [req(c, 64, 1), req(a, 32, 4), req(x, 64, 3)],
              [req(x, 64, 1), req(c, 32, 4), req(a, 64, 3), req(c, 16, 2), req(x, 40, 4)]]
    for reqs in orders:
        alone = [_serve(ctx, scs, [r])[0] for r in reqs]
        for step_rays in (8000, 0, 3000):
            got = _serve(ctx, scs, reqs, step_rays, big)
            for k, (g, w) in enumerate(zip(got, alone)):
                assert g[0] == w[0] == rsh.RSH_OK
                assert np.array_equal(g[1], w[1]), f"hits of request {k}, {step_rays} rays a step"
                assert np.array_equal(g[2], w[2]), f"flags of request {k}, {step_rays} rays a step"
                assert g[3] == w[3] > 0
        for r, w in zip(reqs, alone):
            ctx.set_camera(r.camera)
            ctx.set_lights([{"position": tuple(r.lights[0].position)}])
            ctx.render(scs[r.scene_index], r.width, r.height, r.depth)
            n = r.width * r.height
            for b in range(r.depth):
                assert np.array_equal(ctx.frame_hits(b, n), w[1][b * n:(b + 1) * n])
                assert np.array_equal(ctx.frame_shadow(b, n), w[2][b * n:(b + 1) * n])
    ctx.check_device_errors()
    for s in scs:
        s.destroy()
    ctx.destroy()


def test_tuning_changed_between_the_stages_of_a_request():
    """A scene's switch level set anew while its requests are in flight changes no record."""
    ctx = rsh.Context(grid_bits=5, dir_log2=4, packet_size=8, cluster_size=8, reflect_jitter=1.0)
    s = scenes.soup(n_spheres=300, extent=20.0)
    sc = ctx.scene(s.positions, s.normals, s.material_ids, s.materials)
    reqs = [_request(0, rsh.camera_look_at(s.eye, s.target, s.up, s.fov, W, W), W, W, 4, s.lights[:1]) for W in (320, 97)]
    want = [_serve(ctx, [sc], [r])[0] for r in reqs]
    L = rsh.lib()
    arr = (C.c_void_p * 1)(sc.handle)
    srv = C.c_void_p()
    rsh.check(L.rsh_server_create(ctx.handle, arr, 1, 4 << 30, 64, C.byref(srv)), "server")
    for trial in range(6):
        ids = []
        for r in reqs * 4:
            i = C.c_uint64()
            rsh.check(L.rsh_server_submit(srv, C.byref(r), C.byref(i)), "submit")
            ids.append(i.value)
        for k, i in enumerate(ids):
            sc.set_tuning(ray_level=15 * (k & 1))
            r, w = reqs[k % 2], want[k % 2]
            hits, flags = np.empty_like(w[1]), np.empty_like(w[2])
            assert L.rsh_server_wait(srv, i, 120_000, None, hits.ctypes.data, flags.ctypes.data) == rsh.RSH_OK
            assert np.array_equal(hits, w[1]) and np.array_equal(flags, w[2]), (trial, k)
    L.rsh_server_destroy(srv)
    sc.destroy()
    ctx.destroy()
