"""The order in which rays alone are traced -- as they come, listed by ray generation, or hashed and sorted --
changes no result. Batches on either side of the count above which they are sorted, with one segment, a power of
two of them and one more, empty and rayless segments among them, directly and as a captured graph: every record
of the large batch equals that of the same rays in small (unsorted) calls, and brute force on a sample. Frames
whose ray lists end inside a warp or a block equal the oracle, ray by ray, in both forms."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

import frame_check
import oracle
import rsh
from rsh import scenes

pytestmark = pytest.mark.gpu

SORT_RAYS = 2_000_000


@pytest.mark.parametrize("nseg,total", [(1, SORT_RAYS), (1, SORT_RAYS + 1), (4, SORT_RAYS + 77), (5, 2_300_001)])
def test_batches_around_the_sorted_count(nseg, total):
    c = rsh.Context(rsh.default_config())
    data = [scenes.random_soup(t, np.random.default_rng(t)) for t in (3000, 12_000)]
    scs = [c.scene(s.positions, s.normals, s.material_ids, s.materials) for s in data]
    rng = np.random.default_rng(nseg)
    sizes = [total] if nseg == 1 else [0, 4099] + [(total - 4099) // (nseg - 2)] * (nseg - 2)
    sizes[-1] += total - sum(sizes)
    segs = (rsh.BatchSegment * nseg)()
    rays, bufs = [], []
    for i, n in enumerate(sizes):
        s, any_hit = data[i % 2], i % 2 == 1
        r = scenes.surface_rays(s, max(n, 1), rng)[:n]
        if any_hit:
            r["tmax"] = rng.uniform(0.1, 10.0, n).astype(np.float32)
        r["tmax"][3::11] = -1.0
        if i == 1:
            r["tmax"] = -1.0  # a segment without a ray
        d = rsh.DeviceArray.from_numpy(r) if n else rsh.DeviceArray(1, rsh.RAY_DTYPE)
        o = rsh.DeviceArray(max(n, 1), np.uint32 if any_hit else np.uint64)
        o.fill_bytes(0x5A)
        rays.append(r)
        bufs.append((d, o))
        segs[i].scene, segs[i].rays, segs[i].n, segs[i].any_hit = scs[i % 2].handle, d.ptr, n, int(any_hit)
        segs[i].hits, segs[i].flags = (None, o.ptr) if any_hit else (o.ptr, None)
    rsh.check(rsh.lib().rsh_batch_trace(c.handle, segs, nseg, None), "batch")
    c.check_device_errors()
    st = rsh.FrameStats()
    rsh.check(rsh.lib().rsh_batch_stats_get(c.handle, C.byref(st)), "stats")
    assert st.reflection_rays == sum(int((r["tmax"] > r["tmin"]).sum()) for r in rays)
    want = []
    for i, n in enumerate(sizes):
        any_hit = i % 2 == 1
        parts = [c.trace(scs[i % 2], rays[i][a:a + 500_000], any_hit, fused=True) for a in range(0, n, 500_000)]
        want.append(np.concatenate(parts) if parts else np.zeros(0, np.uint32 if any_hit else np.uint64))
        assert np.array_equal(bufs[i][1].numpy(n), want[i]), i
        pick = np.sort(rng.permutation(n)[:2000])
        assert np.array_equal(want[i][pick], oracle.brute(data[i % 2].positions, rays[i][pick], any_hit)), i
    stream, graph = C.c_void_p(), C.c_void_p()
    rsh.check(rsh.lib().rsh_stream_create(C.byref(stream)), "stream")
    rsh.check(rsh.lib().rsh_batch_graph_create(c.handle, segs, nseg, stream, C.byref(graph)), "graph")
    for _, o in bufs:
        o.fill_bytes(0x5A)
    for _ in range(2):
        rsh.check(rsh.lib().rsh_batch_graph_launch(graph, stream), "launch")
    rsh.check(rsh.lib().rsh_stream_synchronize(stream), "sync")
    for i, n in enumerate(sizes):
        assert np.array_equal(bufs[i][1].numpy(n), want[i]), i
    c.check_device_errors()
    rsh.lib().rsh_batch_graph_destroy(graph)
    rsh.lib().rsh_stream_destroy(stream)
    for sc in scs:
        sc.destroy()
    c.destroy()


@pytest.mark.parametrize("flags", [0, rsh.FLAG_FUSED, rsh.FLAG_FUSED | rsh.FLAG_SOFT_SHADOWS])
@pytest.mark.parametrize("W,H,lights", [(1, 1, 1), (7, 3, 2), (33, 17, 3), (130, 9, 8)])
def test_frames_with_ragged_ray_lists(cornell, W, H, lights, flags):
    s = dataclasses.replace(cornell, lights=[dict(cornell.lights[0], position=(0.1 * i, 0.9 - 0.05 * i, 0.05 * i))
                                             for i in range(lights)])
    c = rsh.Context(rsh.default_config(flags=flags, reflect_jitter=1.0))
    sc = c.scene(s.positions, s.normals, s.material_ids, s.materials)
    samples = 16 if flags & rsh.FLAG_SOFT_SHADOWS else 1
    st, _ = frame_check.check_frame(c, s, sc, W, H, 2, 1.0, samples=samples, image=W > 1)
    assert st["chunks"] == st["shadow_rays"] + st["reflection_rays"]
    sc.destroy()
    c.destroy()
