"""The ray-space hierarchy at the edges of its CTAs (64 packets each) and levels: one ray, one packet, around a
CTA's rays, a single node on top, a device count anywhere below the capacity, padding ids, packets without a ray
and nodes at a 4-byte offset. Bit for bit the CPU oracle's nodes (a NaN is a NaN); nothing is written past the used ones."""
import numpy as np
import pytest

import oracle
import rsh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [8, 16, 32])
@pytest.mark.parametrize("packets", [1, 2, 7, 8, 9, 63, 64, 65, 128, 64 * 3 + 1])
def test_build_rsh_edges(P, packets):
    rng = np.random.default_rng(P * 1000 + packets)
    for m in sorted({packets * P, packets * P - 1, packets * P - P + 1}):
        n = m + int(rng.integers(0, 3 * 64 * P))  # capacity
        rays = np.zeros(n, rsh.RAY_DTYPE)
        rays["o"] = rng.uniform(-5, 5, (n, 3)).astype(np.float32)
        d = rng.normal(size=(n, 3))
        rays["d"] = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        rays["tmin"], rays["tmax"] = 1e-4, rng.uniform(0.5, 9, n).astype(np.float32)
        rays["tmax"][rng.random(n) < 0.1] = -1.0
        ids = rng.permutation(n).astype(np.uint32)
        rays["tmax"][ids[:P]] = -1.0  # the first packet has no ray
        nodes_cap = rsh.lib().rsh_hierarchy_capacity(n, P, (off := (rsh.C.c_uint32 * 4)()))
        words = rsh.NODE_DTYPE.itemsize // 4
        buf = rsh.DeviceArray(nodes_cap * words + 1, np.uint32)
        buf.fill_bytes(0x5A)
        cnt = rsh.DeviceArray.from_numpy(np.array([m], np.uint32))
        d_rays, d_ids = rsh.DeviceArray.from_numpy(rays), rsh.DeviceArray.from_numpy(ids)
        for own in (True, False):  # through the ids, or the rays in order
            rsh.check(rsh.lib().rsh_build_rsh(d_rays.ptr, d_ids.ptr if own else None, n, cnt.ptr, P, buf.ptr + 4, None),
                      "build")
            g = buf.numpy()[1:].reshape(nodes_cap, words)
            want, _ = oracle.build_rsh(rays, ids if own else None, m, P, max_rays=n)
            used = np.zeros(nodes_cap, bool)
            c = m
            for lvl, k in enumerate((P, 8, 8)):
                c = (c + k - 1) // k
                used[off[lvl]:off[lvl] + c] = True
                a = g[off[lvl]:off[lvl] + c]
                b = want[off[lvl]:off[lvl] + c].view(np.uint32).reshape(c, words)
                nan = np.isnan(a.view(np.float32)) & np.isnan(b.view(np.float32))  # the centre of a packet without rays
                assert np.all((a == b) | nan), (m, own, lvl)
            assert np.all(g[~used] == 0x5A5A5A5A), (m, own)
