"""The pair sort at the edges of its tile shapes and of their choice by size: one pair, around a small and a large
tile, around the size that changes the shape, more tiles than SMs, with the device count anywhere below the
capacity, every count of digit passes, keys that are all equal or all ones, and arrays at a 4-byte offset. Equal
to numpy's stable sort, bit for bit; nothing is written past the count."""
import numpy as np
import pytest

import rsh

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 2047, 2048, 2049, 7167, 7168, 7169, 152 * 2048 + 5, (1 << 19) - 1, 1 << 19, (1 << 19) + 1,
         2 * 152 * 7168 + 1]


@pytest.mark.parametrize("bits", [1, 8, 9, 24, 31, 32])
@pytest.mark.parametrize("n_max", SIZES)
def test_sort_pairs_edges(n_max, bits):
    ctx = rsh.Context(rsh.default_config())
    rng = np.random.default_rng(n_max + bits)
    mask = np.uint32((1 << (8 * ((bits + 7) // 8))) - 1)  # the sort looks at the whole 8-bit digits that `bits` reaches
    for kind, n in (("random", n_max), ("counted", max(1, n_max * 2 // 3)), ("none", 0), ("equal", n_max), ("ones", n_max)):
        keys = rng.integers(0, 1 << 32, n_max, dtype=np.uint64).astype(np.uint32)
        if kind == "equal":
            keys[:] = keys[0]
        if kind == "ones":
            keys[::3] = 0xFFFFFFFF
        vals = rng.integers(0, 1 << 32, n_max, dtype=np.uint64).astype(np.uint32)
        off = 4 if kind == "random" else 0  # arrays 4 bytes past an aligned address
        dk, dv = rsh.DeviceArray(n_max + 1, np.uint32), rsh.DeviceArray(n_max + 1, np.uint32)
        ok, ov = rsh.DeviceArray(n_max + 1, np.uint32), rsh.DeviceArray(n_max + 1, np.uint32)
        pad = np.zeros(off // 4, np.uint32)
        dk.upload(np.concatenate([pad, keys]))
        dv.upload(np.concatenate([pad, vals]))
        ok.fill_bytes(0x5A)
        ov.fill_bytes(0x5A)
        cnt = rsh.DeviceArray.from_numpy(np.array([n], np.uint32))
        own = kind in ("counted", "ones")
        rsh.check(rsh.lib().rsh_sort_pairs(ctx.handle, dk.ptr + off, dv.ptr + off if own else None, ok.ptr + off,
                                           ov.ptr + off, n_max, None if n == n_max else cnt.ptr, bits, None), "sort")
        ctx.check_device_errors()
        order = np.argsort(keys[:n] & mask, kind="stable")
        gk, gv = ok.numpy()[off // 4:][:n_max], ov.numpy()[off // 4:][:n_max]
        assert np.array_equal(gk[:n], keys[:n][order]), kind
        assert np.array_equal(gv[:n], vals[:n][order] if own else order.astype(np.uint32)), kind
        assert np.all(gk[n:] == 0x5A5A5A5A) and np.all(gv[n:] == 0x5A5A5A5A), kind
    ctx.destroy()
