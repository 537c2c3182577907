"""The pair sort where its tiles change: a tile's rows follow from the count and the number of CTAs (2 to 10 rows of
512 keys, then 14 at once), the number of CTAs from the capacity (one an SM up to SMs x 7168 keys, then two). One key
either side of every such line, for the capacity itself and for a device count below a larger capacity. Equal to
numpy's stable sort, bit for bit; nothing is written past the count."""
import numpy as np
import pytest

import rsh

pytestmark = pytest.mark.gpu

# rows a tile at the line, CTAs an SM of the capacity that gives them (None: the capacity is the count)
LINES = [(2, None), (3, None), (10, None), (11, None), (14, None), (2, 1), (10, 1), (11, 1), (2, 2), (10, 2), (14, 2)]


@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("rows,per_sm", LINES)
def test_sort_rows(rows, per_sm, side):
    sms = rsh.lib().rsh_sm_count()
    n = sms * 512 * rows * (per_sm or 1) + side
    cap = {None: n, 1: sms * 7168, 2: 3 * sms * 7168}[per_sm]
    if per_sm == 1:
        n = min(n, cap)
    rng = np.random.default_rng(rows * 10 + side)
    keys = rng.integers(0, 1 << 20, cap, dtype=np.uint32)
    keys[::5] = keys[0]
    dk = rsh.DeviceArray.from_numpy(keys)
    ok, ov = rsh.DeviceArray(cap, np.uint32), rsh.DeviceArray(cap, np.uint32)
    ok.fill_bytes(0x5A)
    ov.fill_bytes(0x5A)
    cnt = rsh.DeviceArray.from_numpy(np.array([n], np.uint32))
    ctx = rsh.Context(rsh.default_config())
    rsh.check(rsh.lib().rsh_sort_pairs(ctx.handle, dk.ptr, None, ok.ptr, ov.ptr, cap, cnt.ptr if per_sm else None, 20,
                                       None), "sort")
    ctx.check_device_errors()
    order = np.argsort(keys[:n], kind="stable").astype(np.uint32)
    gk, gv = ok.numpy(), ov.numpy()
    assert np.array_equal(gk[:n], keys[:n][order]) and np.array_equal(gv[:n], order)
    assert np.all(gk[n:] == 0x5A5A5A5A) and np.all(gv[n:] == 0x5A5A5A5A)
    ctx.destroy()
