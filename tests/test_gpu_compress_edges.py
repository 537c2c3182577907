"""Trim + compress, the pair sort and decompress at the edges of their rows (32 slots), warps and CTAs: few slots,
around a row, around the size where every CTA has work, more than one batch of rows per warp; runs that cross
rows, warps and CTAs, no ray at all, one chunk, a chunk per ray, keys at a 4-byte offset. Bit for bit the CPU
oracle, launched and replayed from a captured graph; nothing is written past the counts."""
import numpy as np
import pytest

import oracle
import rsh

pytestmark = pytest.mark.gpu
NONE = 0xFFFFFFFF


def _keys(kind, n, rng):
    if kind == "runs":
        k = np.repeat(rng.integers(0, 1 << 24, n, dtype=np.uint64), rng.integers(1, 90, n))[:n].astype(np.uint32)
        k[rng.random(n) < 0.3] = NONE
        return k
    if kind == "holes":  # long stretches without a ray, inside runs too
        k = (np.arange(n, dtype=np.uint32) // 2500) % 7
        k[(np.arange(n) // 700) % 3 == 1] = NONE
        return k
    if kind == "each":
        return rng.permutation(n).astype(np.uint32)
    return np.full(n, NONE if kind == "none" else 5, np.uint32)


@pytest.mark.parametrize("kind", ["runs", "holes", "each", "none", "one"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 511, 513, 2049, 608 * 512, 608 * 512 + 1, 608 * 8 * 32 * 8 + 77, 1_700_003])
def test_compress_sort_decompress_edges(n, kind):
    ctx = rsh.Context(rsh.default_config())
    rng = np.random.default_rng(n)
    keys = _keys(kind, n, rng)
    tr, ck, cb, _ = oracle.compress(keys)
    R, Cn = len(tr), len(ck)
    dk = rsh.DeviceArray(n + 1, np.uint32)
    dk.upload(np.concatenate([np.zeros(1, np.uint32), keys]))
    # trimmed ids, chunk keys, chunk bases, sorted chunk keys and values, sorted ray keys and ids
    out = [rsh.DeviceArray(n + 2, np.uint32) for _ in range(7)]
    counts = rsh.DeviceArray(2, np.uint32)
    L, (dtr, dck, dcb, dsk, dsv, dok, doi) = rsh.lib(), out

    def run(stream):
        rsh.check(L.rsh_compress(ctx.handle, dk.ptr + 4, n, dtr.ptr, dck.ptr, dcb.ptr, None, counts.ptr, stream), "compress")
        rsh.check(L.rsh_sort_pairs(ctx.handle, dck.ptr, None, dsk.ptr, dsv.ptr, n, counts.ptr + 4, 32, stream), "sort")
        rsh.check(L.rsh_decompress(ctx.handle, dsk.ptr, dsv.ptr, dcb.ptr, dtr.ptr, counts.ptr, n, dok.ptr, doi.ptr,
                                   stream), "decompress")

    def verify(what):
        ctx.check_device_errors()
        assert list(counts.numpy()) == [R, Cn], what
        sk, sv = oracle.sort_pairs(ck, None, 32)
        ok, oi = oracle.decompress(sk, sv, cb, tr)
        for got, want in zip(out, (tr, ck, cb[:Cn + 1], sk, sv, ok, oi)):
            g = got.numpy()
            assert np.array_equal(g[:len(want)], want), what
            assert np.all(g[len(want):] == 0x5A5A5A5A), what

    for a in out:
        a.fill_bytes(0x5A)
    run(None)
    verify("launched")
    import torch

    for a in out:
        a.fill_bytes(0x5A)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        run(stream.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    verify("replayed")
    ctx.destroy()
