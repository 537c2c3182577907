// Decompression of sorted chunks into the sorted ray permutation.
//
// Reference: RayDecompressionWrapper (RayTracer.cu:2411-2467): CreateSortedRaySkeleton (:993-1010,
// skeleton[x] = size[sortedValue[x]]) -> cub ExclusiveSum -> CreateSortedRays (:1012-1059), where one
// thread copies a whole chunk serially (load-imbalanced; the largest sort-stage cost in the thesis
// timings). Here:
//  1. exclusive scan of the sorted chunk sizes -> off[x], reduce-then-scan over a fixed number of CTAs, a
//     contiguous range of whole rows of 32 chunks per warp (k_dc_reduce: sums; k_dc_write: each CTA folds the
//     sums before its own and writes the chunk offsets); every chunk also records itself as the first chunk of
//     each 2048-output expand tile that starts inside it (tile_chunk[m]);
//  2. k_dc_expand: every CTA owns 2048 consecutive OUTPUT rays, reads its chunk range from tile_chunk, stages
//     what those chunks add to an output index and their keys in shared memory, and marks their first outputs in
//     a 2048-bit mask: a ray's chunk is the number of marks up to it. Work per CTA is fixed whatever the chunk
//     sizes.
// us for 2.76 M rays in 600,000 chunks: 4.4 + 5.7 + 10 (2048-chunk tiles with a launch of their own for the scan of
// the sums, and a binary search per ray: 9.5 + 3.0 + 4.7 + 15); with the launches chained 16 less of 165 from raygen
// to the hierarchy.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace rsh {

namespace {
constexpr uint32_t DS_THREADS = 256, DS_WARPS = DS_THREADS / 32;
constexpr uint32_t DS_CTAS = 4 * 152;  // most CTAs of the scan: four per SM
constexpr uint32_t DS_BATCH = 4;       // rows whose loads are in flight together
constexpr uint32_t DE_THREADS = 256;
constexpr uint32_t DE_ITEMS = 8;
constexpr uint32_t DE_TILE = DE_THREADS * DE_ITEMS;  // output rays per expand CTA

// the chunks of a warp: whole rows, the same number for every warp but the last ones
RSH_DEV void warp_range(uint32_t C, uint32_t& b, uint32_t& e) {
    const uint32_t warps = gridDim.x * DS_WARPS;
    const uint64_t per = 32ull * (((uint64_t)C + 32ull * warps - 1u) / (32ull * warps));
    const uint64_t x = per * (blockIdx.x * DS_WARPS + (threadIdx.x >> 5));
    b = (uint32_t)min(x, (uint64_t)C);
    e = (uint32_t)min(x + per, (uint64_t)C);
}
RSH_DEV uint32_t warp_sum(uint32_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
}  // namespace

// Gathers each sorted chunk's base and size once (the only random reads of the chunk table) into sorted order, and
// sums the sizes: csum per CTA, wsum per warp.
__global__ void __launch_bounds__(DS_THREADS)
k_dc_reduce(const uint32_t* __restrict__ vals, const uint32_t* __restrict__ bases,
            const uint32_t* __restrict__ counts, uint32_t max_chunks, uint32_t* __restrict__ csum,
            uint32_t* __restrict__ wsum, uint32_t* __restrict__ sbase, uint32_t* __restrict__ ssize) {
    __shared__ uint32_t s_warp[DS_WARPS];
    asm volatile("griddepcontrol.launch_dependents;");
    const uint32_t C = counts[1] < max_chunks ? counts[1] : max_chunks;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t b, e, sum = 0;
    warp_range(C, b, e);
    for (uint32_t q = b; q < e; q += 32u * DS_BATCH) {
        uint32_t c[DS_BATCH], lo[DS_BATCH], hi[DS_BATCH];
#pragma unroll
        for (uint32_t i = 0; i < DS_BATCH; ++i) {
            const uint32_t x = q + 32u * i + lane;
            c[i] = x < e ? __ldg(vals + x) : C;
        }
#pragma unroll
        for (uint32_t i = 0; i < DS_BATCH; ++i) {
            lo[i] = c[i] < C ? __ldg(bases + c[i]) : 0u;
            hi[i] = c[i] < C ? __ldg(bases + c[i] + 1) : 0u;
        }
#pragma unroll
        for (uint32_t i = 0; i < DS_BATCH; ++i) {
            const uint32_t x = q + 32u * i + lane;
            if (x < e) {
                sbase[x] = lo[i];
                ssize[x] = hi[i] - lo[i];
            }
            sum += hi[i] - lo[i];
        }
    }
    sum = warp_sum(sum);
    if (lane == 0u) {
        s_warp[warp] = sum;
        wsum[blockIdx.x * DS_WARPS + warp] = sum;
    }
    __syncthreads();
    if (warp == 0u) {
        const uint32_t t = warp_sum(lane < DS_WARPS ? s_warp[lane] : 0u);
        if (lane == 0u) csum[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(DS_THREADS)
k_dc_write(const uint32_t* __restrict__ ssize, const uint32_t* __restrict__ counts, uint32_t max_chunks,
           const uint32_t* __restrict__ csum, const uint32_t* __restrict__ wsum, uint32_t* __restrict__ off,
           uint32_t* __restrict__ tile_chunk, uint32_t mcap) {
    __shared__ uint32_t s_warp[DS_WARPS];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t C = counts[1] < max_chunks ? counts[1] : max_chunks;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    // what comes before the warp: the CTAs before this one, and the warps before it
    uint32_t run = 0;
    for (uint32_t c = threadIdx.x; c < blockIdx.x; c += DS_THREADS) run += ld_chain(csum + c);
    run = warp_sum(run);
    if (lane == 0u) s_warp[warp] = run;
    __syncthreads();
    run = lane < DS_WARPS ? s_warp[lane] : 0u;
    if (lane < warp) run += ld_chain(wsum + blockIdx.x * DS_WARPS + lane);  // (warp < DS_WARPS)
    run = warp_sum(run);
    uint32_t b, e;
    warp_range(C, b, e);
    for (uint32_t q = b; q < e; q += 32u * DS_BATCH) {
        uint32_t sz[DS_BATCH];
#pragma unroll
        for (uint32_t i = 0; i < DS_BATCH; ++i) {
            const uint32_t x = q + 32u * i + lane;
            sz[i] = x < e ? ld_chain(ssize + x) : 0u;
        }
#pragma unroll
        for (uint32_t i = 0; i < DS_BATCH; ++i) {
            const uint32_t x = q + 32u * i + lane;
            uint32_t inc = sz[i];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= (uint32_t)d) inc += y;
            }
            const uint32_t at = run + inc - sz[i];
            if (x < e) {
                off[x] = at;
                // expand tiles whose first output lies in this chunk (sizes are >= 1)
                if (sz[i] > 0u)
                    for (uint32_t m = (at + DE_TILE - 1u) / DE_TILE; m <= (at + sz[i] - 1u) / DE_TILE && m < mcap; ++m)
                        tile_chunk[m] = x;
            }
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
    }
}

__global__ void __launch_bounds__(DE_THREADS)
k_dc_expand(const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ sbase,
            const uint32_t* __restrict__ trimmed,
            const uint32_t* __restrict__ counts, uint32_t max_rays, const uint32_t* __restrict__ off,
            const uint32_t* __restrict__ tile_chunk, uint32_t* __restrict__ sorted_keys,
            uint32_t* __restrict__ sorted_ids, PaddedOut po) {
    constexpr uint32_t WORDS = DE_TILE / 32;
    __shared__ uint32_t s_add[DE_TILE + 1];  // trimmed index less output index
    __shared__ uint32_t s_key[DE_TILE + 1];
    __shared__ uint32_t s_mark[WORDS], s_rank[WORDS];
    static_assert(WORDS == 64, "two warps rank the marks");
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    if (tid < WORDS) s_mark[tid] = 0u;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t R = counts[0] < max_rays ? counts[0] : max_rays;
    const uint32_t C = counts[1];
    const uint32_t k0 = blockIdx.x * DE_TILE;
    if (k0 >= R || C == 0) return;
    // chunks x0..x1 cover the tile's outputs: x0 holds the first, and the chunk holding the next tile's first
    // output is at or after the one holding this one's last (one extra chunk may be staged)
    const uint32_t ntiles = (R + DE_TILE - 1) / DE_TILE;
    const uint32_t x0 = min(ld_chain(tile_chunk + blockIdx.x), C - 1u);
    uint32_t x1 = (blockIdx.x + 1 < ntiles) ? ld_chain(tile_chunk + blockIdx.x + 1) : C - 1;
    if (x1 >= C) x1 = C - 1;
    if (x1 < x0) x1 = x0;
    const uint32_t m = (x1 - x0 + 1 < DE_TILE + 1) ? x1 - x0 + 1 : DE_TILE + 1;
    __syncthreads();
    for (uint32_t i = tid; i < m; i += DE_THREADS) {
        const uint32_t x = x0 + i, o = ld_chain(off + x);
        s_add[i] = ld_chain(sbase + x) - o;
        s_key[i] = skeys ? __ldg(skeys + x) : 0u;
        const uint32_t at = o > k0 ? o - k0 : 0u;  // only the first one may start before the tile
        if (at < DE_TILE) atomicOr(&s_mark[at >> 5], 1u << (at & 31u));
    }
    __syncthreads();
    if (warp < 2u) {
        // the marks before each word (the second warp starts from the first one's)
        const uint32_t other = warp ? warp_sum(__popc(s_mark[lane])) : 0u;
        uint32_t inc = __popc(s_mark[tid]);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= (uint32_t)d) inc += y;
        }
        s_rank[tid] = other + inc - __popc(s_mark[tid]);
    }
    __syncthreads();
    const uint32_t upto = lanemask_lt() | (1u << lane);
    uint32_t ix[DE_ITEMS], id[DE_ITEMS];
#pragma unroll
    for (uint32_t it = 0; it < DE_ITEMS; ++it) {
        const uint32_t w = it * (DE_THREADS / 32) + warp, k = k0 + 32u * w + lane;
        ix[it] = max(s_rank[w] + __popc(s_mark[w] & upto), 1u) - 1u;  // (the first output is marked)
        const uint32_t src = k < R ? s_add[ix[it]] + k : R;
        id[it] = src < R ? __ldg(trimmed + src) : 0u;
    }
#pragma unroll
    for (uint32_t it = 0; it < DE_ITEMS; ++it) {
        const uint32_t k = k0 + it * DE_THREADS + tid;
        if (k >= R) break;
        if (po.padded) {
            const uint32_t q = k + __ldg(po.seg_delta + (s_key[ix[it]] >> po.tag_shift));
            if (q < po.max_padded) po.padded[q] = id[it];
        } else {
            sorted_ids[k] = id[it];
        }
        if (sorted_keys) sorted_keys[k] = s_key[ix[it]];
    }
}

size_t decompress_scratch_bytes(uint32_t max_chunks) {
    const size_t etiles = (max_chunks + DE_TILE - 1) / DE_TILE + 1;
    return (size_t)DS_CTAS * (1 + DS_WARPS) * 4 + (size_t)max_chunks * 12 + etiles * 4 + 512;
}

cudaError_t launch_decompress(const uint32_t* sorted_chunk_keys, const uint32_t* sorted_chunk_vals,
                              const uint32_t* chunk_bases, const uint32_t* trimmed_ids,
                              const uint32_t* counts, uint32_t max_rays, uint32_t* sorted_keys,
                              uint32_t* sorted_ids, void* scratch, uint32_t* err, cudaStream_t s,
                              const PaddedOut* padded_out) {
    (void)err;  // no step of this form waits on another CTA
    if (max_rays == 0) return cudaSuccess;
    const uint32_t max_chunks = max_rays;
    uint32_t* csum = static_cast<uint32_t*>(scratch);
    uint32_t* wsum = csum + DS_CTAS;
    uint32_t* off = wsum + DS_CTAS * DS_WARPS;
    uint32_t* sbase = off + max_chunks;  // sorted chunk bases and sizes
    uint32_t* ssize = sbase + max_chunks;
    uint32_t* tile_chunk = ssize + max_chunks;
    const uint32_t etiles = (max_rays - 1u) / DE_TILE + 1u;
    const uint32_t ctas = std::min(DS_CTAS, (max_chunks - 1u) / DS_THREADS + 1u);  // a row a warp at least
    k_dc_reduce<<<ctas, DS_THREADS, 0, s>>>(sorted_chunk_vals, chunk_bases, counts, max_chunks, csum, wsum, sbase, ssize);
    note_launch();
    cudaError_t e = launch_chained(true, k_dc_write, ctas, DS_THREADS, 0, s, ssize, counts, max_chunks, csum, wsum, off,
                                   tile_chunk, etiles + 1u);
    note_launch();
    if (e != cudaSuccess) return e;
    e = launch_chained(true, k_dc_expand, etiles, DE_THREADS, 0, s, sorted_chunk_keys, sbase, trimmed_ids, counts, max_rays,
                       off, tile_chunk, sorted_keys, sorted_ids,
                       padded_out ? *padded_out : PaddedOut{nullptr, 0u, 0u, nullptr});
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace rsh
