// Trim + compress in one pass over the ray keys.
//
// Reference: RayTrimmingWrapper (RayTracer.cu:2276-2324: CUB InclusiveSum of "no ray" flags, then
// CreateTrimmedRays :844-884, then a blocking D2H of the count) followed by RayCompressionWrapper
// (:2326-2383: CreateChunkFlags :886-918 -> InclusiveSum -> D2H -> CreateChunkBases :920-954 ->
// CreateChunkSizes :956-991). Semantics kept: trimmed order = slot order; a chunk is a maximal run of
// equal keys in trimmed order; chunk c has key, base (trimmed index of its head) and size.
//
// GB300 form: reduce-then-scan in two launches, with no inter-CTA waiting at all:
//   k_compress_reduce  a fixed number of CTAs share the slots; each warp reduces a contiguous range of whole rows of
//                      32 to the associative summary (valid count, head count, first key, last key);
//   k_compress_write   the same CTAs fold the summaries before theirs, re-read their keys (an L2 hit at frame sizes)
//                      and write trimmed ids, chunk keys and chunk bases.
// A lane takes a slot of each row, and ballots give the places: reads and writes are coalesced without staging
// (16 consecutive slots a thread staged through shared memory, 16-way bank conflicts, and a third launch for the scan
// of the tiles' summaries before: with 2.76 M slots 3 us more of 152 from raygen to the hierarchy). A few hundred
// summaries are cheap for every CTA to fold; a single pass with decoupled look-back spends most of its time in the
// first wave's chain at frame sizes. Bound by issue slots (65% busy), 9 + 13 us. Counts stay on the device.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace rsh {

namespace {
constexpr uint32_t CT_THREADS = 256, CT_WARPS = CT_THREADS / 32;
constexpr uint32_t CT_CTAS = 4 * 152;   // most CTAs: four per SM
constexpr uint32_t CT_BATCH = 16;       // rows whose loads are in flight together

struct Summ {  // summary of a key range: valid count, heads (first valid counted), first/last key
    uint32_t n, h, first, last;
};
RSH_DEV Summ combine(const Summ& a, const Summ& b) {
    Summ r;
    r.n = a.n + b.n;
    r.h = a.h + b.h - ((a.n > 0u && b.n > 0u && a.last == b.first) ? 1u : 0u);
    r.first = a.n > 0u ? a.first : b.first;
    r.last = b.n > 0u ? b.last : a.last;
    return r;
}
RSH_DEV Summ shfl_up(const Summ& s, int d) {
    Summ r;
    r.n = __shfl_up_sync(0xffffffffu, s.n, d);
    r.h = __shfl_up_sync(0xffffffffu, s.h, d);
    r.first = __shfl_up_sync(0xffffffffu, s.first, d);
    r.last = __shfl_up_sync(0xffffffffu, s.last, d);
    return r;
}
RSH_DEV uint4 to4(const Summ& s) { return make_uint4(s.n, s.h, s.first, s.last); }
RSH_DEV Summ from4(const uint4& v) { return Summ{v.x, v.y, v.z, v.w}; }


// The warp's slots [b, e), row by row: f(slot, key, valid lanes, heads) with the lanes that hold a ray and the ones
// that start a chunk, given the last key before (if any). Returns the heads and rays added to n and h; first is set
// at the first ray of the range (`any` false).
struct Range {
    uint32_t n, h, last;
    bool any;
};
RSH_DEV void load_rows(const uint32_t* __restrict__ keys, uint32_t q, uint32_t e, uint32_t (&k)[CT_BATCH]) {
#pragma unroll
    for (uint32_t i = 0; i < CT_BATCH; ++i) {
        const uint32_t s = 32u * i + lane_id();
        k[i] = q < e && s < e - q ? __ldg(keys + q + s) : RSH_KEY_NONE;
    }
}
template <class F>
RSH_DEV void rows(const uint32_t* __restrict__ keys, uint32_t b, uint32_t e, uint32_t (&k)[CT_BATCH], Range& r, F f) {
    const uint32_t lane = lane_id(), below = lanemask_lt();
    for (uint32_t q = b; q < e;) {
        const uint32_t next = e - q > 32u * CT_BATCH ? q + 32u * CT_BATCH : e;
        uint32_t kn[CT_BATCH];
        load_rows(keys, next, e, kn);
#pragma unroll
        for (uint32_t i = 0; i < CT_BATCH; ++i) {
            const bool valid = k[i] != RSH_KEY_NONE;
            const uint32_t v = __ballot_sync(0xffffffffu, valid);
            if (v == 0u) continue;
            const uint32_t vb = v & below;
            const uint32_t before = __shfl_sync(0xffffffffu, k[i], vb ? 31 - __clz(vb) : 0);
            const bool head = valid && (vb ? before != k[i] : !r.any || r.last != k[i]);
            const uint32_t hm = __ballot_sync(0xffffffffu, head);
            f(q + 32u * i + lane, k[i], v, hm, valid, head);
            r.n += __popc(v);
            r.h += __popc(hm);
            r.last = __shfl_sync(0xffffffffu, k[i], 31 - __clz(v));
            r.any = true;
        }
#pragma unroll
        for (uint32_t i = 0; i < CT_BATCH; ++i) k[i] = kn[i];
        q = next;
    }
}

// The slots of a warp: whole rows, the same number for every warp but the last ones.
RSH_DEV void warp_range(uint32_t n_slots, uint32_t ctas, uint32_t& b, uint32_t& e) {
    const uint64_t per = 32ull * (((uint64_t)n_slots + 32ull * CT_WARPS * ctas - 1u) / (32ull * CT_WARPS * ctas));
    const uint64_t x = per * (blockIdx.x * CT_WARPS + (threadIdx.x >> 5));
    b = (uint32_t)min(x, (uint64_t)n_slots);
    e = (uint32_t)min(x + per, (uint64_t)n_slots);
}
}  // namespace

// csumm: a summary per CTA; wsumm: per warp
__global__ void __launch_bounds__(CT_THREADS)
k_compress_reduce(const uint32_t* __restrict__ keys, uint32_t n_slots, uint4* __restrict__ csumm,
                  uint4* __restrict__ wsumm) {
    __shared__ Summ s_warp[CT_WARPS];
    asm volatile("griddepcontrol.launch_dependents;");
    uint32_t b, e;
    warp_range(n_slots, gridDim.x, b, e);
    uint32_t k[CT_BATCH];
    load_rows(keys, b, e, k);
    Range r{0u, 0u, 0u, false};
    uint32_t first = 0u;
    rows(keys, b, e, k, r, [&](uint32_t, uint32_t key, uint32_t v, uint32_t, bool, bool) {
        if (!r.any) first = __shfl_sync(0xffffffffu, key, __ffs(v) - 1);
    });
    const uint32_t warp = threadIdx.x >> 5;
    if (lane_id() == 0u) {
        s_warp[warp] = Summ{r.n, r.h, first, r.last};
        wsumm[blockIdx.x * CT_WARPS + warp] = to4(s_warp[warp]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        Summ t = s_warp[0];
        for (uint32_t w = 1; w < CT_WARPS; ++w) t = combine(t, s_warp[w]);
        csumm[blockIdx.x] = to4(t);
    }
}

__global__ void __launch_bounds__(CT_THREADS)
k_compress_write(const uint32_t* __restrict__ keys, uint32_t n_slots, const uint4* __restrict__ csumm,
                 const uint4* __restrict__ wsumm, uint32_t* __restrict__ trimmed_ids,
                 uint32_t* __restrict__ chunk_keys, uint32_t* __restrict__ chunk_bases,
                 uint32_t* __restrict__ counts) {
    constexpr uint32_t PER = (CT_CTAS + CT_THREADS - 1) / CT_THREADS;
    __shared__ Summ s_fold[CT_WARPS], s_own[CT_WARPS];
    uint32_t b, e, k[CT_BATCH];
    warp_range(n_slots, gridDim.x, b, e);
    load_rows(keys, b, e, k);  // (what the kernel before this one reads too)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    // the CTAs before this one: a few in a row per thread, then in order across the lanes and the warps
    Summ t{0u, 0u, 0u, 0u};
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i) {
        const uint32_t c = threadIdx.x * PER + i;
        if (c < blockIdx.x) t = combine(t, from4(ld_chain(csumm + c)));
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const Summ o = shfl_up(t, d);
        if (lane >= (uint32_t)d) t = combine(o, t);
    }
    if (lane == 31u) s_fold[warp] = t;
    if (threadIdx.x < CT_WARPS) s_own[threadIdx.x] = from4(ld_chain(wsumm + blockIdx.x * CT_WARPS + threadIdx.x));
    __syncthreads();
    Summ pre{0u, 0u, 0u, 0u};
    for (uint32_t w = 0; w < CT_WARPS; ++w) pre = combine(pre, s_fold[w]);
    for (uint32_t w = 0; w < warp; ++w) pre = combine(pre, s_own[w]);
    if (blockIdx.x == gridDim.x - 1u && threadIdx.x == CT_THREADS - 32u) {  // the last warp: the totals
        const Summ all = combine(pre, s_own[warp]);
        counts[0] = all.n;
        counts[1] = all.h;
        chunk_bases[all.h] = all.n;
    }
    Range r{pre.n, pre.h, pre.last, pre.n > 0u};
    const uint32_t below = lanemask_lt();
    rows(keys, b, e, k, r, [&](uint32_t slot, uint32_t key, uint32_t v, uint32_t hm, bool valid, bool head) {
        const uint32_t at = r.n + __popc(v & below), c = r.h + __popc(hm & below);
        if (valid && at < n_slots) trimmed_ids[at] = slot;
        if (head && c < n_slots) {
            chunk_keys[c] = key;
            chunk_bases[c] = at;
        }
    });
}

size_t compress_scratch_bytes(uint32_t n_slots) {
    (void)n_slots;
    return (size_t)CT_CTAS * (1 + CT_WARPS) * sizeof(uint4) + 256;
}

cudaError_t launch_compress(const uint32_t* keys, uint32_t n_slots, uint32_t* trimmed_ids,
                            uint32_t* chunk_keys, uint32_t* chunk_bases, uint32_t* counts,
                            void* scratch, uint32_t* err, cudaStream_t s) {
    (void)err;  // no step of this form waits on another CTA
    if (n_slots == 0) {
        cudaMemsetAsync(counts, 0, 2 * sizeof(uint32_t), s);
        cudaMemsetAsync(chunk_bases, 0, sizeof(uint32_t), s);
        return cudaGetLastError();
    }
    // two rows a warp at least
    const uint32_t ctas = std::min(CT_CTAS, (n_slots - 1u) / (64u * CT_WARPS) + 1u);
    uint4* csumm = static_cast<uint4*>(scratch);
    uint4* wsumm = csumm + ctas;
    k_compress_reduce<<<ctas, CT_THREADS, 0, s>>>(keys, n_slots, csumm, wsumm);
    note_launch();
    const cudaError_t e = launch_chained(true, k_compress_write, ctas, CT_THREADS, 0, s, keys, n_slots, csumm, wsumm,
                                         trimmed_ids, chunk_keys, chunk_bases, counts);
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

__global__ void k_chunk_sizes(const uint32_t* __restrict__ bases, const uint32_t* __restrict__ counts,
                              uint32_t max_chunks, uint32_t* sizes) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t C = counts[1] < max_chunks ? counts[1] : max_chunks;
    if (c >= C) return;
    sizes[c] = bases[c + 1] - bases[c];
}

cudaError_t launch_chunk_sizes(const uint32_t* chunk_bases, const uint32_t* counts, uint32_t max_chunks,
                               uint32_t* chunk_sizes, cudaStream_t s) {
    if (max_chunks == 0) return cudaSuccess;
    k_chunk_sizes<<<(max_chunks + 255) / 256, 256, 0, s>>>(chunk_bases, counts, max_chunks, chunk_sizes);
    note_launch();
    return cudaGetLastError();
}

}  // namespace rsh
