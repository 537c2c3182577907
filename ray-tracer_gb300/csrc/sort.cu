// Stable LSD radix sort of (u32 key, u32 value) pairs, onesweep form (Adinets & Merrill 2022).
//
// Reference: RaySortingWrapper -> cub::DeviceRadixSort::SortPairs over all 32 key bits
// (RayTracer.cu:2385-2409, temp storage sized at :2127-2139). Here: our own kernels, and only the
// ceil(key_bits / 8) digit passes the hash actually uses.
//
//  1. one histogram kernel reads the keys once and builds all passes' 256-bin digit histograms; its last
//     CTA turns them into per-pass exclusive digit offsets;
//  2. one kernel per 8-bit digit pass: each CTA takes a tile by atomic ticket, ranks its keys stably (the lanes
//     of a row of 32 keys find the others of their digit through a lane mask in shared memory, per warp and
//     digit beside the count so far), publishes its per-digit counts, scatters keys and values into shared
//     memory in digit order, resolves the per-digit exclusive prefix over earlier tiles by decoupled look-back
//     (bounded spin), and writes runs of one digit. A status word holds flag and count together and nothing else
//     is read through it, so it is published and read with relaxed (not release / acquire) accesses: no memory
//     barrier per tile. The passes are chained (programmatic dependent launch): a pass's CTAs are placed as the
//     ones before it leave.
// What bounds a pass: at 16 M random pairs 102 us (2.5 TB/s of its 16 B a pair), with the shared-memory pipe at
// 70%: a row of 32 keys costs about 44 of its cycles (random banks: ranking, counters, scatter). Eight ballots a
// key instead of the lane mask were bound by issue slots (139 us a pass at 24 warps an SM; alternating the two
// row by row 103 us). 16 M random 31-bit pairs: 625 us before, now 423; 20,000: 54 -> 33.5.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace rsh {

namespace {
constexpr uint32_t FLAG_AGG = 1u << 30;
constexpr uint32_t FLAG_PRE = 2u << 30;
constexpr uint32_t VAL_MASK = (1u << 30) - 1u;
constexpr uint32_t SW_T = 512, SW_I = 14, SW_MIN = 2;  // threads, most and fewest rows of T keys a tile
constexpr int SW_MB = 2;                                // CTAs per SM
// Rows of a tile, from the actual count, which a kernel knows and the host may not: as many as make one tile a CTA,
// within the limits. Large tiles give long runs of one digit in the output and few tiles to look back over; small
// ones leave no SM without a tile. us, against 2048-key tiles up to 512 K pairs of capacity and 7168-key tiles above:
// 320,000 random pairs 53 -> 48, 600,000 of a capacity of 2.76 M 70 -> 60, 50,000 of it 63 -> 38; the same at 20,000
// and 16 M. From SW_NEAR rows on all SW_I: nearly as few idle SMs, and nothing to check row by row.
constexpr uint32_t SW_NEAR = 11;
__host__ __device__ __forceinline__ uint32_t tile_rows(uint32_t n, uint32_t ctas) {
    const uint32_t r = (uint32_t)(((uint64_t)n + (uint64_t)ctas * SW_T - 1u) / ((uint64_t)ctas * SW_T));
    return r < SW_MIN ? SW_MIN : r >= SW_NEAR ? SW_I : r;
}
// The CTAs of a pass for up to n_max keys on `sms` SMs: one a tile and SM while the tiles that gives hold the keys
// (a tile that shares its SM ends last), else as many as are resident at once.
inline uint32_t sweep_ctas(uint32_t n_max, uint32_t sms) {
    return n_max <= sms * SW_T * SW_I ? std::min(sms, (n_max + SW_T * SW_MIN - 1) / (SW_T * SW_MIN))
                                      : sms * (uint32_t)SW_MB;
}
inline size_t most_tiles(uint32_t n_max, uint32_t ctas) {
    return std::max<size_t>(ctas, (n_max + SW_T * SW_I - 1) / (SW_T * SW_I)) + 1;
}
inline uint32_t sm_count() {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (uint32_t)sms;
}
inline uint32_t num_passes(uint32_t key_bits) { return key_bits == 0 ? 1u : (key_bits + 7u) / 8u; }
}  // namespace

__global__ void k_sort_zero(uint32_t* __restrict__ w) {
    asm volatile("griddepcontrol.launch_dependents;");
    w[blockIdx.x * blockDim.x + threadIdx.x] = 0u;
}

// --- histograms of every pass in one read; also clears the look-back status rows of the tiles that
// the passes will use (ceil(n / tile) rows of 256 words per pass, pass stride `stride` words)
__global__ void k_sort_hist(const uint32_t* __restrict__ keys, uint32_t n_max,
                            const uint32_t* __restrict__ d_count, uint32_t passes, uint32_t ctas,
                            uint32_t* __restrict__ hist, uint32_t* __restrict__ status, size_t stride,
                            uint32_t* __restrict__ done) {
    __shared__ uint32_t sh[4][256];
    __shared__ uint32_t s_last;
    asm volatile("griddepcontrol.launch_dependents;");
    for (uint32_t i = threadIdx.x; i < 4u * 256u; i += blockDim.x) (&sh[0][0])[i] = 0u;
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the zeroed counters (k_sort_zero)
    const uint32_t n = dev_count(d_count, n_max);
    {
        const uint32_t tile_keys = SW_T * tile_rows(n, ctas);
        const size_t words = (size_t)((n + tile_keys - 1) / tile_keys) * 256u;  // multiple of 4
        const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (size_t)gridDim.x * blockDim.x;
        for (uint32_t p = 0; p < passes; ++p) {
            uint4* row = reinterpret_cast<uint4*>(status + p * stride);
            for (size_t i = tid; i < words / 4; i += nth) row[i] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    // each thread counts a contiguous run of keys and adds equal consecutive digits up before one shared
    // atomic: the keys arrive coherent (hash runs in ray order), so their upper digits repeat in long runs
    // that would otherwise pile up on one shared counter. The run is loaded once into registers (four
    // 16-byte loads when the keys are 16-byte aligned) and every pass counts from there: one 4-byte load
    // per key and pass, with the lanes' runs 64 bytes apart, kept the L1 busy a line per lane.
    {
        constexpr uint32_t RUN = 16;
        const uint32_t nth = gridDim.x * blockDim.x;
        const bool a16 = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0u;
        for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) * RUN; base < n; base += nth * RUN) {
            const uint32_t cnt = min(n - base, RUN);
            uint32_t k[RUN];
            if (a16 && cnt == RUN) {
                const uint4* q = reinterpret_cast<const uint4*>(keys + base);
#pragma unroll
                for (uint32_t j = 0; j < RUN / 4u; ++j) {
                    const uint4 v = __ldg(q + j);
                    k[4u * j] = v.x;
                    k[4u * j + 1u] = v.y;
                    k[4u * j + 2u] = v.z;
                    k[4u * j + 3u] = v.w;
                }
            } else {
#pragma unroll
                for (uint32_t i = 0; i < RUN; ++i) k[i] = i < cnt ? __ldg(keys + base + i) : 0u;
            }
            for (uint32_t p = 0; p < passes; ++p) {
                const uint32_t sh_p = 8u * p;
                uint32_t prev = (k[0] >> sh_p) & 255u, run = 0;
#pragma unroll
                for (uint32_t i = 0; i < RUN; ++i) {
                    if (i < cnt) {
                        const uint32_t d = (k[i] >> sh_p) & 255u;
                        if (d != prev) {
                            atomicAdd(&sh[p][prev], run);
                            prev = d;
                            run = 0;
                        }
                        ++run;
                    }
                }
                atomicAdd(&sh[p][prev], run);
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < passes * 256u; i += blockDim.x) {
        const uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(hist + i, v);
    }
    // the last CTA to finish turns the counts into exclusive digit offsets, in place
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(done, 1u) == gridDim.x - 1u) ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // exclusive digit offsets: a block-wide scan of the 256 bins, of all passes at once
    {
        const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;  // blockDim.x == 256
        uint32_t v[4], x[4];
#pragma unroll
        for (uint32_t p = 0; p < 4; ++p) v[p] = x[p] = p < passes ? __ldcg(hist + 256u * p + t) : 0u;
#pragma unroll
        for (uint32_t p = 0; p < 4; ++p) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x[p], o);
                if (lane >= (uint32_t)o) x[p] += y;
            }
            if (lane == 31u) sh[p][warp] = x[p];  // the shared counters are free now
        }
        __syncthreads();
#pragma unroll
        for (uint32_t p = 0; p < 4; ++p) {
            uint32_t before = 0;
            for (uint32_t w = 0; w < warp; ++w) before += sh[p][w];
            if (p < passes) hist[256u * p + t] = before + x[p] - v[p];
        }
    }
}

// One digit pass. T threads, up to I keys a thread; MB CTAs per SM.
template <int T, int I>
struct SweepSmem {
    uint32_t keys[T * I];
    uint32_t vals[T * I];
    // per warp and digit, while ranking: (count so far, lanes of the row at hand) in one 64-bit word; then, in
    // the counts' place, the tile-local position of each warp's run
    uint2 rk[T / 32][256];
    uint32_t gbase[256];             // global position of the tile's first key of a digit, less its local one
    uint32_t scan[8];
    uint32_t tile, next;
};

// FULL: every tile has I rows (known before the launch: no count on the device).
template <int T, int I, int MB, bool FULL>
__global__ void __launch_bounds__(T, MB)
k_onesweep(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
           uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n_max,
           const uint32_t* __restrict__ d_count, uint32_t shift, const uint32_t* __restrict__ hist,
           uint32_t* __restrict__ status, uint32_t* __restrict__ ticket, uint32_t* err, uint32_t spin_limit,
           uint32_t ctas) {
    constexpr uint32_t W = T / 32;
    static_assert(T >= 256, "a thread per digit");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SweepSmem<T, I>& S = *reinterpret_cast<SweepSmem<T, I>*>(smem_raw);
    // the next pass may take this one's place CTA by CTA; this one reads what the kernel before it wrote only
    // once that is complete (a no-op in a launch that is not chained)
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t n = dev_count(d_count, n_max);
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const uint32_t rows = FULL ? I : tile_rows(n, ctas), TILE = T * rows;
    const uint32_t num_tiles = (n + TILE - 1) / TILE;
    uint2* rk = S.rk[warp];
    uint32_t key[I];
    auto load_keys = [&](uint32_t t) {
        if (t >= num_tiles) return;
        const uint32_t b = t * TILE + warp * (rows * 32u) + lane;
        const bool whole = t * TILE + TILE <= n;
#pragma unroll
        for (int j = 0; j < I; ++j)
            if (FULL || (uint32_t)j < rows) key[j] = whole || b + j * 32u < n ? ld_chain(keys_in + b + j * 32u) : 0xFFFFFFFFu;
    };
    if (tid == 0) S.tile = atomicAdd(ticket, 1u);
    __syncthreads();
    uint32_t tile = S.tile;
    load_keys(tile);
    // tiles by ticket until none is left (the grid is capped at the resident CTAs); the next tile's keys are
    // loaded while this one waits for its prefix and is written out
    while (tile < num_tiles) {
        if (tid == 0) S.next = atomicAdd(ticket, 1u);
        {
            uint4* z = reinterpret_cast<uint4*>(&S.rk[0][0]);
            for (uint32_t i = tid; i < W * 128u; i += T) z[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();
        const uint32_t base = tile * TILE, wbase = base + warp * (rows * 32u);
        const bool full = base + TILE <= n;  // the whole tile holds valid items
        // stable in-warp ranking: items in (j, lane) order = index order. The lanes of a digit find each other
        // through a lane mask in shared memory
        uint32_t rank[(I + 1) / 2];  // two 16-bit ranks a word
#pragma unroll
        for (int j = 0; j < I; ++j) {
            if (!FULL && (uint32_t)j >= rows) break;
            const bool valid = full || wbase + j * 32u + lane < n;
            const uint32_t d = (key[j] >> shift) & 255u;
            if (valid) atomicOr(&rk[d].y, 1u << lane);
            __syncwarp();
            const uint2 e = rk[d];
            const uint32_t before = e.y & lanemask_lt();
            __syncwarp();
            if (valid && before == 0u) rk[d] = make_uint2(e.x + __popc(e.y), 0u);
            __syncwarp();
            const uint32_t r = e.x + __popc(before);
            if (j & 1) rank[j / 2] |= r << 16;
            else rank[j / 2] = r;
        }
        __syncthreads();
        // per digit (thread = digit): warp-exclusive offsets and the tile count, published early so that
        // successors can proceed
        uint32_t tcount = 0u, start = 0u;
        uint32_t* st = status + (size_t)tile * 256u + tid;
        uint32_t x = 0u;
        if (tid < 256u) {
#pragma unroll
            for (uint32_t w = 0; w < W; ++w) {
                const uint32_t c = S.rk[w][tid].x;
                S.rk[w][tid].x = tcount;
                tcount += c;
            }
            st_relaxed_u32(st, (tile == 0 ? FLAG_PRE : FLAG_AGG) | tcount);
            x = tcount;  // exclusive scan over the digits
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= (uint32_t)d) x += y;
            }
            if (lane == 31) S.scan[warp] = x;
        }
        __syncthreads();
        if (tid < 256u) {
            start = x - tcount;
            for (uint32_t w = 0; w < warp; ++w) start += S.scan[w];
#pragma unroll
            for (uint32_t w = 0; w < W; ++w) S.rk[w][tid].x += start;
        }
        __syncthreads();
        // scatter into shared memory in tile-sorted order (before the look-back, whose predecessors gain time)
        {
            uint32_t val[I];
#pragma unroll
            for (int j = 0; j < I; ++j) {
                if (!FULL && (uint32_t)j >= rows) break;
                const uint32_t idx = wbase + j * 32u + lane;
                val[j] = idx;
                if (vals_in && (full || idx < n)) val[j] = ld_chain(vals_in + idx);
            }
#pragma unroll
            for (int j = 0; j < I; ++j) {
                if (!FULL && (uint32_t)j >= rows) break;
                if (full || wbase + j * 32u + lane < n) {
                    const uint32_t pos = rk[(key[j] >> shift) & 255u].x + ((rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu);
                    S.keys[pos] = key[j];
                    S.vals[pos] = val[j];
                }
            }
        }
        const uint32_t next = S.next;
        load_keys(next);
        if (tid < 256u) {
            // global digit offset of this pass (exclusive, from the histogram kernel)
            const uint32_t gex = ld_chain(hist + tid);
            // decoupled look-back for this digit, LB predecessors per step: their status words are loaded
            // together (flag and count share one word, so relaxed loads suffice) and folded newest first up to
            // the first one holding an inclusive prefix; a not-yet-published word restarts the step there
            uint32_t excl = 0u;
            if (tile > 0) {
                constexpr int LB = 8;
                int64_t j = (int64_t)tile - 1;
                uint32_t spins = 0;
                while (j >= 0) {
                    uint32_t sv[LB];
#pragma unroll
                    for (int q = 0; q < LB; ++q)
                        sv[q] = (j - q >= 0) ? ld_relaxed_u32(status + (size_t)(j - q) * 256u + tid) : FLAG_PRE;
                    int used = 0;
                    bool done = false, stall = false;
#pragma unroll
                    for (int q = 0; q < LB; ++q) {
                        if (done || stall) continue;
                        const uint32_t f = sv[q] & ~VAL_MASK;
                        if (f == 0u) {
                            stall = true;
                            continue;
                        }
                        excl += sv[q] & VAL_MASK;
                        ++used;
                        if (f == FLAG_PRE) done = true;
                    }
                    if (done) break;
                    j -= used;
                    if (stall) {
                        if (++spins > spin_limit) {
                            raise_device_error(err, RSH_DEVERR_TIMEOUT);
                            break;
                        }
                        if (spins > 16) __nanosleep(32);
                    }
                }
                st_relaxed_u32(st, FLAG_PRE | (excl + tcount));
            }
            S.gbase[tid] = gex + excl - start;
        }
        __syncthreads();
        const uint32_t tn = full ? TILE : n - base;
#pragma unroll 4
        for (uint32_t i = tid; i < tn; i += T) {
            const uint32_t k = S.keys[i];
            const uint32_t g = S.gbase[(k >> shift) & 255u] + i;
            if (g < n) {  // only false after a look-back timeout (error word raised)
                if (keys_out) keys_out[g] = k;
                vals_out[g] = S.vals[i];
            }
        }
        __syncthreads();  // shared state is reused by the next tile
        tile = next;
    }
}

namespace {

// One pass over up to n_max keys: `ctas` CTAs (at most those resident at once: every ticket below a CTA's tile is
// held by a running CTA, which is the look-back's forward progress).
cudaError_t sweep(uint32_t n_max, uint32_t sms, uint32_t ctas, uint32_t grid, bool chained, const uint32_t* ki,
                  const uint32_t* vi, uint32_t* ko, uint32_t* vo, const uint32_t* d_count, uint32_t shift,
                  const uint32_t* hist, uint32_t* status, uint32_t* ticket, uint32_t* err, uint32_t spin_limit,
                  cudaStream_t s) {
    const auto kernel = !d_count && tile_rows(n_max, ctas) == SW_I ? k_onesweep<(int)SW_T, (int)SW_I, SW_MB, true>
                                                                   : k_onesweep<(int)SW_T, (int)SW_I, SW_MB, false>;
    constexpr size_t smem = sizeof(SweepSmem<(int)SW_T, (int)SW_I>), MOST = 227 * 1024;
    static_assert(SW_MB * (smem + 1024) <= 228 * 1024, "SW_MB CTAs fit an SM");
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MOST);
    if (e != cudaSuccess) return e;
    // A chained launch's CTAs are placed while the pass before it still runs, on whichever SMs have room: with
    // room for more CTAs than an SM's share, some SMs get several and others none. With no more CTAs than SMs,
    // asking for an SM's shared memory leaves room for one (1 M random pairs: 61 us, 71 unchained, 75 chained
    // without this; 16 M: 428 / 440).
    e = launch_chained(chained, kernel, grid, SW_T, ctas <= sms ? MOST : smem, s, ki, vi, ko, vo, n_max, d_count, shift,
                       hist, status, ticket, err, spin_limit, ctas);
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

size_t sort_scratch_bytes(uint32_t n_max, uint32_t key_bits) {
    const size_t passes = num_passes(key_bits);
    const size_t words = 4 * 256 + 16 + passes * most_tiles(n_max, sweep_ctas(n_max, sm_count())) * 256;
    return words * 4 + 2 * (size_t)n_max * 4 + 1024;
}

cudaError_t launch_sort_pairs(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                              uint32_t* vals_out, uint32_t n_max, const uint32_t* d_count,
                              uint32_t key_bits, void* scratch, uint32_t* err, cudaStream_t s, bool keys_wanted) {
    if (n_max == 0) return cudaSuccess;
    const uint32_t passes = num_passes(key_bits);
    const uint32_t sms = sm_count(), ctas = sweep_ctas(n_max, sms);
    const size_t tiles = most_tiles(n_max, ctas);
    uint32_t* w = static_cast<uint32_t*>(scratch);
    uint32_t* hist = w;                       // passes * 256 (room for 4)
    uint32_t* tickets = w + 4 * 256;          // 16: one per pass, [8] = histogram CTAs done
    uint32_t* status = tickets + 16;          // passes * tiles * 256
    uint32_t* alt_keys = status + passes * tiles * 256;
    alt_keys = reinterpret_cast<uint32_t*>((reinterpret_cast<uintptr_t>(alt_keys) + 255) & ~uintptr_t(255));
    uint32_t* alt_vals = alt_keys + n_max;
    // a kernel, not a memset: the next launch can be chained behind it (20,000 pairs 34.9 -> 33.5 us, 1 M 58.6 ->
    // 56.9)
    k_sort_zero<<<5, 208, 0, s>>>(w);
    note_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // four CTAs per SM count 16 M keys in half the time of two; fewer when there is not a run of 16 keys for each
    // thread
    const uint32_t hgrid = std::min<uint32_t>(sms * 4u, (n_max + 4095u) / 4096u);
    e = launch_chained(true, k_sort_hist, hgrid, 256, 0, s, keys_in, n_max, d_count, passes, ctas, hist, status, tiles * 256,
                       tickets + 8);
    note_launch();
    if (e != cudaSuccess) return e;
    // ping-pong so that the last pass lands in the output
    const uint32_t* ki = keys_in;
    const uint32_t* vi = vals_in;
    for (uint32_t p = 0; p < passes; ++p) {
        // choose destinations: passes alternate between out and alt, ending in out
        const bool to_out = ((passes - 1 - p) % 2u) == 0u;
        uint32_t* ko = to_out ? keys_out : alt_keys;
        uint32_t* vo = to_out ? vals_out : alt_vals;
        if (p + 1 == passes && !keys_wanted) ko = nullptr;
        e = sweep(n_max, sms, ctas, ctas, true, ki, vi, ko, vo, d_count, 8u * p, hist + 256u * p,
                  status + p * tiles * 256, tickets + p, err, RSH_SPIN_LIMIT, s);
        if (e != cudaSuccess) return e;
        ki = ko;
        vi = vo;
    }
    return cudaSuccess;
}

constexpr uint32_t SELF_TILE = SW_T * SW_MIN;  // two tiles for two CTAs: of the fewest rows

// Self-test of the bounded look-back wait: one sort pass over two tiles whose first tile is never run
// (its ticket is taken before the launch), so the second tile waits on a status word that nothing
// publishes. The wait must give up after `spin_limit` polls and raise RSH_DEVERR_TIMEOUT in *err
// instead of hanging; every write stays in bounds. Buffers (2 tiles of keys in/out, status, tickets)
// come from the caller's scratch of sort_selftest_scratch_bytes().
size_t sort_selftest_scratch_bytes() { return (size_t)(4 * 2 * SELF_TILE + 2 * 256 + 256 + 8) * 4 + 1024; }

cudaError_t sort_selftest_timeout(void* scratch, uint32_t* err, uint32_t spin_limit, cudaStream_t s) {
    uint32_t* w = static_cast<uint32_t*>(scratch);
    const uint32_t n = 2 * SELF_TILE;
    uint32_t* keys_in = w;
    uint32_t* vals_in = keys_in + n;
    uint32_t* keys_out = vals_in + n;
    uint32_t* vals_out = keys_out + n;
    uint32_t* status = vals_out + n;      // 2 tiles x 256 digits, all "not yet published"
    uint32_t* hist = status + 2 * 256;    // 256 exclusive digit offsets: all 0 (every key is digit 0)
    uint32_t* ticket = hist + 256;
    cudaError_t e = cudaMemsetAsync(w, 0, sort_selftest_scratch_bytes() - 1024, s);
    if (e != cudaSuccess) return e;
    const uint32_t one = 1u;  // tile 0's ticket is already gone: the one CTA gets tile 1
    if ((e = cudaMemcpyAsync(ticket, &one, 4, cudaMemcpyHostToDevice, s)) != cudaSuccess) return e;
    e = sweep(n, sm_count(), 2u, 1u, false, keys_in, vals_in, keys_out, vals_out, nullptr, 0u, hist, status, ticket, err,
              spin_limit, s);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(s);
}

}  // namespace rsh
