// Shared device helpers for the sm_103a ray-space-hierarchy kernels.
//
// Numerics: the library is compiled with -fmad=false, so every a*b+c below is two rounded IEEE
// operations unless written as an explicit fmaf(). Hash keys, run heads, hierarchy nodes and
// intersection results are therefore reproducible bit for bit by a CPU restatement compiled with
// -ffp-contract=off. Division and square root use the IEEE-rounded defaults (-prec-div/-prec-sqrt).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "../../include/rsh.h"

#define RSH_DEV __device__ __forceinline__

// ------------------------------------------------------------------ small vector math (own)
struct v3 {
    float x, y, z;
};
RSH_DEV v3 mk3(float x, float y, float z) { return v3{x, y, z}; }
RSH_DEV v3 mk3(float4 a) { return v3{a.x, a.y, a.z}; }
RSH_DEV v3 operator+(v3 a, v3 b) { return v3{a.x + b.x, a.y + b.y, a.z + b.z}; }
RSH_DEV v3 operator-(v3 a, v3 b) { return v3{a.x - b.x, a.y - b.y, a.z - b.z}; }
RSH_DEV v3 operator*(v3 a, float s) { return v3{a.x * s, a.y * s, a.z * s}; }
RSH_DEV v3 operator-(v3 a) { return v3{-a.x, -a.y, -a.z}; }
// dot as ((x*x + y*y) + z*z): the fixed evaluation order the CPU restatement uses
RSH_DEV float dot3(v3 a, v3 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }
RSH_DEV v3 cross3(v3 a, v3 b) {
    return v3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
RSH_DEV float len3(v3 a) { return sqrtf(dot3(a, a)); }
// normalize by three IEEE divisions (not a reciprocal multiply), reproducible on the host
RSH_DEV v3 norm3(v3 a) {
    float l = len3(a);
    return v3{a.x / l, a.y / l, a.z / l};
}

// ------------------------------------------------------------------ ray storage
// rsh_ray is 32 bytes: two float4 halves, loaded with 128-bit accesses.
RSH_DEV void load_ray(const rsh_ray* rays, uint32_t i, float4& o, float4& d) {
    const float4* p = reinterpret_cast<const float4*>(rays) + 2ull * i;
    o = __ldg(p);
    d = __ldg(p + 1);
}
RSH_DEV void store_ray(rsh_ray* rays, uint32_t i, float4 o, float4 d) {
    float4* p = reinterpret_cast<float4*>(rays) + 2ull * i;
    p[0] = o;
    p[1] = d;
}
// The same ray as one 256-bit store (st.global.v8.f32, sm_100 and later): each lane writes its whole
// 32-byte sector in one instruction. Only for an array whose base is 32-byte aligned (a32, checked by the
// caller once per thread); otherwise the two 16-byte stores above.
RSH_DEV void store_ray32(rsh_ray* rays, uint32_t i, float4 o, float4 d, bool a32) {
    if (a32) {
        float* p = reinterpret_cast<float*>(rays) + 8ull * i;
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(o.x), "f"(o.y),
                     "f"(o.z), "f"(o.w), "f"(d.x), "f"(d.y), "f"(d.z), "f"(d.w)
                     : "memory");
    } else {
        store_ray(rays, i, o, d);
    }
}

// ------------------------------------------------------------------ device error word
// Bounded device waits and overflow checks report here (never __trap()); the host reads it back with
// rsh_check_device_errors. Bits: 1 = look-back timeout, 2 = overflow.
#ifndef RSH_DEVERR_TIMEOUT
#define RSH_DEVERR_TIMEOUT 1u
#define RSH_DEVERR_OVERFLOW 2u
#endif
#define RSH_SPIN_LIMIT (1u << 22)   // polls before a look-back wait gives up (~0.1-1 s)

RSH_DEV void raise_device_error(uint32_t* err, uint32_t bit) {
    if (err) atomicOr(err, bit);
}

RSH_DEV uint32_t ld_acquire_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
RSH_DEV void st_release_u32(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
RSH_DEV void st_relaxed_u32(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
RSH_DEV uint32_t ld_relaxed_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
RSH_DEV unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

RSH_DEV uint32_t lane_id() { return threadIdx.x & 31u; }
RSH_DEV uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

RSH_DEV void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Decoupled look-back over tiles that each contribute two counts (a, b < 2^24), packed a | b << 24; one status
// word per tile holds a state, an epoch (words of an earlier launch over the same array do not count, so the
// array is cleared once per 2^14 launches, not per launch) and the packed counts. Called by one whole warp of
// the tile's block, with the tile's own sum; returns the sum over the tiles before it. Tiles are taken by
// ticket, so every earlier tile is running or done. A wait that gives up raises RSH_DEVERR_TIMEOUT, publishes
// LB_DEAD, which every later tile passes on, and returns LB_FAILED: the caller then writes nothing.
constexpr unsigned long long LB_COUNTS = (1ull << 48) - 1ull;
constexpr unsigned long long LB_FAILED = ~0ull;
constexpr uint32_t LB_SUM = 1u, LB_PREFIX = 2u, LB_DEAD = 3u;
constexpr uint32_t LB_EPOCHS = 1u << 14;
RSH_DEV unsigned long long look_back2(unsigned long long* status, uint32_t tile, unsigned long long sum,
                                      uint32_t epoch, uint32_t* err) {
    const uint32_t lane = lane_id();
    auto word = [&](uint32_t state, unsigned long long v) {
        return ((unsigned long long)state << 62) | ((unsigned long long)epoch << 48) | v;
    };
    if (tile == 0u) {
        if (lane == 0) st_relaxed_u64(status, word(LB_PREFIX, sum));
        return 0ull;
    }
    if (lane == 0) st_relaxed_u64(status + tile, word(LB_SUM, sum));
    unsigned long long excl = 0ull;
    int64_t j = (int64_t)tile - 1;  // newest tile not yet added
    uint32_t spins = 0;
    bool dead = false;
    for (;;) {
        const int64_t q = j - (int64_t)lane;
        const unsigned long long v = q >= 0 ? ld_relaxed_u64(status + q) : word(LB_PREFIX, 0ull);
        const bool ready = ((uint32_t)(v >> 48) & (LB_EPOCHS - 1u)) == epoch && (v >> 62) != 0ull;
        const uint32_t state = (uint32_t)(v >> 62);
        const uint32_t waiting = __ballot_sync(0xffffffffu, !ready);
        const uint32_t stops = __ballot_sync(0xffffffffu, ready && state != LB_SUM);
        // the lanes to add: up to the first prefix, or up to the first tile still to wait for
        const uint32_t first_stop = stops ? (uint32_t)__ffs(stops) - 1u : 32u;
        const uint32_t first_wait = waiting ? (uint32_t)__ffs(waiting) - 1u : 32u;
        const bool found = first_stop < first_wait;
        const uint32_t upto = found ? first_stop + 1u : min(first_wait, 32u);
        unsigned long long add = lane < upto ? v & LB_COUNTS : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
        excl += add;
        if (found) {
            dead = __shfl_sync(0xffffffffu, state, (int)first_stop) == LB_DEAD;
            break;
        }
        j -= (int64_t)upto;
        if (waiting) {
            if (++spins > RSH_SPIN_LIMIT) {
                if (lane == 0) raise_device_error(err, RSH_DEVERR_TIMEOUT);
                dead = true;
                break;
            }
            if (spins > 16u) __nanosleep(32);
        }
    }
    if (lane == 0) st_relaxed_u64(status + tile, dead ? word(LB_DEAD, 0ull) : word(LB_PREFIX, (excl + sum) & LB_COUNTS));
    return dead ? LB_FAILED : excl;
}

// First in every kernel that launch_chained launches: the next one's CTAs may be placed from here on, and what the one
// before wrote may be read (all its CTAs are done; a kernel that skipped the wait could be done before it).
// The rule of a chained kernel's loads: what another kernel of the chain writes -- while this one's CTAs may already be
// resident -- is read with ld_chain, or plainly through a pointer that is not const __restrict__. A read-only load
// (__ldg, or a plain one through a const __restrict__ pointer) is taken to read memory that nothing writes while the
// kernel lives: it may be moved above the wait and may be served from an L1 line older than the write. Data complete
// before the chain's first kernel starts (scenes, the sort's and the compression's input keys) may be read either way.
RSH_DEV void chain() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// A load of what an earlier kernel of the chain wrote: coherent whatever the pointer's qualifiers, and, being volatile
// like the wait, never above it. (Not for what this kernel itself writes.)
template <class T>
RSH_DEV T ld_chain(const T* p) {
    static_assert(sizeof(T) == 4 || sizeof(T) == 8 || sizeof(T) == 16, "one load");
    T r;
    if constexpr (sizeof(T) == 4) {
        uint32_t v;
        asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
        memcpy(&r, &v, 4);
    } else if constexpr (sizeof(T) == 8) {
        unsigned long long v;
        asm volatile("ld.global.b64 %0, [%1];" : "=l"(v) : "l"(p));
        memcpy(&r, &v, 8);
    } else {
        uint4 v;
        asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
        memcpy(&r, &v, 16);
    }
    return r;
}
RSH_DEV void load_ray_chain(const rsh_ray* rays, uint32_t i, float4& o, float4& d) {
    const float4* p = reinterpret_cast<const float4*>(rays) + 2ull * i;
    o = ld_chain(p);
    d = ld_chain(p + 1);
}

// device count helper: n = *d_count when given (clamped to n_max), else n_max
RSH_DEV uint32_t dev_count(const uint32_t* d_count, uint32_t n_max) {
    if (!d_count) return n_max;
    uint32_t n = *d_count;
    return n < n_max ? n : n_max;
}

// ------------------------------------------------------------------ Morton interleaving
RSH_DEV uint32_t spread3(uint32_t v) {  // 10 bits -> every third bit
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}
RSH_DEV uint32_t spread2(uint32_t v) {  // 16 bits -> every second bit
    v &= 0xFFFFu;
    v = (v | (v << 8)) & 0x00FF00FFu;
    v = (v | (v << 4)) & 0x0F0F0F0Fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}
