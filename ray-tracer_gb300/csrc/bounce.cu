// A frame's work between two traversals, in one kernel: everything a pixel needs there -- shading of the surface
// whose shadow rays have been traced, resolving the hit that is the next surface, that surface's shadow and
// reflection rays and their lists -- depends on that pixel alone.
//
// Reference: the stages between two castRays calls, one wrapper each (colorShadowRays / createReflectionRays /
// colorReflectionRays, main.cpp:685-1054). As separate kernels (resolve, two ray generations, shading, packing)
// each re-read what the one before it wrote: 112 bytes a pixel and bounce of surface and ray, and 5 launches a
// bounce. In one kernel the surface and the incident direction stay in registers.
// What bounds it: memory traffic (a 4-light bounce of the 1080p architecture frame moves about 290 bytes a pixel)
// and, with shading, its divides and powf. 10 CTAs an SM and a surface's shadow flags loaded together instead of light
// by light: that frame 2.74 -> 2.71 ms.
#include "common.cuh"
#include "kernels.h"
#include "pixel.cuh"

namespace rsh {

namespace {
constexpr uint32_t BT = 128;

// SHADE: shade the surface a.sh.spos / snrm; GEN: write the rays of the resolved surface; FINAL: shade the
// resolved surface too, unshadowed, and pack the image.
template <bool SHADE, bool GEN, bool FINAL>
__global__ void __launch_bounds__(BT, 10) k_bounce(const __grid_constant__ BounceArgs a) {
    __shared__ rsh_light s_light[8];
    __shared__ float s_lp[8 * 3];
    __shared__ uint32_t s_bal[BT / 32][8 * 16];  // per warp and light sample: the lanes with a ray
    __shared__ uint32_t s_cnt[2][BT / 32];
    asm volatile("griddepcontrol.launch_dependents;");
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    if (SHADE || FINAL) stage_lights(a.sh, s_light);
    if (GEN && threadIdx.x < 3u * a.lights.count) s_lp[threadIdx.x] = (&a.lights.pos[0][0])[threadIdx.x];
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!GEN && blockIdx.x == 0)
        for (int q = 0; q < 2; ++q) {
            for (uint32_t i = threadIdx.x; i < a.counters.n[q]; i += BT) a.counters.to[q][i] = ld_chain(a.counters.p[q] + i);
            __syncthreads();  // one after the other, like copies in a stream
        }
    const uint32_t pix = blockIdx.x * BT + threadIdx.x, w = a.w;
    const bool in_range = pix < w * a.h;
    const uint32_t y = pix / w, x = pix - y * w;
    // ---- the ray that was traced and its hit
    const uint32_t k = a.tiles_x ? primary_of_pixel(x, y, a.tiles_x, a.tiles_y) : pix;
    const unsigned long long h = in_range ? a.hits[k] : RSH_HIT_NONE;
    float4 ro = make_float4(0.f, 0.f, 0.f, 0.f), rd = ro, sp, sn;
    if (h != RSH_HIT_NONE) load_ray_chain(a.rays, k, ro, rd);
    // ---- shading of the surface the ray left
    float4 acc = make_float4(0.f, 0.f, 0.f, 1.f);
    if (SHADE && in_range) {
        if (a.sh.bounce > 0) acc = a.sh.accum[pix];
        const float4 p4 = a.sh.spos[pix];
        if (p4.w != 0.0f && acc.w > 0.0f) {
            v3 inc;
            if (a.sh.incident) {
                float4 io, id;
                load_ray_chain(a.sh.incident, pix, io, id);
                inc = mk3(id);
            } else {
                inc = norm3(mk3(p4) - v3{a.sh.eye[0], a.sh.eye[1], a.sh.eye[2]});
            }
            shade_surface(a.sh, s_light, a.sh.shadow, x, y, p4, a.sh.snrm[pix], inc, acc);
        } else {
            acc.w = 0.0f;
        }
        if (!FINAL) a.sh.accum[pix] = acc;
    }
    // ---- the next surface
    resolve_hit(a.pos, a.nrm, a.mat, ro, rd, h, sp, sn);
    const bool surface = sp.w != 0.0f;
    if (in_range && a.spos) {
        a.spos[pix] = sp;
        a.snrm[pix] = sn;
    }
    // its incident direction: the camera's for the primary surface, else the ray's
    const v3 p = mk3(sp);
    const bool camera = a.tiles_x != 0u;
    if (FINAL && in_range) {
        if (surface && acc.w > 0.0f) {
            const v3 inc = camera ? norm3(p - v3{a.sh.eye[0], a.sh.eye[1], a.sh.eye[2]}) : mk3(rd);
            shade_surface(a.sh, s_light, nullptr, x, y, sp, sn, inc, acc);
        }
        a.rgba[pix] = pack_rgba(acc);
    }
    if (!GEN) return;
    // ---- its shadow and reflection rays
    const bool s32 = (reinterpret_cast<uintptr_t>(a.srays) & 31u) == 0u, r32 = (reinterpret_cast<uintptr_t>(a.rrays) & 31u) == 0u;
    const v3 nn = surface ? norm3(mk3(sn)) : v3{0.f, 0.f, 0.f};
    const uint32_t S = a.lights.samples ? a.lights.samples : 1u, V = a.lights.count * S;
    uint32_t nshadow = 0;  // the warp's shadow rays
    for (uint32_t v = 0; v < V; ++v) {
        const uint32_t slot = x + w * (v + V * y), l = S == 1u ? v : v / S, sm = S == 1u ? 0u : v % S;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f), d = make_float4(0.f, 0.f, 0.f, -1.f);
        const bool valid =
            surface && shadow_ray(p, nn, mk3(s_lp[3u * l], s_lp[3u * l + 1u], s_lp[3u * l + 2u]), a.eps, S, sm, o, d);
        if (in_range) {
            store_ray32(a.srays, slot, o, d, s32);
            a.sflags[slot] = 0u;
        }
        const uint32_t b = __ballot_sync(0xffffffffu, valid);
        nshadow += __popc(b);
        if (lane == 0) s_bal[warp][v] = b;
    }
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f), d = make_float4(0.f, 0.f, 0.f, -1.f);
    bool reflects = false;
    if (surface) {
        const v3 i = camera ? norm3(p - v3{a.eye[0], a.eye[1], a.eye[2]}) : mk3(rd);
        reflects = reflect_ray(p, nn, i, a.eps, a.jitter, a.seed, pix, a.bounce, o, d);
    }
    if (in_range) {
        store_ray32(a.rrays, pix, o, d, r32);
        a.rhits[pix] = RSH_HIT_NONE;
    }
    const uint32_t br = __ballot_sync(0xffffffffu, reflects);
    if (lane == 0) {
        s_cnt[0][warp] = nshadow;
        s_cnt[1][warp] = __popc(br);
    }
    __syncthreads();
    // the block's place in both lists: one atomic each, by two threads at once
    __shared__ uint32_t s_at[2];
    if (threadIdx.x < 2u) {
        uint32_t all = 0;
        for (uint32_t q = 0; q < BT / 32; ++q) all += s_cnt[threadIdx.x][q];
        s_at[threadIdx.x] = all ? atomicAdd(threadIdx.x ? a.rcount : a.scount, all) : 0u;
    }
    __syncthreads();
    uint32_t at = s_at[0], rat = s_at[1];
    for (uint32_t q = 0; q < warp; ++q) {
        at += s_cnt[0][q];
        rat += s_cnt[1][q];
    }
    if (reflects) a.rids[rat + __popc(br & lanemask_lt())] = pix;
    for (uint32_t v = 0; v < V; ++v) {
        const uint32_t b = s_bal[warp][v];
        if ((b >> lane) & 1u) a.sids[at + __popc(b & lanemask_lt())] = x + w * (v + V * y);
        at += __popc(b);
    }
}

template <bool SHADE, bool GEN, bool FINAL>
cudaError_t launch(const BounceArgs& a, cudaStream_t s) {
    const cudaError_t e = launch_chained(true, k_bounce<SHADE, GEN, FINAL>, (a.w * a.h + BT - 1u) / BT, BT, 0, s, a);
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

cudaError_t launch_bounce(const BounceArgs& a, bool shade, bool gen, bool final_image, cudaStream_t s) {
    if (gen) return shade ? launch<true, true, false>(a, s) : launch<false, true, false>(a, s);
    if (final_image) return shade ? launch<true, false, true>(a, s) : launch<false, false, true>(a, s);
    return launch<false, false, false>(a, s);
}

}  // namespace rsh
