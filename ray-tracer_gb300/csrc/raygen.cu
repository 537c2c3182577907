// Ray generation fused with the 32-bit ray hash.
//
// Reference: CreateShadowRays (RayTracer.cu:682-740), CreateReflectionRays (:742-791), the ray
// creation tail of ColorAndCreateReflectionRay (:1995-2016), the camera ray of RayTracer.cu:666-667 /
// CUDA-Naive-Ray-Tracer RayTracer.cu:606-607. The reference hash (CreateShadowRayIndex :147-168,
// CreateReflectionRayIndex :170-198) used atan2(x, x), which is constant, so the key is redefined:
//   key = tag << (3g + 2b) | morton3(origin cell, g bits per axis) << 2b | morton2(octahedral bin)
// using only +, -, *, /, abs, min/max and truncation, so a CPU restatement reproduces it bit for bit.
#include "common.cuh"
#include "hash.cuh"
#include "kernels.h"
#include "pixel.cuh"

namespace rsh {

// ------------------------------------------------------------------ primary rays (tile order)
__global__ void k_raygen_primary(CameraP cam, uint32_t w, uint32_t h, uint32_t tiles_x, uint32_t tiles_y, uint32_t n,
                                 rsh_ray* rays, uint32_t* pixel_of_ray, const Words2 zero) {
    asm volatile("griddepcontrol.launch_dependents;");  // the traversal waits for the rays itself
    if (blockIdx.x == 0)
        for (int q = 0; q < 2; ++q)
            for (uint32_t i = threadIdx.x; i < zero.n[q]; i += blockDim.x) zero.p[q][i] = 0u;
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t tile = k >> 6, within = k & 63u;
    const uint32_t x = (tile % tiles_x) * 8u + (within & 7u);
    const uint32_t y = tile_row(tile / tiles_x, tiles_y) * 8u + (within >> 3);
    float4 o = make_float4(cam.eye[0], cam.eye[1], cam.eye[2], 0.0f);
    float4 d;
    if (x < w && y < h) {
        const float a = (float)x / (float)w - 0.5f;
        const float b = (float)y / (float)h - 0.5f;
        v3 q = mk3((cam.dir[0] + cam.right[0] * a) + cam.up[0] * b,
                   (cam.dir[1] + cam.right[1] * a) + cam.up[1] * b,
                   (cam.dir[2] + cam.right[2] * a) + cam.up[2] * b);
        v3 dn = norm3(q);
        d = make_float4(dn.x, dn.y, dn.z, __int_as_float(0x7f800000));  // tmax = +inf
        if (pixel_of_ray) pixel_of_ray[k] = y * w + x;
    } else {
        d = make_float4(0.0f, 0.0f, 1.0f, -1.0f);  // tmax < tmin: no ray
        if (pixel_of_ray) pixel_of_ray[k] = 0xFFFFFFFFu;
    }
    store_ray(rays, k, o, d);
}

cudaError_t launch_raygen_primary(const CameraP& cam, uint32_t w, uint32_t h, rsh_ray* rays,
                                  uint32_t* pixel_of_ray, cudaStream_t s, const Words2& zero) {
    const uint32_t tx = (w + 7u) / 8u, ty = (h + 7u) / 8u;
    const uint32_t n = tx * ty * 64u;
    if (n == 0) return cudaSuccess;
    k_raygen_primary<<<(n + 255u) / 256u, 256, 0, s>>>(cam, w, h, tx, ty, n, rays, pixel_of_ray, zero);
    note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ shadow rays
// One thread per pixel: the pixel's surface point and normal are read and the normal normalised once,
// then its V = L x S slots are written (slot = x + W (v + V y), RayTracer.cu:700-702 with S samples per
// light), each with the same arithmetic as a thread per slot would use. The block's rays are counted once
// (RayOut). The light positions are copied to shared memory
// first: indexing the parameter bank with the light number is a constant load with a register index, which the
// SM issues through its narrow address-divergence pipe, and three of those per slot made that pipe the kernel's
// bound. 12 blocks per SM (at most 40 registers, no spills) keep enough warps in flight to cover the surface
// reads.
constexpr uint32_t RS_THREADS = 128;
// BATCH: for a batched call (out), else keys of its own or none. One hash in the loop instead of two, and no tests for
// the other form: 2.76 M slots 32.6 -> 28.2 us, bound by issue slots (exact divides and roots, the hash).
template <bool BATCH>
__global__ void __launch_bounds__(RS_THREADS, 12)
k_raygen_shadow(const float4* __restrict__ spos, const float4* __restrict__ snrm, uint32_t w, uint32_t h,
                LightsP lights, float eps, HashP hp, rsh_ray* rays, uint32_t* keys, RayOut out) {
    __shared__ float s_lp[8 * 3];
    __shared__ uint32_t s_cnt[RS_THREADS / 32];
    const uint32_t L = lights.count, S = lights.samples ? lights.samples : 1u, V = L * S;
    const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x, lane = lane_id(), warp = threadIdx.x >> 5;
    const bool in_range = pix < w * h;
    const bool a32 = (reinterpret_cast<uintptr_t>(rays) & 31u) == 0u;
    uint32_t nvalid = 0;  // the warp's rays
    if (threadIdx.x < 3u * L) s_lp[threadIdx.x] = (&lights.pos[0][0])[threadIdx.x];
    __syncthreads();
    const uint32_t y = pix / w, x = pix - y * w;
    const float4 p4 = in_range ? __ldg(spos + pix) : make_float4(0.f, 0.f, 0.f, 0.f);
    const bool surface = p4.w != 0.0f;
    const v3 p = mk3(p4);
    const v3 nn = surface ? norm3(mk3(__ldg(snrm + pix))) : v3{0.f, 0.f, 0.f};
    for (uint32_t v = 0; v < V; ++v) {
        const uint32_t slot = x + w * (v + V * y);
        const uint32_t l = S == 1u ? v : v / S, sm = S == 1u ? 0u : v % S;
        bool valid = false;
        float4 ro = make_float4(0.f, 0.f, 0.f, 0.f), rd = make_float4(0.f, 0.f, 0.f, -1.f);
        uint32_t key = RSH_KEY_NONE;
        if (surface) {
            const v3 lp = mk3(s_lp[3u * l], s_lp[3u * l + 1u], s_lp[3u * l + 2u]);
            valid = shadow_ray(p, nn, lp, eps, S, sm, ro, rd);
            if (!BATCH && valid && keys) key = ray_hash(ro.x, ro.y, ro.z, rd.x, rd.y, rd.z, hp, v);
        }
        if (in_range) {
            // an empty slot holds an explicit no-ray (tmax < tmin) for consumers without keys
            store_ray32(rays, slot, ro, rd, a32);
            if (!BATCH && keys) keys[slot] = key;
            if (BATCH) {
                out.keys[slot] = valid ? out.tag | (ray_hash(ro.x, ro.y, ro.z, rd.x, rd.y, rd.z, out.hp, 0u) >> out.drop)
                                       : RSH_KEY_NONE;
                if (out.flags) out.flags[slot] = 0u;
                else out.hits[slot] = RSH_HIT_NONE;
            }
        }
        if (BATCH) {
            const uint32_t b = __ballot_sync(0xffffffffu, valid);
            nvalid += __popc(b);
        }
    }
    if (BATCH) {
        if (lane == 0) s_cnt[warp] = nvalid;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t all = 0;
#pragma unroll
            for (uint32_t q = 0; q < RS_THREADS / 32; ++q) all += s_cnt[q];
            if (all) atomicAdd(out.count, all);
        }
    }
}

cudaError_t launch_raygen_shadow(const float4* spos, const float4* snrm, uint32_t w, uint32_t h,
                                 const LightsP& lights, float eps, const HashP& hp, rsh_ray* rays,
                                 uint32_t* keys, cudaStream_t s, const RayOut& out) {
    const uint32_t n = w * h;
    if (n == 0 || lights.count == 0) return cudaSuccess;
    const auto kernel = out.count ? k_raygen_shadow<true> : k_raygen_shadow<false>;
    kernel<<<(n + RS_THREADS - 1u) / RS_THREADS, RS_THREADS, 0, s>>>(spos, snrm, w, h, lights, eps, hp, rays, keys, out);
    note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ reflection rays
__global__ void k_raygen_reflect(const float4* __restrict__ spos, const float4* __restrict__ snrm,
                                 const rsh_ray* __restrict__ prev, v3 eye, uint32_t n, float eps,
                                 float jitter, uint32_t seed, uint32_t bounce, HashP hp,
                                 rsh_ray* rays, uint32_t* keys, RayOut out) {
    __shared__ uint32_t s_cnt[8];
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in_range = slot < n;
    const bool a32 = (reinterpret_cast<uintptr_t>(rays) & 31u) == 0u;
    bool valid = false;
    float4 ro = make_float4(0.f, 0.f, 0.f, 0.f), rd = make_float4(0.f, 0.f, 0.f, -1.f);
    if (in_range) {
        const float4 p4 = __ldg(spos + slot);
        uint32_t key = RSH_KEY_NONE;
        if (p4.w != 0.0f) {
            const v3 p = mk3(p4);
            const v3 nn = norm3(mk3(__ldg(snrm + slot)));
            v3 i;
            if (prev) {
                float4 po, pd;
                load_ray(prev, slot, po, pd);
                i = mk3(pd);
            } else {
                i = norm3(p - eye);
            }
            valid = reflect_ray(p, nn, i, eps, jitter, seed, slot, bounce, ro, rd);
            if (valid && keys) key = ray_hash(ro.x, ro.y, ro.z, rd.x, rd.y, rd.z, hp, 0u);
        }
        // no ray: stored as such, also for the next bounce, which reads this array as its incident rays
        store_ray32(rays, slot, ro, rd, a32);
        if (keys) keys[slot] = key;
    }
    if (out.count) {
        if (in_range) {
            if (out.keys)
                out.keys[slot] = valid ? out.tag | (ray_hash(ro.x, ro.y, ro.z, rd.x, rd.y, rd.z, out.hp, 0u) >> out.drop)
                                       : RSH_KEY_NONE;
            if (out.flags) out.flags[slot] = 0u;
            else out.hits[slot] = RSH_HIT_NONE;
        }
        const uint32_t warp = threadIdx.x >> 5, b = __ballot_sync(0xffffffffu, valid);
        if (lane_id() == 0) s_cnt[warp] = __popc(b);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t all = 0;
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) all += s_cnt[q];  // 256 threads
            if (all) atomicAdd(out.count, all);
        }
    }
}

cudaError_t launch_raygen_reflect(const float4* spos, const float4* snrm, const rsh_ray* prev,
                                  const float eye[3], uint32_t w, uint32_t h, float eps,
                                  float jitter, uint32_t seed, uint32_t bounce, const HashP& hp,
                                  rsh_ray* rays, uint32_t* keys, cudaStream_t s, const RayOut& out) {
    const uint32_t n = w * h;
    if (n == 0) return cudaSuccess;
    k_raygen_reflect<<<(n + 255u) / 256u, 256, 0, s>>>(spos, snrm, prev, v3{eye[0], eye[1], eye[2]}, n,
                                                     eps, jitter, seed, bounce, hp, rays, keys, out);
    note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ refraction rays
// CreateRefractionRays (RayTracer.cu:793-842): direction refract(i, n, eta) (GLSL's formula: k = 1 -
// eta^2 (1 - (n.i)^2), t = eta i - (eta n.i + sqrt k) n; no ray when k < 0, total internal reflection),
// i = normalize(p - eye) or the incident ray, the surface normal as stored; renormalised, origin offset by
// eps, interval (eps, inf). The reference creates these rays but never casts them.
__global__ void k_raygen_refract(const float4* __restrict__ spos, const float4* __restrict__ snrm,
                                 const rsh_ray* __restrict__ prev, v3 eye, uint32_t n, float eps, float eta,
                                 HashP hp, rsh_ray* rays, uint32_t* keys) {
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= n) return;
    const float4 p4 = __ldg(spos + slot);
    uint32_t key = RSH_KEY_NONE;
    if (p4.w != 0.0f) {
        const v3 p = mk3(p4);
        const v3 nn = norm3(mk3(__ldg(snrm + slot)));
        v3 i;
        if (prev) {
            float4 po, pd;
            load_ray(prev, slot, po, pd);
            i = mk3(pd);
        } else {
            i = norm3(p - eye);
        }
        const float d = dot3(nn, i);
        const float k = 1.0f - eta * eta * (1.0f - d * d);
        if (k >= 0.0f) {
            const v3 t = norm3(i * eta - nn * (eta * d + sqrtf(k)));
            if (t.x == t.x && t.y == t.y && t.z == t.z) {
                const v3 o = p + t * eps;
                store_ray(rays, slot, make_float4(o.x, o.y, o.z, eps),
                          make_float4(t.x, t.y, t.z, __int_as_float(0x7f800000)));
                key = ray_hash(o.x, o.y, o.z, t.x, t.y, t.z, hp, 0u);
            }
        }
    }
    if (key == RSH_KEY_NONE)
        store_ray(rays, slot, make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, -1.f));
    keys[slot] = key;
}

cudaError_t launch_raygen_refract(const float4* spos, const float4* snrm, const rsh_ray* prev, const float eye[3],
                                  uint32_t w, uint32_t h, float eps, float eta, const HashP& hp, rsh_ray* rays,
                                  uint32_t* keys, cudaStream_t s) {
    const uint32_t n = w * h;
    if (n == 0) return cudaSuccess;
    k_raygen_refract<<<(n + 255u) / 256u, 256, 0, s>>>(spos, snrm, prev, v3{eye[0], eye[1], eye[2]}, n, eps, eta,
                                                     hp, rays, keys);
    note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ hash of given rays
__global__ void k_hash(const rsh_ray* __restrict__ rays, uint32_t n, HashP hp, uint32_t tag,
                       uint32_t* keys) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 o, d;
    load_ray(rays, i, o, d);
    keys[i] = (d.w > o.w) ? ray_hash(o.x, o.y, o.z, d.x, d.y, d.z, hp, tag) : RSH_KEY_NONE;
}

cudaError_t launch_hash(const rsh_ray* rays, uint32_t n, const HashP& hp, uint32_t tag,
                        uint32_t* keys, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_hash<<<(n + 255u) / 256u, 256, 0, s>>>(rays, n, hp, tag, keys);
    note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ fills
__global__ void k_fill_u64(unsigned long long* p, unsigned long long v, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        p[i] = v;
}
cudaError_t launch_fill_u64(unsigned long long* p, unsigned long long v, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    size_t blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    k_fill_u64<<<(unsigned)blocks, 256, 0, s>>>(p, v, n);
    note_launch();
    return cudaGetLastError();
}

}  // namespace rsh
