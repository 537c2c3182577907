// Hit resolve (hit point + interpolated normal -> surface buffer) and Blinn-Phong shading.
//
// Reference: the resolve half of ColorReflectionRay / ColorAndCreateReflectionRay
// (RayTracer.cu:1806-1843: re-intersect the winning triangle, hit point, area-ratio barycentric
// normal) and the shading of ColorPrimaryShadowRay (:1616-1709) / ColorReflectionRay (:1845-1880):
// Blinn-Phong per unoccluded light with attenuation 1 / (0.75 + 0.0005 d + 0.00005 d^2) (:1667).
// The surface buffer replaces the GL G-buffer: position.w = 1 marks a surface, normal.w carries the
// material id bits.
#include "common.cuh"
#include "kernels.h"
#include "pixel.cuh"

namespace rsh {

__global__ void k_resolve(const float4* __restrict__ pos, const float4* __restrict__ nrm,
                          const uint32_t* __restrict__ mat_ids, const rsh_ray* __restrict__ rays,
                          const unsigned long long* __restrict__ hits,
                          const uint32_t* __restrict__ pixel_of_ray, uint32_t n, float4* spos,
                          float4* snrm) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t pix = pixel_of_ray ? __ldg(pixel_of_ray + k) : k;
    if (pix == 0xFFFFFFFFu) return;
    const unsigned long long h = __ldg(hits + k);
    float4 o, d, sp, sn;
    if (h != RSH_HIT_NONE) load_ray(rays, k, o, d);
    resolve_hit(pos, nrm, mat_ids, o, d, h, sp, sn);
    spos[pix] = sp;
    snrm[pix] = sn;
}

cudaError_t launch_resolve(const float4* tris_orig_pos, const float4* tris_orig_nrm,
                           const uint32_t* mat_ids, const rsh_ray* rays, const unsigned long long* hits,
                           const uint32_t* pixel_of_ray, uint32_t n, float4* spos, float4* snrm,
                           cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_resolve<<<(n + 255) / 256, 256, 0, s>>>(tris_orig_pos, tris_orig_nrm, mat_ids, rays, hits,
                                              pixel_of_ray, n, spos, snrm);
    note_launch();
    return cudaGetLastError();
}

__global__ void k_shade(ShadeArgs a) {
    __shared__ rsh_light s_light[8];
    stage_lights(a, s_light);
    __syncthreads();
    const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= a.w * a.h) return;
    float4 acc = a.bounce == 0 ? make_float4(0.f, 0.f, 0.f, 1.f) : a.accum[pix];
    const float4 p4 = a.spos[pix];
    if (p4.w != 0.0f && acc.w > 0.0f) {
        v3 inc;
        if (a.incident) {
            float4 o, d;
            load_ray(a.incident, pix, o, d);
            inc = mk3(d);
        } else {
            inc = norm3(mk3(p4) - v3{a.eye[0], a.eye[1], a.eye[2]});
        }
        shade_surface(a, s_light, a.shadow, pix % a.w, pix / a.w, p4, a.snrm[pix], inc, acc);
    } else {
        acc.w = 0.0f;
    }
    a.accum[pix] = acc;
}

cudaError_t launch_shade(const ShadeArgs& a, cudaStream_t s) {
    const uint32_t n = a.w * a.h;
    if (n == 0) return cudaSuccess;
    k_shade<<<(n + 255) / 256, 256, 0, s>>>(a);
    note_launch();
    return cudaGetLastError();
}

__global__ void k_pack(const float4* __restrict__ acc, uint32_t n, uint32_t* rgba) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    rgba[i] = pack_rgba(acc[i]);
}

cudaError_t launch_pack_rgba(const float4* accum, uint32_t n, uint32_t* rgba, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_pack<<<(n + 255) / 256, 256, 0, s>>>(accum, n, rgba);
    note_launch();
    return cudaGetLastError();
}

}  // namespace rsh
