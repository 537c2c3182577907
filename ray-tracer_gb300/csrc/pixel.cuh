// The per-pixel steps of a frame -- hit resolve, shadow and reflection rays, shading -- as device functions: the
// single-step kernels (raygen.cu, shade.cu) and the fused bounce kernel (bounce.cu) run the same arithmetic.
#pragma once
#include "common.cuh"
#include "hash.cuh"
#include "kernels.h"

namespace rsh {

// ------------------------------------------------------------------ primary rays (tile order)
// Tile row r of the ray order is image tile row tile_row(r): from the middle outwards (m, m - 1, m + 1,
// m - 2, ... with m = rows / 2). Primary rays run longest in the view's centre band (on typical views the
// horizon, where rays travel far), so a persistent traversal starts them first instead of ending on them.
RSH_DEV uint32_t tile_row(uint32_t r, uint32_t rows) {
    const uint32_t m = rows >> 1;
    return (r & 1u) ? m - ((r + 1u) >> 1) : m + (r >> 1);
}

// Its inverse: the place of image tile row y in the ray order.
RSH_DEV uint32_t tile_row_place(uint32_t y, uint32_t rows) {
    const uint32_t m = rows >> 1;
    return y < m ? 2u * (m - y) - 1u : 2u * (y - m);
}
// The primary ray of pixel (x, y).
RSH_DEV uint32_t primary_of_pixel(uint32_t x, uint32_t y, uint32_t tiles_x, uint32_t tiles_y) {
    return ((tile_row_place(y >> 3, tiles_y) * tiles_x + (x >> 3)) << 6) + ((y & 7u) << 3) + (x & 7u);
}

// ------------------------------------------------------------------ shadow rays
// Soft-shadow sample k (0..15) around light position lp for the shadow direction d: the reference's 4x4
// grid without its centre row/column (RayTracer.cu:1550-1599): k = i + 4 j, a = i (+1 from i = 2),
// b = j (+1 from j = 2), position lp + axis0 (a - 2) / 8 + axis1 (b - 2) / 8, axis0 = cross(e, d) for the
// axis e the reference picks by min(|dx|, max(|dy|, |dz|)), axis1 = cross(d, axis0) (neither normalised).
RSH_DEV v3 soft_sample_pos(v3 lp, v3 d, uint32_t k) {
    const uint32_t i = k & 3u, j = k >> 2;
    const float ca = (float)((int)(i + (i >= 2u ? 1u : 0u)) - 2), cb = (float)((int)(j + (j >= 2u ? 1u : 0u)) - 2);
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    const float mn = fminf(ax, fmaxf(ay, az));
    const v3 e = (ax == mn) ? v3{1.f, 0.f, 0.f} : (ay == mn) ? v3{0.f, 1.f, 0.f} : v3{0.f, 0.f, 1.f};
    const v3 a0 = cross3(e, d);
    const v3 a1 = cross3(d, a0);
    return v3{(lp.x + (a0.x * ca) * 0.125f) + (a1.x * cb) * 0.125f, (lp.y + (a0.y * ca) * 0.125f) + (a1.y * cb) * 0.125f,
              (lp.z + (a0.z * ca) * 0.125f) + (a1.z * cb) * 0.125f};
}

// The shadow ray of surface point p (unit normal nn) for light position lp, sample sm of S; false: no ray.
RSH_DEV bool shadow_ray(v3 p, v3 nn, v3 lp, float eps, uint32_t S, uint32_t sm, float4& ro, float4& rd) {
    const v3 vl = p - lp;
    const float len = len3(vl);
    const v3 d = v3{vl.x / len, vl.y / len, vl.z / len};
    const float diffuse = dot3(d, -nn);
    const float tmax = len - 2.0f * eps;
    if (!(diffuse > 0.0f && tmax > eps)) return false;
    v3 src = lp, dir = d;
    float tm = tmax;
    if (S > 1) {  // a sample of the 4x4 grid: its own origin, direction and interval
        src = soft_sample_pos(lp, d, sm);
        const v3 vs = p - src;
        const float ls = len3(vs);
        dir = v3{vs.x / ls, vs.y / ls, vs.z / ls};
        tm = ls - 2.0f * eps;
        if (!(tm > eps)) return false;
    }
    const v3 o = src + dir * eps;
    ro = make_float4(o.x, o.y, o.z, eps);
    rd = make_float4(dir.x, dir.y, dir.z, tm);
    return true;
}

// ------------------------------------------------------------------ reflection rays
// Integer hash of (seed, slot, bounce) -> 32 random bits (PCG output permutation on an LCG step).
RSH_DEV uint32_t rng_next(uint32_t& state) {
    state = state * 747796405u + 2891336453u;
    uint32_t w = ((state >> ((state >> 28) + 4u)) ^ state) * 277803737u;
    return (w >> 22) ^ w;
}
// Uniform point on the unit sphere by Marsaglia's (1972) rejection method: sqrt only.
RSH_DEV v3 sphere_sample(uint32_t seed, uint32_t slot, uint32_t bounce) {
    uint32_t st = seed ^ (slot * 0x9E3779B9u) ^ (bounce * 0x85EBCA6Bu);
    rng_next(st);
    for (int it = 0; it < 32; ++it) {
        const float x1 = (float)(rng_next(st) >> 9) * (1.0f / 4194304.0f) - 1.0f;
        const float x2 = (float)(rng_next(st) >> 9) * (1.0f / 4194304.0f) - 1.0f;
        const float q = x1 * x1 + x2 * x2;
        if (q < 1.0f && q > 0.0f) {
            const float t = 2.0f * sqrtf(1.0f - q);
            return v3{x1 * t, x2 * t, 1.0f - 2.0f * q};
        }
    }
    return v3{0.0f, 0.0f, 1.0f};
}

// The reflection ray of surface point p (unit normal nn) for incident direction i; false: no ray (a degenerate
// direction).
RSH_DEV bool reflect_ray(v3 p, v3 nn, v3 i, float eps, float jitter, uint32_t seed, uint32_t slot, uint32_t bounce,
                         float4& ro, float4& rd) {
    const float k2 = 2.0f * dot3(nn, i);
    v3 r = i - nn * k2;  // reflect(i, n)
    if (jitter > 0.0f) {
        const v3 u = sphere_sample(seed, slot, bounce);
        r = r + u * jitter;
        const float rn = dot3(r, nn);
        if (rn < 0.0f) r = r - nn * (2.0f * rn);
    }
    r = norm3(r);
    if (!(r.x == r.x && r.y == r.y && r.z == r.z)) return false;
    const v3 o = p + r * eps;
    ro = make_float4(o.x, o.y, o.z, eps);
    rd = make_float4(r.x, r.y, r.z, __int_as_float(0x7f800000));
    return true;
}

// ------------------------------------------------------------------ hit resolve
// The surface of hit record h of ray (o, d): position (w = 1), interpolated normal (w = material id bits); a
// miss: zeros.
RSH_DEV void resolve_hit(const float4* __restrict__ pos, const float4* __restrict__ nrm,
                         const uint32_t* __restrict__ mat_ids, float4 o, float4 d, unsigned long long h, float4& sp,
                         float4& sn) {
    sp = sn = make_float4(0.f, 0.f, 0.f, 0.f);
    if (h == RSH_HIT_NONE) return;
    const uint32_t tri = (uint32_t)h;
    const float t = __uint_as_float((uint32_t)(h >> 32));
    const v3 p = v3{o.x + d.x * t, o.y + d.y * t, o.z + d.z * t};
    const v3 a = mk3(__ldg(pos + 3ull * tri)), b = mk3(__ldg(pos + 3ull * tri + 1)),
             c = mk3(__ldg(pos + 3ull * tri + 2));
    const float abc = len3(cross3(b - a, c - a));
    const float pbc = len3(cross3(b - p, c - p));
    const float pca = len3(cross3(a - p, c - p));
    const float b0 = pbc / abc, b1 = pca / abc, b2 = (1.0f - b0) - b1;
    const v3 n0 = mk3(__ldg(nrm + 3ull * tri)), n1 = mk3(__ldg(nrm + 3ull * tri + 1)),
             n2 = mk3(__ldg(nrm + 3ull * tri + 2));
    const v3 nn = v3{(n0.x * b0 + n1.x * b1) + n2.x * b2, (n0.y * b0 + n1.y * b1) + n2.y * b2,
                     (n0.z * b0 + n1.z * b1) + n2.z * b2};
    const uint32_t mid = mat_ids ? __ldg(mat_ids + tri) : 0u;
    sp = make_float4(p.x, p.y, p.z, 1.0f);
    sn = make_float4(nn.x, nn.y, nn.z, __uint_as_float(mid));
}

// ------------------------------------------------------------------ shading
// Soft-shadow weight of sample k (RayTracer.cu:1680-1690): inner four 0.55/16, corners 0.5375/16,
// edges 0.525/16.
RSH_DEV float soft_weight(uint32_t k) {
    if (k == 5 || k == 6 || k == 9 || k == 10) return 0.55f / 16.0f;
    if (k == 0 || k == 3 || k == 12 || k == 15) return 0.5375f / 16.0f;
    return 0.525f / 16.0f;
}

// One bounce's shading of pixel pix = (x, y) whose surface is (p4, n4) and incident direction inc, added to acc
// (rgb, weight in w); shadow == nullptr: unshadowed. Blinn-Phong per unoccluded light (RayTracer.cu:1616-1709).
RSH_DEV void shade_surface(const ShadeArgs& a, const rsh_light* s_light, const uint32_t* shadow,
                           uint32_t x, uint32_t y, float4 p4, float4 n4, v3 inc, float4& acc) {
    const v3 p = mk3(p4);
    const v3 n = norm3(mk3(n4));
    uint32_t mid = __float_as_uint(n4.w);
    if (mid >= a.material_count) mid = 0;
    const rsh_material m = a.materials[mid];
    float cr = 0.f, cg = 0.f, cb = 0.f;
    const uint32_t S = a.samples ? a.samples : 1u;
    // one sample a light: the flags of all lights (at most 8) before any of them is used, so that their loads overlap
    uint32_t occluded = 0;
    if (S == 1 && shadow) {
        const uint32_t* f = shadow + (x + (size_t)a.w * a.lights * y);
#pragma unroll 4
        for (uint32_t l = 0; l < a.lights; ++l) occluded |= (ld_chain(f + a.w * l) == RSH_OCCLUDED ? 1u : 0u) << l;
    }
    for (uint32_t l = 0; l < a.lights; ++l) {
        float factor = 1.0f;
        if (S == 1) {
            if ((occluded >> l) & 1u) continue;
        } else if (shadow) {
            // soft shadows (RayTracer.cu:1680-1696): weighted unoccluded samples, log2(1 + 2 sum)
            float sf = 0.0f;
            for (uint32_t k = 0; k < S; ++k)
                if (ld_chain(shadow + (x + a.w * ((l * S + k) + a.lights * S * y))) != RSH_OCCLUDED) sf += soft_weight(k);
            factor = log2f(1.0f + sf * 2.0f);
        }
        const rsh_light& L = s_light[l];
        v3 ld = v3{L.position[0], L.position[1], L.position[2]} - p;
        const float dist = len3(ld);
        ld = v3{ld.x / dist, ld.y / dist, ld.z / dist};
        const float att = 1.0f / (0.75f + dist * 0.0005f + dist * dist * 0.00005f);
        const float diff = fminf(fmaxf(dot3(ld, n), 0.0f), 1.0f);
        if (diff > 0.0f) {
            const v3 hv = norm3(ld - inc);
            const float sp = fminf(fmaxf(powf(fmaxf(dot3(hv, n), 0.0f), m.specular[3]), 0.0f), 1.0f);
            const float kd = diff * L.diffuse_intensity * att * factor, ks = sp * L.specular_intensity * att * factor;
            cr += (m.diffuse[0] * kd + m.specular[0] * ks) * L.color[0];
            cg += (m.diffuse[1] * kd + m.specular[1] * ks) * L.color[1];
            cb += (m.diffuse[2] * kd + m.specular[2] * ks) * L.color[2];
        }
    }
    acc.x += acc.w * cr;
    acc.y += acc.w * cg;
    acc.z += acc.w * cb;
    acc.w *= m.diffuse[3];  // reflectance carried to the next bounce
}
// The lights into shared memory (all threads; the caller synchronises): indexing the parameter bank with the
// light number would be a constant load with a register index per field, issued through the SM's narrow
// address-divergence pipe.
RSH_DEV void stage_lights(const ShadeArgs& a, rsh_light* s_light) {
    static_assert(sizeof(rsh_light) == 8 * sizeof(float), "rsh_light is 8 floats");
    if (threadIdx.x < 8u * a.lights)
        reinterpret_cast<float*>(s_light)[threadIdx.x] = reinterpret_cast<const float*>(a.light)[threadIdx.x];
}
RSH_DEV uint32_t pack_rgba(float4 c) {
    const uint32_t r = (uint32_t)fminf(fmaxf(c.x * 255.0f, 0.0f), 255.0f);
    const uint32_t g = (uint32_t)fminf(fmaxf(c.y * 255.0f, 0.0f), 255.0f);
    const uint32_t b = (uint32_t)fminf(fmaxf(c.z * 255.0f, 0.0f), 255.0f);
    return r | (g << 8) | (b << 16) | (255u << 24);
}

}  // namespace rsh
