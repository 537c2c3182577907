// Bottom-up build of the ray-space hierarchy (cone + sphere nodes).
//
// Reference: HierarchyCreationWrapper (RayTracer.cu:2469-2535) with CreateHierarchyLevel0 (:1061-1108,
// 8 consecutive sorted rays -> sphere of origins + cone of directions via CreateHierarchySphere
// :427-446 / CreateHierarchyCone0 :379-406) and CreateHierarchyLevelN (:1110-1150, 8 children via
// CreateHierarchyConeN :408-425). Those merges use acos/cos/sin and are not conservative (a cone can
// miss a ray), so the nodes are redefined to be conservative by construction:
//   leaf (P rays, four to a lane):
//     centre = midpoint of the origins' bounding box, radius = max |o - centre|,
//     axis = normalize(sum of directions), cos_spread = min dot(axis, d) - 4e-6 (<= 0: full cone),
//     reach = max(|o - centre| + tmax)  (how far any ray of the node can get from the centre);
//   level L (8 children): box of child spheres -> centre, radius = max(|c_i - c| + r_i),
//     axis = normalize(sum count_i * axis_i), cos_spread = min cos(angle(axis, axis_i) + spread_i),
//     reach = max(|c_i - c| + reach_i).
// A leaf's sums are pairwise trees in index order (1, 2, 4, ...), a level's run over the children in order:
// reproducible on the host.
#include "common.cuh"
#include "kernels.h"

namespace rsh {

namespace {
constexpr float kRadSlack = 1.0f + 1.0f / 1048576.0f;  // 1 + 2^-20
constexpr float kCosMargin = 4e-6f;
}

uint32_t hierarchy_capacity(uint32_t max_rays, uint32_t packet, uint32_t offsets[4]) {
    const uint32_t n0 = (max_rays + packet - 1) / packet;
    const uint32_t n1 = (n0 + 7) / 8;
    const uint32_t n2 = (n1 + 7) / 8;
    offsets[0] = 0;
    offsets[1] = n0;
    offsets[2] = n0 + n1;
    offsets[3] = n0 + n1 + n2;
    return offsets[3];
}

namespace {
constexpr uint32_t BN_LEAVES = 64, BN_THREADS = 128;  // a CTA: 64 leaves, 16 a warp; 8 nodes over them; one on top
constexpr int BN_RPL = 4;                             // rays per lane

// nodes[0..m) of shared memory -> global memory by a warp, word by word (a node is 48 bytes at any 4-byte address)
RSH_DEV void store_nodes(const rsh_node* __restrict__ src, rsh_node* __restrict__ dst, uint32_t m) {
    const uint32_t* a = reinterpret_cast<const uint32_t*>(src);
    uint32_t* b = reinterpret_cast<uint32_t*>(dst);
    for (uint32_t i = lane_id(); i < m * (uint32_t)(sizeof(rsh_node) / 4); i += 32u) b[i] = a[i];
}

// The node over the m (1..8) children ch[0..m) of shared memory, by a group of 8 lanes, a child each (all 32 lanes of
// the warp are here). The sums run over the children in order.
RSH_DEV rsh_node merge8(const rsh_node* ch, uint32_t m) {
    const float inf = __int_as_float(0x7f800000);
    const uint32_t i = lane_id() & 7u, g = lane_id() & ~7u;
    const rsh_node q = ch[i < m ? i : 0u];
    const bool on = i < m && q.count != 0u;
    const uint32_t on8 = (__ballot_sync(0xffffffffu, on) >> g) & 255u;
    bool full = ((__ballot_sync(0xffffffffu, on && !(q.cos_spread > 0.f)) >> g) & 255u) != 0u;
    // (a NaN bound counts as none)
    float mnx = on ? fminf(inf, q.c[0] - q.radius) : inf, mxx = on ? fmaxf(-inf, q.c[0] + q.radius) : -inf;
    float mny = on ? fminf(inf, q.c[1] - q.radius) : inf, mxy = on ? fmaxf(-inf, q.c[1] + q.radius) : -inf;
    float mnz = on ? fminf(inf, q.c[2] - q.radius) : inf, mxz = on ? fmaxf(-inf, q.c[2] + q.radius) : -inf;
    uint32_t count = on ? q.count : 0u;
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
        mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, off));
        mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, off));
        mnz = fminf(mnz, __shfl_xor_sync(0xffffffffu, mnz, off));
        mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, off));
        mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, off));
        mxz = fmaxf(mxz, __shfl_xor_sync(0xffffffffu, mxz, off));
        count += __shfl_xor_sync(0xffffffffu, count, off);
    }
    const float w = (float)q.count;
    const float ax = q.axis[0] * w, ay = q.axis[1] * w, az = q.axis[2] * w;
    float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
        const float x = __shfl_sync(0xffffffffu, ax, g + j), y = __shfl_sync(0xffffffffu, ay, g + j),
                    z = __shfl_sync(0xffffffffu, az, g + j);
        if ((on8 >> j) & 1u) {
            sx = sx + x;
            sy = sy + y;
            sz = sz + z;
        }
    }
    rsh_node nd;
    nd.first = ch[0].first;
    nd.count = count;
    const v3 c = v3{(mnx + mxx) * 0.5f, (mny + mxy) * 0.5f, (mnz + mxz) * 0.5f};
    const float sl = sqrtf((sx * sx + sy * sy) + sz * sz);
    if (!(sl > 1e-20f)) full = true;
    const v3 a = full ? v3{0.f, 0.f, 1.f} : v3{sx / sl, sy / sl, sz / sl};
    float rad = 0.f, reach = 0.f, cs = 1.f;
    if (on) {
        const v3 dc = v3{q.c[0] - c.x, q.c[1] - c.y, q.c[2] - c.z};
        const float dl = len3(dc);
        rad = fmaxf(rad, dl + q.radius);
        reach = fmaxf(reach, dl + q.reach);
        if (!full) {
            float ca = dot3(a, v3{q.axis[0], q.axis[1], q.axis[2]});
            ca = fminf(fmaxf(ca, -1.f), 1.f);
            const float sa = sqrtf((1.f - ca) * (1.f + ca));
            cs = fminf(cs, ca * q.cos_spread - sa * q.sin_spread);
        }
    }
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
        rad = fmaxf(rad, __shfl_xor_sync(0xffffffffu, rad, off));
        reach = fmaxf(reach, __shfl_xor_sync(0xffffffffu, reach, off));
        cs = fminf(cs, __shfl_xor_sync(0xffffffffu, cs, off));
    }
    cs = cs - kCosMargin;
    if (!(cs > 0.f)) full = true;
    nd.c[0] = c.x;
    nd.c[1] = c.y;
    nd.c[2] = c.z;
    nd.radius = rad * kRadSlack;
    nd.axis[0] = a.x;
    nd.axis[1] = a.y;
    nd.axis[2] = a.z;
    nd.cos_spread = full ? -1.f : cs;
    nd.sin_spread = full ? 0.f : sqrtf((1.f - cs) * (1.f + cs));
    nd.reach = reach * kRadSlack;
    if (count == 0) {
        nd.c[0] = nd.c[1] = nd.c[2] = 0.f;
        nd.radius = 0.f;
        nd.reach = 0.f;
    }
    return nd;
}
}  // namespace

// All three levels in one launch: the children of a node are nodes of the same CTA, still in shared memory.
// Bound by issue slots before it is by memory: a lane takes four rays, so that most of the pairwise tree needs no
// shuffle and a packet's roots and quotients are computed by two lanes, not eight. 2.76 M rays in packets of 8 (100 MB
// gathered and read): 32 us; a lane per ray 50, with each level in a launch of its own, a thread a node, 72.
template <int P>
__global__ void __launch_bounds__(BN_THREADS)
k_build_nodes(const rsh_ray* __restrict__ rays, const uint32_t* __restrict__ sorted_ids, uint32_t max_rays,
              const uint32_t* __restrict__ d_count, rsh_node* __restrict__ nodes, uint32_t off1, uint32_t off2) {
    constexpr uint32_t LP = P / BN_RPL, WL = BN_LEAVES / (BN_THREADS / 32), ROW = 32 * BN_RPL;
    static_assert(WL == 16 && WL * P % ROW == 0, "two groups of eight leaves a warp, in whole rows");
    __shared__ __align__(16) rsh_node s_leaf[BN_LEAVES], s_mid[8], s_top;
    const float inf = __int_as_float(0x7f800000);
    const uint32_t n = dev_count(d_count, max_rays);
    const uint32_t nl = (n + P - 1) / P, l0 = blockIdx.x * BN_LEAVES;
    if (l0 >= nl) return;  // whole CTA beyond the last packet
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t w0 = l0 + WL * warp, here = w0 < nl ? min(nl - w0, WL) : 0u;  // the warp's leaves
    const bool a16 = (reinterpret_cast<uintptr_t>(sorted_ids) & 15u) == 0u;
    rsh_node* leaf = s_leaf + WL * warp;
    for (uint32_t row = 0; row < here * P; row += ROW) {
        const uint32_t k = w0 * P + row + lane * BN_RPL;  // a multiple of BN_RPL
        uint32_t id[BN_RPL];
        if (sorted_ids && a16 && k + BN_RPL <= n) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(sorted_ids + k));
            id[0] = v.x;
            id[1] = v.y;
            id[2] = v.z;
            id[3] = v.w;
        } else {
#pragma unroll
            for (int u = 0; u < BN_RPL; ++u)
                id[u] = k + u < n ? (sorted_ids ? __ldg(sorted_ids + k + u) : k + u) : 0xFFFFFFFFu;
        }
        float4 o[BN_RPL], d[BN_RPL];
#pragma unroll
        for (int u = 0; u < BN_RPL; ++u) {
            o[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            d[u] = make_float4(0.f, 0.f, 0.f, -1.f);
            if (id[u] != 0xFFFFFFFFu) load_ray(rays, id[u], o[u], d[u]);  // (padding slots hold no ray)
        }
        bool act[BN_RPL];
        float mn[3][BN_RPL], mx[3][BN_RPL], sm[3][BN_RPL];
        uint32_t cnt = 0;
#pragma unroll
        for (int u = 0; u < BN_RPL; ++u) {
            act[u] = d[u].w > o[u].w;
            cnt += act[u] ? 1u : 0u;
            mn[0][u] = act[u] ? o[u].x : inf;
            mn[1][u] = act[u] ? o[u].y : inf;
            mn[2][u] = act[u] ? o[u].z : inf;
            mx[0][u] = act[u] ? o[u].x : -inf;
            mx[1][u] = act[u] ? o[u].y : -inf;
            mx[2][u] = act[u] ? o[u].z : -inf;
            sm[0][u] = act[u] ? d[u].x : 0.f;
            sm[1][u] = act[u] ? d[u].y : 0.f;
            sm[2][u] = act[u] ? d[u].z : 0.f;
        }
        // the pairwise tree: within the lane first, then across the packet's lanes
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            mn[x][0] = fminf(fminf(mn[x][0], mn[x][1]), fminf(mn[x][2], mn[x][3]));
            mx[x][0] = fmaxf(fmaxf(mx[x][0], mx[x][1]), fmaxf(mx[x][2], mx[x][3]));
            sm[x][0] = (sm[x][0] + sm[x][1]) + (sm[x][2] + sm[x][3]);
        }
#pragma unroll
        for (uint32_t off = 1; off < LP; off <<= 1) {
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                mn[x][0] = fminf(mn[x][0], __shfl_xor_sync(0xffffffffu, mn[x][0], off));
                mx[x][0] = fmaxf(mx[x][0], __shfl_xor_sync(0xffffffffu, mx[x][0], off));
                sm[x][0] = sm[x][0] + __shfl_xor_sync(0xffffffffu, sm[x][0], off);
            }
            cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
        }
        const float sx = sm[0][0], sy = sm[1][0], sz = sm[2][0];
        const v3 c = v3{(mn[0][0] + mx[0][0]) * 0.5f, (mn[1][0] + mx[1][0]) * 0.5f, (mn[2][0] + mx[2][0]) * 0.5f};
        const float sl = sqrtf((sx * sx + sy * sy) + sz * sz);
        bool full = !(sl > 1e-20f);
        const v3 a = full ? v3{0.f, 0.f, 1.f} : v3{sx / sl, sy / sl, sz / sl};
        // second phase: radius, cone spread, reach
        float mr2, dt, rc;
#pragma unroll
        for (int u = 0; u < BN_RPL; ++u) {
            const v3 oc = v3{o[u].x - c.x, o[u].y - c.y, o[u].z - c.z};
            const float r2 = act[u] ? dot3(oc, oc) : 0.f;
            const float t = act[u] ? dot3(a, mk3(d[u])) : inf, f = act[u] ? sqrtf(r2) + d[u].w : 0.f;
            mr2 = u ? fmaxf(mr2, r2) : r2;  // (NaN only where every ray gives NaN: then the cone is full)
            dt = u ? fminf(dt, t) : t;
            rc = u ? fmaxf(rc, f) : f;
        }
#pragma unroll
        for (uint32_t off = 1; off < LP; off <<= 1) {
            mr2 = fmaxf(mr2, __shfl_xor_sync(0xffffffffu, mr2, off));
            dt = fminf(dt, __shfl_xor_sync(0xffffffffu, dt, off));
            rc = fmaxf(rc, __shfl_xor_sync(0xffffffffu, rc, off));
        }
        const uint32_t li = (row + lane * BN_RPL) / P;
        if ((lane & (LP - 1u)) != 0u || li >= here) continue;
        float cs = dt - kCosMargin;
        if (!(cs > 0.f)) full = true;
        rsh_node nd;
        nd.c[0] = c.x;
        nd.c[1] = c.y;
        nd.c[2] = c.z;
        nd.radius = sqrtf(mr2) * kRadSlack;
        nd.axis[0] = a.x;
        nd.axis[1] = a.y;
        nd.axis[2] = a.z;
        nd.cos_spread = full ? -1.f : cs;
        nd.sin_spread = full ? 0.f : sqrtf((1.f - cs) * (1.f + cs));
        nd.reach = rc * kRadSlack;
        nd.first = k;
        nd.count = cnt;
        leaf[li] = nd;
    }
    __syncwarp();
    if (here) {
        store_nodes(leaf, nodes + w0, here);
        const uint32_t mids = (here + 7u) / 8u, g = (lane >> 3) < mids ? lane >> 3 : 0u;  // (spare groups repeat the first)
        const rsh_node nd = merge8(leaf + 8u * g, min(here - 8u * g, 8u));
        if ((lane & 7u) == 0u && (lane >> 3) < mids) s_mid[2u * warp + g] = nd;
        __syncwarp();
        store_nodes(s_mid + 2u * warp, nodes + off1 + w0 / 8u, mids);
    }
    __syncthreads();
    if (warp == 0u) {
        const rsh_node nd = merge8(s_mid, (min(nl - l0, BN_LEAVES) + 7u) / 8u);
        if (lane == 0u) s_top = nd;
        __syncwarp();
        store_nodes(&s_top, nodes + off2 + blockIdx.x, 1u);
    }
}

cudaError_t launch_build_rsh(const rsh_ray* rays, const uint32_t* sorted_ids, uint32_t max_rays,
                             const uint32_t* d_count, uint32_t packet, rsh_node* nodes,
                             cudaStream_t s) {
    if (max_rays == 0) return cudaSuccess;
    if (packet != 8 && packet != 16 && packet != 32) return cudaErrorInvalidValue;
    uint32_t off[4];
    hierarchy_capacity(max_rays, packet, off);
    const auto kernel = packet == 8 ? k_build_nodes<8> : packet == 16 ? k_build_nodes<16> : k_build_nodes<32>;
    kernel<<<(off[1] + BN_LEAVES - 1) / BN_LEAVES, BN_THREADS, 0, s>>>(rays, sorted_ids, max_rays, d_count, nodes, off[1],
                                                                       off[2]);
    note_launch();
    return cudaGetLastError();
}

}  // namespace rsh
