// Object bounding-sphere hierarchy over the scene's triangles.
//
// Reference: one minimal enclosing sphere per mesh from the GPL Miniball (BoundingSphere.cpp:9-63),
// packed as {centre, radius, firstTri, lastTri} (main.cpp:2445-2470) and culled against the top ray
// nodes (CalculateBoundingSpheresIntersections, RayTracer.cu:1152-1280); triangles then get a bounding
// sphere each (CreateTriangleBoundingSphere, :301-376) inside the descent. Here the object spheres
// become a full sphere tree built on the GPU, level by level, every level a list of nodes whose children
// are consecutive nodes of the level below:
//   1. Morton code (10 bits per axis) of every triangle centroid over the cube around the scene box;
//   2. stable onesweep sort of (code, triangle id) -> cluster order; gather the triangles (original id
//      kept in the first vertex's w);
//   3. boundary strength before sorted triangle k: the highest differing bit of the 64-bit keys
//      (code << 32 | k) of triangles k-1 and k (the splits of a binary radix tree over the keys);
//   4. level 0 groups triangles into clusters of at most `cluster`, every level above groups the level
//      below into nodes of at most 8: the items are cut exactly where the recursive split at the
//      strongest boundary would stop, i.e. boundary j is a cut iff the range it splits (bounded by the
//      nearest stronger boundaries on either side) holds more than G items -- decided from a window of
//      G items on each side; the cut positions are compacted in the same launch (look-back over tiles). A
//      level whose groups would reduce too little (< 2x for clusters, < 4x above) is cut into fixed groups
//      of G;
//   5. every node's sphere from all vertices of its triangle range: centre = midpoint of the vertex
//      box (of the children's boxes, which is the same box: min and max are exact in any order), radius =
//      max vertex distance (x (1 + 2^-20));
//   6. up to the first level with at most 8 nodes (the children of the virtual root).
// Level sizes stay on the device until the end: each level's launches are sized by the most items it can have
// (a level is at most half, above the clusters a quarter, of the one below), and once that is at most
// TAIL_ITEMS one block builds all remaining levels. The radii of every level above the clusters come from one
// pass over the vertices. A warp per node over all of its vertices, level by level with the sizes read back
// between, left the top levels to a handful of warps that each read the whole scene: 3.06 of the 6.6 ms of
// kernels of a frame of 1001 moving objects (320,032 triangles), against 0.12 ms for this form.
// Every sphere encloses every vertex below it, so the hierarchy never culls a real hit. Child ranges are
// stored per level as size + 1 starts: node j of level l covers [kids[l][j], kids[l][j + 1]) of level l-1
// (of the triangles, for level 0).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace rsh {

namespace {
constexpr float kRadSlack = 1.0f + 1.0f / 1048576.0f;
}

__global__ void k_morton(const float4* pos, uint32_t n, v3 lo, v3 sc, uint32_t* codes) {
    chain();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = ld_chain(pos + 3ull * i), b = ld_chain(pos + 3ull * i + 1), c = ld_chain(pos + 3ull * i + 2);
    const float cx = ((a.x + b.x) + c.x) / 3.0f;
    const float cy = ((a.y + b.y) + c.y) / 3.0f;
    const float cz = ((a.z + b.z) + c.z) / 3.0f;
    float fx = fminf(fmaxf((cx - lo.x) * sc.x, 0.f), 1023.f);
    float fy = fminf(fmaxf((cy - lo.y) * sc.y, 0.f), 1023.f);
    float fz = fminf(fmaxf((cz - lo.z) * sc.z, 0.f), 1023.f);
    codes[i] = (spread3((uint32_t)fx) << 2) | (spread3((uint32_t)fy) << 1) | spread3((uint32_t)fz);
}

__global__ void k_gather_tris(const float4* pos, const uint32_t* perm,
                              uint32_t n, float4* tris, uint32_t* order) {
    chain();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t t = ld_chain(perm + k);
    float4 a = ld_chain(pos + 3ull * t);
    a.w = __uint_as_float(t);
    tris[3ull * k] = a;
    tris[3ull * k + 1] = ld_chain(pos + 3ull * t + 1);
    tris[3ull * k + 2] = ld_chain(pos + 3ull * t + 2);
    order[k] = t;
}

// boundary strength before sorted triangle k (k = 0 and k = T: 64, stronger than any)
__global__ void k_delta_tri(const uint32_t* scode, uint32_t T, uint32_t* dtri) {
    chain();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > T) return;
    uint32_t d = 64u;
    if (k > 0 && k < T) {
        const uint32_t a = ld_chain(scode + k - 1), b = ld_chain(scode + k);
        d = (a != b) ? 32u + (31u - (uint32_t)__clz(a ^ b)) : 31u - (uint32_t)__clz((k - 1) ^ k);
    }
    dtri[k] = d;
}

namespace {

constexpr uint32_t LV_TILE = 256;      // items per tile of k_level_cuts
constexpr uint32_t TAIL_ITEMS = 4096;  // levels over at most this many items: one block
constexpr uint32_t TAIL_THREADS = 1024;
constexpr uint32_t MAX_G = 64;         // the largest group (cluster_size)

// one level's record (device): its node count, its first node's index over all levels, fixed groups of G
struct Level {
    uint32_t size, off, fixed;
};
// a node's vertex box without padding
struct RawBox {
    float lo[3], hi[3];
};

// A level's boundary strengths [j0, j0 + count) into shared memory (out of range: 64, stronger than any); start ==
// nullptr: the items are the triangles themselves. One round of loads for a tile, instead of two dependent
// loads for each step of a boundary's window.
RSH_DEV void load_deltas(uint32_t* s, const uint32_t* dtri, const uint32_t* start, uint32_t n, int64_t j0,
                         uint32_t count) {
    for (uint32_t q = threadIdx.x; q < count; q += blockDim.x) {
        const int64_t j = j0 + q;
        s[q] = (j <= 0 || j >= (int64_t)n) ? 64u : dtri[start ? start[j] : (uint32_t)j];
    }
}
// Is boundary j (strength s[0], its neighbours' around it; n items) a cut? The window is G boundaries on each side.
RSH_DEV bool is_cut(const uint32_t* s, uint32_t n, uint32_t G, uint32_t j) {
    if (j == 0) return true;
    const uint32_t d = s[0];
    uint32_t left = 0, right = 0;  // distance to the nearest stronger boundary (0: none in the window)
    for (uint32_t q = 1; q <= G && q <= j; ++q)
        if (s[-(int)q] > d) {
            left = q;
            break;
        }
    for (uint32_t q = 1; q <= G && j + q <= n; ++q)
        if (s[q] > d) {
            right = q;
            break;
        }
    return left == 0u || right == 0u || left + right > G;
}

// The level's size from the count of its Morton groups: fixed groups of G when those reduce too little.
RSH_DEV void level_size(uint32_t groups, uint32_t items, uint32_t l, uint32_t G, uint32_t& size, uint32_t& fixed) {
    fixed = ((l == 0 && 2ull * groups > (uint64_t)items + 1) || (l > 0 && 4ull * groups > (uint64_t)items + 3) ||
             groups == 0)
                ? 1u
                : 0u;
    size = fixed ? (items + G - 1) / G : groups;
}

// Node g of level l, whose children are the items [f, f1): its child-range start (triangle starts at level 0),
// its triangle start, its boxes and its sphere's centre; level 0 also its radius (squared). Returns nothing for
// a node outside the child-count invariant but raises RSH_DEVERR_OVERFLOW (its entry then lists 1 or 8).
// A node's padded box holds its child link in the spare w words, as raw u32 bits. A cluster (level 0): lo.w =
// its first triangle, hi.w = its triangle count. A node of level l >= 1: lo.w = its whole single-ray job-stack
// entry, l << 27 | (children - 1) << 24 | absolute node index of its first child (`child_off` + the level's
// child-range start), hi.w = its child count. A single ray that tests a node's box pushes that word as it is
// and, when it pops it, loads the children's boxes directly, with no child-range lookup in between.
RSH_DEV void write_node(const float4* tris, const RawBox* child_raw, uint32_t l, uint32_t g, uint32_t f, uint32_t f1,
                        uint32_t child_off, RawBox* raw, float4* sph, float4* box, float pad, uint32_t* err) {
    const float inf = __int_as_float(0x7f800000);
    float mn[3] = {inf, inf, inf}, mx[3] = {-inf, -inf, -inf};
    if (l == 0) {
        for (uint64_t v = 3ull * f; v < 3ull * f1; ++v) {
            const float4 p = ld_chain(tris + v);
            mn[0] = fminf(mn[0], p.x), mn[1] = fminf(mn[1], p.y), mn[2] = fminf(mn[2], p.z);
            mx[0] = fmaxf(mx[0], p.x), mx[1] = fmaxf(mx[1], p.y), mx[2] = fmaxf(mx[2], p.z);
        }
    } else {
        for (uint32_t c = f; c < f1; ++c) {
            const RawBox b = child_raw[c];
            for (int a = 0; a < 3; ++a) {
                mn[a] = fminf(mn[a], b.lo[a]);
                mx[a] = fmaxf(mx[a], b.hi[a]);
            }
        }
    }
    uint32_t link = f, n = f1 - f;  // level 0: the first triangle and the count
    if (l > 0u) {
        if (f1 <= f || n > 8u) {
            raise_device_error(err, RSH_DEVERR_OVERFLOW);
            n = f1 <= f ? 1u : 8u;
        }
        link = (l << 27) | ((n - 1u) << 24) | ((child_off + f) & 0xFFFFFFu);
    }
    for (int a = 0; a < 3; ++a) {
        raw[g].lo[a] = mn[a];
        raw[g].hi[a] = mx[a];
    }
    box[2ull * g] = make_float4(mn[0] - pad, mn[1] - pad, mn[2] - pad, __uint_as_float(link));
    box[2ull * g + 1] = make_float4(mx[0] + pad, mx[1] + pad, mx[2] + pad, __uint_as_float(f1 - f));
    const v3 c = v3{(mn[0] + mx[0]) * 0.5f, (mn[1] + mx[1]) * 0.5f, (mn[2] + mx[2]) * 0.5f};
    float r2 = 0.f;
    if (l == 0)
        for (uint64_t v = 3ull * f; v < 3ull * f1; ++v) {
            const float4 p = ld_chain(tris + v);
            const v3 d = v3{p.x - c.x, p.y - c.y, p.z - c.z};
            r2 = fmaxf(r2, dot3(d, d));
        }
    sph[g] = make_float4(c.x, c.y, c.z, r2);
}

// the arrays of every level (indexed like ObjHierarchy's, tstart like kids)
struct LevelArrays {
    const float4* tris;
    const uint32_t* dtri;
    uint32_t n;        // triangles
    uint32_t cluster;
    Level* lv;         // 16 records, then the launch's own
    uint32_t* kids;
    uint32_t* tstart;
    RawBox* raw;
    float4* sph;
    float4* box;
    float pad;
    uint32_t* err;
};

// items of level l and whether the level exists (the one below it has more than 8 nodes)
RSH_DEV bool level_items(const LevelArrays& A, uint32_t l, uint32_t& items, uint32_t& off, const uint32_t*& start) {
    if (l == 0) {
        items = A.n;
        off = 0;
        start = nullptr;
        return true;
    }
    const Level& p = A.lv[l - 1];
    items = p.size;
    off = p.off + p.size;
    start = A.tstart + p.off + (l - 1);
    return items > 8u;
}

}  // namespace

// One level's cuts, compacted: firsts[k] = the first item of Morton group k. The last tile writes the level's
// record (size 0: the level does not exist).
__global__ void __launch_bounds__(LV_TILE)
k_level_cuts(LevelArrays A, uint32_t l, uint32_t* firsts, unsigned long long* status,
             uint32_t* ticket) {
    chain();
    __shared__ uint32_t s_tile, s_warp[LV_TILE / 32], s_delta[LV_TILE + 2 * MAX_G];
    __shared__ unsigned long long s_excl;
    uint32_t items, off;
    const uint32_t* start;
    const uint32_t G = l == 0 ? A.cluster : 8u;
    if (!level_items(A, l, items, off, start)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) A.lv[l] = Level{0u, off, 0u};
        return;
    }
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile, tiles = (items + LV_TILE - 1) / LV_TILE;
    if (tile >= tiles) return;
    const uint32_t j = tile * LV_TILE + threadIdx.x, lane = lane_id(), warp = threadIdx.x >> 5;
    load_deltas(s_delta, A.dtri, start, items, (int64_t)tile * LV_TILE - MAX_G, LV_TILE + 2 * MAX_G);
    __syncthreads();
    const bool cut = j < items && is_cut(s_delta + MAX_G + threadIdx.x, items, G, j);
    const uint32_t bal = __ballot_sync(0xffffffffu, cut);
    if (lane == 0) s_warp[warp] = __popc(bal);
    __syncthreads();
    if (warp == 0) {
        uint32_t sum = lane < LV_TILE / 32 ? s_warp[lane] : 0u;
        sum = __reduce_add_sync(0xffffffffu, sum);
        const unsigned long long ex = look_back2(status, tile, sum, l + 1u, A.err);
        if (lane == 0) {
            s_excl = ex;
            if (tile == tiles - 1) {
                Level r{0u, off, 0u};
                if (ex != LB_FAILED) level_size((uint32_t)ex + sum, items, l, G, r.size, r.fixed);
                A.lv[l] = r;
            }
        }
    }
    __syncthreads();
    if (s_excl == LB_FAILED || !cut) return;
    uint32_t k = (uint32_t)s_excl + __popc(bal & lanemask_lt());
    for (uint32_t w = 0; w < warp; ++w) k += s_warp[w];
    firsts[k] = j;
}

// Node g of the new level: children [firsts[g], firsts[g+1]) of the items, triangles
// [start(firsts[g]), start(firsts[g+1])).
__global__ void __launch_bounds__(128) k_level_nodes(LevelArrays A, uint32_t l, const uint32_t* firsts) {
    chain();
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t items, off;
    const uint32_t* start;
    if (!level_items(A, l, items, off, start)) return;
    const Level r = A.lv[l];
    const uint32_t G = l == 0 ? A.cluster : 8u;
    if (r.size == 0u || g > r.size) return;
    auto first = [&](uint32_t q) -> uint32_t { return q >= r.size ? items : r.fixed ? q * G : firsts[q]; };
    const uint32_t f = first(g);
    const uint32_t ts = f >= items ? A.n : (start ? start[f] : f);
    A.kids[off + l + g] = f;  // level 0: items are triangles, so f is the triangle start
    A.tstart[off + l + g] = ts;
    if (g < r.size)
        write_node(A.tris, l ? A.raw + A.lv[l - 1].off : nullptr, l, g, f, first(g + 1), l ? A.lv[l - 1].off : 0u,
                   A.raw + off, A.sph + off, A.box + 2ull * off, A.pad, A.err);
}

// Every level from l0 on (over at most TAIL_ITEMS items) in one block: cuts, a block scan, nodes.
__global__ void __launch_bounds__(TAIL_THREADS) k_level_tail(LevelArrays A, uint32_t l0, uint32_t* firsts) {
    chain();
    __shared__ uint32_t s_warp[32], s_total, s_delta[TAIL_ITEMS + 2 * MAX_G];
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    constexpr uint32_t PER = TAIL_ITEMS / TAIL_THREADS;
    for (uint32_t l = l0; l < 16; ++l) {
        uint32_t items, off;
        const uint32_t* start;
        const bool some = level_items(A, l, items, off, start) && items <= TAIL_ITEMS;
        if (!some) {
            if (threadIdx.x == 0) A.lv[l] = Level{0u, off, 0u};
            __syncthreads();
            continue;
        }
        const uint32_t G = l == 0 ? A.cluster : 8u;
        load_deltas(s_delta, A.dtri, start, items, -(int64_t)MAX_G, items + 2 * MAX_G);
        __syncthreads();
        uint32_t cuts = 0;
        for (uint32_t i = 0; i < PER; ++i) {
            const uint32_t j = threadIdx.x * PER + i;
            if (j < items && is_cut(s_delta + MAX_G + j, items, G, j)) cuts |= 1u << i;
        }
        uint32_t x = __popc(cuts);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= (uint32_t)d) x += y;
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t v = s_warp[lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= (uint32_t)d) v += y;
            }
            s_warp[lane] = v;
            if (lane == 31) s_total = v;
        }
        __syncthreads();
        uint32_t k = (warp ? s_warp[warp - 1] : 0u) + x - __popc(cuts);
        for (uint32_t i = 0; i < PER; ++i)
            if ((cuts >> i) & 1u) firsts[k++] = threadIdx.x * PER + i;
        Level r{0u, off, 0u};
        level_size(s_total, items, l, G, r.size, r.fixed);
        if (threadIdx.x == 0) A.lv[l] = r;
        __syncthreads();
        auto first = [&](uint32_t q) -> uint32_t { return q >= r.size ? items : r.fixed ? q * G : firsts[q]; };
        for (uint32_t g = threadIdx.x; g <= r.size; g += TAIL_THREADS) {
            const uint32_t f = first(g);
            A.kids[off + l + g] = f;
            A.tstart[off + l + g] = f >= items ? A.n : (start ? start[f] : f);
            if (g < r.size)
                write_node(A.tris, l ? A.raw + A.lv[l - 1].off : nullptr, l, g, f, first(g + 1),
                           l ? A.lv[l - 1].off : 0u, A.raw + off, A.sph + off, A.box + 2ull * off, A.pad, A.err);
        }
        __syncthreads();
    }
}

// The squared radii of every node above the clusters, in one pass over the vertices: a warp holds 32 triangles
// and goes down the levels from the top; of the node that holds its first triangle it knows the children, so
// eight lanes find the child that holds it (two dependent loads a level, against a binary search of every
// level). Where all 32 triangles lie in one node their largest distance from its centre is one atomic max (of a
// non-negative float's bits), else every lane's own.
__global__ void __launch_bounds__(256) k_level_radii(LevelArrays A) {
    chain();
    const uint32_t lane = lane_id(), t0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u, t = t0 + lane;
    if (t0 >= A.n) return;
    const uint32_t t1 = min(t0 + 31u, A.n - 1u);
    float4 p[3];
    const bool in = t < A.n;
    for (int v = 0; v < 3; ++v) p[v] = in ? ld_chain(A.tris + 3ull * t + v) : make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t size_l = lane < 16u ? A.lv[lane].size : 0u;
    const uint32_t some = __ballot_sync(0xffffffffu, size_l > 0u);
    if (some == 0u) return;  // a look-back gave up: no levels
    int l = 31 - __clz((int)some);
    uint32_t c0 = 0, c1 = A.lv[l].size;  // the nodes of level l among which t0's lies (the top level: at most 8)
    for (; l >= 1; --l) {
        const uint32_t off = A.lv[l].off;
        const uint32_t* ts = A.tstart + off + l;
        uint32_t g = c0;
        for (uint32_t c = c0; c < c1; c += 32) {  // one round: at most 8
            const uint32_t n = __popc(__ballot_sync(0xffffffffu, c + lane < c1 && ts[c + lane] <= t0));
            g += n;
        }
        if (g > c0) --g;
        const uint32_t* kids = A.kids + off + l;
        c0 = kids[g];
        c1 = kids[g + 1];
        const bool one = ts[g + 1] > t1;
        if (!one && in)
            while (ts[g + 1] <= t) ++g;
        const float4 c = A.sph[off + g];
        float r2 = 0.f;
        if (in)
            for (int v = 0; v < 3; ++v) {
                const v3 d = v3{p[v].x - c.x, p[v].y - c.y, p[v].z - c.z};
                r2 = fmaxf(r2, dot3(d, d));
            }
        if (one) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(r2));
            if (lane == 0) atomicMax(reinterpret_cast<uint32_t*>(&A.sph[off + g].w), m);
        } else if (in) {
            atomicMax(reinterpret_cast<uint32_t*>(&A.sph[off + g].w), __float_as_uint(r2));
        }
    }
}

__global__ void k_level_radii_end(const Level* lv, float4* sph) {
    chain();
    uint32_t total = 0;
    for (uint32_t l = 0; l < 16; ++l) total += lv[l].size;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < total; j += gridDim.x * blockDim.x)
        sph[j].w = sqrtf(sph[j].w) * kRadSlack;
}

namespace {

// node capacity: level 0 holds at most n nodes, every level above at most (size + 3) / 4
size_t node_capacity(uint32_t n) { return (size_t)n + (n + 2) / 3 + 64; }

struct ObjScratch {
    uint32_t *codes, *sorted_codes, *perm, *dtri, *firsts, *tstart, *tickets;
    unsigned long long* status;
    RawBox* raw;
    Level* lv;
    void* sort;
    void* box_tree;
};
size_t obj_layout(uint32_t n, char* base, ObjScratch* o) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + off : nullptr;
        off += (bytes + 255) & ~size_t(255);
        return p;
    };
    ObjScratch s;
    s.codes = reinterpret_cast<uint32_t*>(take(4ull * n));
    s.sorted_codes = reinterpret_cast<uint32_t*>(take(4ull * n));
    s.perm = reinterpret_cast<uint32_t*>(take(4ull * n));
    s.dtri = reinterpret_cast<uint32_t*>(take(4ull * (n + 1)));
    s.firsts = reinterpret_cast<uint32_t*>(take(4ull * (n + 1)));
    s.tstart = reinterpret_cast<uint32_t*>(take(4ull * (node_capacity(n) + 16)));
    s.raw = reinterpret_cast<RawBox*>(take(sizeof(RawBox) * node_capacity(n)));
    s.lv = reinterpret_cast<Level*>(take(sizeof(Level) * 16));
    s.tickets = reinterpret_cast<uint32_t*>(take(4 * 16));
    s.status = reinterpret_cast<unsigned long long*>(take(8ull * ((n + LV_TILE - 1) / LV_TILE + 1)));
    s.sort = take(sort_scratch_bytes(n, 30));
    s.box_tree = take(box_tree_scratch_bytes(n));
    if (o) *o = s;
    return off;
}

template <class T>
cudaError_t fit(T*& p, size_t count) {
    return cudaMalloc(reinterpret_cast<void**>(&p), sizeof(T) * (count ? count : 1));
}

}  // namespace

size_t objh_scratch_bytes(uint32_t tri_count) { return obj_layout(tri_count ? tri_count : 1, nullptr, nullptr); }

void free_object_hierarchy(ObjHierarchy& h) {
    for (void* p : {(void*)h.spheres, (void*)h.kids, (void*)h.tris, (void*)h.order, (void*)h.boxes, (void*)h.wboxes,
                    (void*)h.wtris, (void*)h.wnodes})
        if (p) cudaFree(p);
    h = ObjHierarchy();
}

size_t object_hierarchy_bytes(const ObjHierarchy& h) {
    if (!h.wtris) return 0;
    const size_t n = h.tri_count, cap = node_capacity(h.tri_count);
    return (16 + 4 + 32) * cap + 4 * 16 + (48 + 4) * n + 32 * (2 * n + 8) + 48 * n + 16 * REC_F4 * (size_t)h.wnode_cap;
}

cudaError_t build_object_hierarchy(const float4* positions_dev, uint32_t n, uint32_t cluster,
                                   const float lo[3], const float hi[3], ObjHierarchy& h,
                                   void* scratch, uint32_t* err, cudaStream_t s, cudaStream_t side, void* host) {
    h.levels = 0;
    h.wslots = 0;
    h.wroot = 0;
    if (h.tri_count != n || !h.wtris) {  // a rebuild over the same triangles keeps its arrays
        free_object_hierarchy(h);
        const size_t cap = node_capacity(n);
        cudaError_t e;
        if (n && ((e = fit(h.spheres, cap)) || (e = fit(h.kids, cap + 16)) || (e = fit(h.tris, 3ull * n)) ||
                  (e = fit(h.order, n)) || (e = fit(h.boxes, 2 * cap)) || (e = fit(h.wboxes, 2ull * (2ull * n + 8))) ||
                  (e = fit(h.wtris, 3ull * n)))) {
            free_object_hierarchy(h);
            return e;
        }
    }
    h.tri_count = n;
    h.cluster = cluster;
    if (n == 0) return cudaSuccess;
    cudaError_t e;
    ObjScratch w;
    obj_layout(n, static_cast<char*>(scratch), &w);
    // one scale for all axes (the cube over the largest extent): Morton bits follow physical size, so a
    // flat scene does not spend its high-order splits on its thin axis
    float ext = hi[0] - lo[0];
    if (hi[1] - lo[1] > ext) ext = hi[1] - lo[1];
    if (hi[2] - lo[2] > ext) ext = hi[2] - lo[2];
    const float sc1 = (ext > 0.0f) ? 1024.0f / ext : 0.0f;
    launch_chained(true, k_morton, (n + 255) / 256, 256, 0, s, positions_dev, n, v3{lo[0], lo[1], lo[2]},
                   v3{sc1, sc1, sc1}, w.codes);
    note_launch();
    e = launch_sort_pairs(w.codes, nullptr, w.sorted_codes, w.perm, n, nullptr, 30, w.sort, err, s);
    if (e != cudaSuccess) return e;
    launch_chained(true, k_gather_tris, (n + 255) / 256, 256, 0, s, positions_dev, w.perm, n, h.tris, h.order);
    launch_chained(true, k_delta_tri, (n + 256) / 256, 256, 0, s, w.sorted_codes, n, w.dtri);
    note_launch(2);
    // cluster boxes are widened by 1e-5 of the scene's largest coordinate magnitude: far more than the
    // rounding of a float slab test over the scene, so the box cull never drops a hit of the watertight test
    float smax = 0.0f;
    for (int a = 0; a < 3; ++a) smax = fmaxf(smax, fmaxf(fabsf(lo[a]), fabsf(hi[a])));
    const float box_pad = 1e-5f * smax + 1e-30f;
    // The levels and the box tree are independent chains of small launches over the same sorted triangles: side by
    // side (a frame of 1001 moving objects 1.31 -> 1.25 ms).
    if ((e = cudaMemsetAsync(w.tickets, 0, 64, s)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(w.status, 0, 8ull * ((n + LV_TILE - 1) / LV_TILE + 1), s)) != cudaSuccess) return e;
    cudaEvent_t sorted = nullptr;
    if ((e = cudaEventCreateWithFlags(&sorted, cudaEventDisableTiming)) != cudaSuccess) return e;
    if ((e = cudaEventRecord(sorted, s)) == cudaSuccess) e = cudaStreamWaitEvent(side, sorted, 0);
    cudaEventDestroy(sorted);
    if (e != cudaSuccess) return e;
    LevelArrays A{h.tris, w.dtri, n, cluster, w.lv, h.kids, w.tstart, w.raw, h.spheres, h.boxes, box_pad, err};
    uint64_t most = n;  // the most items level l can have
    uint32_t l = 0;
    for (; l < 16 && most > TAIL_ITEMS; ++l) {
        const uint32_t G = (l == 0) ? cluster : 8u;
        const uint64_t nodes = std::max<uint64_t>(l == 0 ? (most + 1) / 2 : (most + 3) / 4, (most + G - 1) / G);
        launch_chained(true, k_level_cuts, (uint32_t)((most + LV_TILE - 1) / LV_TILE), LV_TILE, 0, side, A, l, w.firsts,
                       w.status, w.tickets + l);
        launch_chained(true, k_level_nodes, (uint32_t)((nodes + 128) / 128), 128, 0, side, A, l, w.firsts);
        note_launch(2);
        most = nodes;
    }
    launch_chained(true, k_level_tail, 1, TAIL_THREADS, 0, side, A, l, w.firsts);
    launch_chained(true, k_level_radii, (n + 255) / 256, 256, 0, side, A);
    launch_chained(true, k_level_radii_end, (uint32_t)std::min<size_t>((node_capacity(n) + 255) / 256, 1216), 256, 0, side,
                   w.lv, h.spheres);
    note_launch(3);
    e = cudaGetLastError();
    // the single-ray box tree over the same Morton-ordered triangles, with the same padding
    if (e == cudaSuccess) e = build_box_tree(h, box_pad, w.box_tree, err, s, host);
    // whatever failed, nothing is left in flight on either stream
    static_assert(16 * sizeof(Level) <= BUILD_HOST_BYTES, "the levels fit");
    Level* lv = static_cast<Level*>(host);  // (the box tree's build is done with it)
    cudaError_t e2 = cudaMemcpyAsync(lv, w.lv, 16 * sizeof(Level), cudaMemcpyDeviceToHost, side);
    for (const cudaStream_t q : {side, s}) {
        const cudaError_t e3 = cudaStreamSynchronize(q);
        if (e2 == cudaSuccess) e2 = e3;
    }
    if (e != cudaSuccess) return e;
    if (e2 != cudaSuccess) return e2;
    for (uint32_t i = 0; i < 16 && lv[i].size; ++i) {
        h.level_off[i] = lv[i].off;
        h.level_size[i] = lv[i].size;
        h.levels = i + 1;
    }
    if (h.levels == 0 || h.level_off[h.levels - 1] + h.level_size[h.levels - 1] > node_capacity(n))
        return cudaErrorInvalidValue;
    return cudaSuccess;
}

}  // namespace rsh
