// The single-ray box tree: an 8-wide bounding-volume tree over the scene's triangles that the batched form's
// rays-only kernel (fused.cu k_fused_rays) descends. It is built beside the object-sphere hierarchy (objh.cu),
// which the packet traversals and the exported level structure keep using.
//
// Build, from the triangles in the object hierarchy's Morton order:
//  1. A binary tree by PLOC (Meister & Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
//     Hierarchy Construction", IEEE TVCG 2018): every pass, each cluster finds the neighbour within R
//     positions of the Morton-ordered cluster list whose merged box has the smallest surface area (ties to
//     the nearer-indexed one), mutual nearest neighbours merge (the merged node takes the lower position),
//     and the list is compacted in order, until one cluster is left. A node's surface-area measure is
//     (x y + y z) + x z of its box extents, all in FP32, so the host restatement builds the same tree.
//  2. Triangles laid out in the binary tree's depth-first order (left first), so every subtree's triangles
//     are one contiguous range.
//  3. Collapse to 8-wide nodes by the surface-area cost of the single-ray traversal, chosen by dynamic
//     programming over the binary tree (children before parents, pass by pass): with A(x) the area
//     measure of subtree x, f(x, k) = the least cost of covering x's subtree with exactly k child slots
//     of its parent: f(x, 1) = min(A(x) (8 + triangles) if x has at most `cluster` triangles (a cluster),
//     min over 2 <= j <= 8 of A(x) (16 + j) + f(x, j) (a node with j children)), ties to the cluster and
//     to the smaller j; f(x, k >= 2) = min over 1 <= i < k of f(left, i) + f(right, k - i), ties to the
//     smaller i; a single triangle has only f(., 1). The weights (16 + children per node step, 8 +
//     triangles per cluster step) follow the traversal kernel, whose cost tracks its steps more than its
//     box tests. Every f is an FP32 sum in a fixed order, so the host restatement makes the same choices.
//     Then breadth first: a node's children are the slots of its decomposition (left parts first), in
//     consecutive slots allocated level after level in queue order.
// How the build is launched. It is a chain of many small dependent passes (47-55 PLOC passes for 0.3-1 M
// triangles, most over a few thousand clusters or fewer, then about 10 breadth-first levels), so launches,
// read-backs and allocations are what it pays for, not bytes: with a launch per scan step, a read-back per pass
// and a collapse and an order pass per PLOC pass it took 700 launches, 75 synchronisations and 40 allocations
// (2.6 ms of kernels and 2.2 ms of gaps for 320,032 triangles). Now a PLOC pass is one launch (neighbours from
// shared memory, positions and ids by look-back over tiles); the cluster count stays on the device, and once at
// most TAIL_CLUSTERS are left one block runs all remaining passes from shared memory. A merge computes its
// collapse costs at once (its children's are known) and tells its children how far right of it they start, so
// neither needs a pass of its own: a triangle's place in the depth-first order is the sum on its way up. A
// breadth-first level is one launch. 0.58 ms of kernels and 2 synchronisations for the same scene (a frame of 1001
// moving objects: 8.6 ms, then 1.8). The build's launches are chained: a pass's CTAs are placed while the one before
// it ends (the same frame 1.40 ms unchained, 1.31 chained).
// Slot layout (2 float4 per slot, padded box lo and hi): a cluster keeps its first triangle in lo.w and
// 0x80000000 | its triangle count in hi.w; a node keeps its single-ray stack entry in lo.w,
// 1 << 27 | (children - 1) << 24 | first child slot, and its child count in hi.w. Slot 0 is unused; the
// root's entry lists its children from slot 1.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace rsh {

namespace {

constexpr int PLOC_R = 8;  // PLOC search radius
constexpr uint32_t CLUSTER_BIT = 0x80000000u;
constexpr uint32_t PT = 256;              // positions per tile of a PLOC pass, items per tile of a level
constexpr uint32_t TAIL_CLUSTERS = 2048;  // clusters at which one block takes over
constexpr uint32_t TAIL_T = 1024;
constexpr uint32_t PLOC_BUNCH = 32;       // PLOC passes enqueued between read-backs
constexpr uint32_t BFS_BUNCH = 12;        // breadth-first levels enqueued between read-backs

struct WNode {
    float4 lo;  // box min xyz, w = triangle count (u32 bits)
    float4 hi;  // box max xyz
};

RSH_DEV float box_area(float4 a, float4 b) {
    const float x = b.x - a.x, y = b.y - a.y, z = b.z - a.z;
    return (x * y + y * z) + x * z;
}

// per node of the binary tree: f(x, 1..8) and its choices packed in one word -- bits 3 (k - 2) .. for the
// split i of f(x, k), k = 2..8; bits 21-23: j - 2 of the node choice; bit 24: x is a cluster
constexpr float COST_NODE = 16.0f, COST_CLUSTER = 8.0f;
constexpr uint32_t CH_CLUSTER = 1u << 24;

// The binary tree: ids 0 .. n - 1 are the triangles (in Morton order), n .. the merged nodes (whose arrays are
// indexed by id - n).
struct Tree {
    uint32_t n;        // triangles
    uint32_t cluster;
    WNode* box;        // every id
    int2* up;          // every id: parent (-1: the root), triangles left of it below the parent
    int2* ch;          // merged: left, right child
    float4* f;         // merged: f(x, 1..8), two float4
    uint32_t* choice;  // merged
    int32_t* left;     // merged: the leftmost triangle below
};

RSH_DEV void costs_of(const Tree& T, int32_t id, const WNode& w, float* f) {
    if ((uint32_t)id < T.n) {  // a triangle is always a cluster of one
        f[0] = box_area(w.lo, w.hi) * (COST_CLUSTER + 1.0f);
        for (int k = 1; k < 8; ++k) f[k] = __int_as_float(0x7f800000);
    } else {
        const float4 a = T.f[2ull * (id - T.n)], b = T.f[2ull * (id - T.n) + 1];
        f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w;
        f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
    }
}

// Merges clusters a (the lower position) and b into node id: box, children, their way up, collapse costs.
RSH_DEV void merge(const Tree& T, int32_t a, int32_t b, const WNode& p, const WNode& q, int32_t id, WNode& m) {
    const uint32_t ca = __float_as_uint(p.lo.w), cnt = ca + __float_as_uint(q.lo.w);
    m.lo = make_float4(fminf(p.lo.x, q.lo.x), fminf(p.lo.y, q.lo.y), fminf(p.lo.z, q.lo.z), __uint_as_float(cnt));
    m.hi = make_float4(fmaxf(p.hi.x, q.hi.x), fmaxf(p.hi.y, q.hi.y), fmaxf(p.hi.z, q.hi.z), 0.f);
    T.box[id] = m;
    T.ch[id - T.n] = make_int2(a, b);
    T.up[a] = make_int2(id, 0);
    T.up[b] = make_int2(id, (int32_t)ca);
    T.left[id - T.n] = (uint32_t)a < T.n ? a : T.left[a - T.n];
    float fl[8], fr[8], f[8];
    costs_of(T, a, p, fl);
    costs_of(T, b, q, fr);
    uint32_t ch = 0;
    const float inf = __int_as_float(0x7f800000);
#pragma unroll
    for (uint32_t k = 2; k <= 8; ++k) {
        float best = inf;
        uint32_t bi = 1;
#pragma unroll
        for (uint32_t i = 1; i < k; ++i) {
            const float c = fl[i - 1] + fr[k - i - 1];
            if (c < best) {
                best = c;
                bi = i;
            }
        }
        f[k - 1] = best;
        ch |= bi << (3u * (k - 2u));
    }
    const float A = box_area(m.lo, m.hi);
    float best = inf;
    uint32_t bj = 0;
#pragma unroll
    for (uint32_t j = 2; j <= 8; ++j) {
        const float c = A * (COST_NODE + (float)j) + f[j - 1];
        if (c < best) {
            best = c;
            bj = j;
        }
    }
    const float ccl = cnt <= T.cluster ? A * (COST_CLUSTER + (float)cnt) : inf;
    if (ccl <= best) {
        f[0] = ccl;
        ch |= CH_CLUSTER;
    } else {
        f[0] = best;
        ch |= (bj - 2u) << 21;
    }
    T.f[2ull * (id - T.n)] = make_float4(f[0], f[1], f[2], f[3]);
    T.f[2ull * (id - T.n) + 1] = make_float4(f[4], f[5], f[6], f[7]);
    T.choice[id - T.n] = ch;
}

// the state before a PLOC pass: clusters left, the next node id, which of the two lists holds them
struct Ploc {
    uint32_t m, next_id, src, pad;
};

__global__ void k_wide_leaves(const float4* tris, Tree T, int32_t* list,
                              Ploc* st) {
    chain();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) st[0] = Ploc{T.n, T.n, 0u, 0u};
    if (k >= T.n) return;
    const float4 a = ld_chain(tris + 3ull * k), b = ld_chain(tris + 3ull * k + 1), c = ld_chain(tris + 3ull * k + 2);
    WNode w;
    w.lo = make_float4(fminf(fminf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z),
                       __uint_as_float(1u));
    w.hi = make_float4(fmaxf(fmaxf(a.x, b.x), c.x), fmaxf(fmaxf(a.y, b.y), c.y), fmaxf(fmaxf(a.z, b.z), c.z), 0.f);
    T.box[k] = w;
    T.up[k] = make_int2(-1, 0);
    list[k] = (int32_t)k;
}

// The neighbour within PLOC_R positions of position i (boxes of the positions around it in shared memory, at
// index i - i0, plane by plane, `stride` floats each) whose merged box is smallest; ties: the lower position.
RSH_DEV int32_t nearest(const float* s, uint32_t stride, int64_t i0, uint32_t i, uint32_t m) {
    const float* me = s + (int64_t)i - i0;
    const float ax = me[0], ay = me[stride], az = me[2 * stride], bx = me[3 * stride], by = me[4 * stride],
                bz = me[5 * stride];
    float best = __int_as_float(0x7f800000);
    int32_t bj = -1;
    // fixed offsets, unrolled: the loads of all neighbours are in flight together
#pragma unroll
    for (int d = -PLOC_R; d <= PLOC_R; ++d) {
        if (d == 0) continue;
        const int32_t j = (int32_t)i + d;
        if (j >= 0 && j < (int32_t)m) {
            const float* q = me + d;
            const float a = box_area(make_float4(fminf(ax, q[0]), fminf(ay, q[stride]), fminf(az, q[2 * stride]), 0.f),
                                     make_float4(fmaxf(bx, q[3 * stride]), fmaxf(by, q[4 * stride]),
                                                 fmaxf(bz, q[5 * stride]), 0.f));
            if (a < best) {
                best = a;
                bj = j;
            }
        }
    }
    return bj;
}

// One PLOC pass over the clusters of list st[p].src, into the other list: mutual nearest neighbours merge, the
// merged node takes the lower position. Each tile finds its own neighbours' neighbours too (PLOC_R positions
// either side), so nothing waits between the search and the merges; where its clusters go and which ids its
// merges take comes from a look-back over the tiles before it.
constexpr uint32_t PT_THREADS = PT + 4 * PLOC_R;  // a thread per position loaded: one round for each step
__global__ void __launch_bounds__(PT_THREADS)
k_ploc_pass(Tree T, Ploc* st, uint32_t p, int32_t* list0, int32_t* list1, unsigned long long* status,
            uint32_t* ticket, uint32_t epoch, uint32_t* err) {
    chain();
    constexpr uint32_t W = PT_THREADS;
    __shared__ float s_box[6 * W];
    __shared__ int32_t s_id[W], s_nn[PT + 2 * PLOC_R];
    __shared__ uint32_t s_tile, s_cnt[PT / 32];
    __shared__ unsigned long long s_excl;
    const Ploc cur = st[p];
    const uint32_t m = cur.m, t = threadIdx.x, lane = lane_id(), warp = t >> 5;
    if (m <= TAIL_CLUSTERS) {  // left to k_ploc_tail
        if (blockIdx.x == 0 && t == 0) st[p + 1] = cur;
        return;
    }
    if (t == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile, tiles = (m + PT - 1) / PT;
    if (tile >= tiles) return;
    const int32_t* src = cur.src ? list1 : list0;
    int32_t* dst = cur.src ? list0 : list1;
    const uint32_t base = tile * PT;
    const int64_t i0 = (int64_t)base - 2 * PLOC_R;
    {
        const int64_t i = i0 + t;
        if (i >= 0 && i < (int64_t)m) {
            const int32_t id = src[i];
            const WNode w = T.box[id];
            s_id[t] = id;
            s_box[t] = w.lo.x, s_box[W + t] = w.lo.y, s_box[2 * W + t] = w.lo.z;
            s_box[3 * W + t] = w.hi.x, s_box[4 * W + t] = w.hi.y, s_box[5 * W + t] = w.hi.z;
        }
    }
    __syncthreads();
    if (t < PT + 2 * PLOC_R) {
        const int64_t i = (int64_t)base - PLOC_R + t;
        s_nn[t] = i >= 0 && i < (int64_t)m ? nearest(s_box, W, i0, (uint32_t)i, m) : -1;
    }
    __syncthreads();
    const uint32_t i = t < PT ? base + t : m;  // the last warp holds no position of the tile
    const int32_t j = i < m ? s_nn[t + PLOC_R] : -1;
    const bool mutual = j >= 0 && s_nn[j - (int32_t)base + PLOC_R] == (int32_t)i;
    const bool lower = mutual && (int32_t)i < j, gone = mutual && (int32_t)i > j;
    const uint32_t bl = __ballot_sync(0xffffffffu, lower), bg = __ballot_sync(0xffffffffu, gone);
    if (lane == 0 && warp < PT / 32) s_cnt[warp] = __popc(bl) | (__popc(bg) << 16);
    __syncthreads();
    if (warp == 0) {
        uint32_t c = lane < PT / 32 ? s_cnt[lane] : 0u;
        c = __reduce_add_sync(0xffffffffu, c);
        const unsigned long long sum = (unsigned long long)(c & 0xFFFFu) | ((unsigned long long)(c >> 16) << 24);
        const unsigned long long ex = look_back2(status, tile, sum, epoch, err);
        if (lane == 0) {
            s_excl = ex;
            if (tile == tiles - 1) {
                const unsigned long long all = ex + sum;
                const uint32_t merges = (uint32_t)all & 0xFFFFFFu, removed = (uint32_t)(all >> 24) & 0xFFFFFFu;
                st[p + 1] = ex == LB_FAILED ? Ploc{0u, cur.next_id, 0u, 0u}
                                            : Ploc{m - removed, cur.next_id + merges, cur.src ^ 1u, 0u};
            }
        }
    }
    __syncthreads();
    if (s_excl == LB_FAILED || i >= m || gone) return;
    uint32_t nl = (uint32_t)s_excl & 0xFFFFFFu, ng = (uint32_t)(s_excl >> 24) & 0xFFFFFFu;
    for (uint32_t w = 0; w < warp; ++w) {
        nl += s_cnt[w] & 0xFFFFu;
        ng += s_cnt[w] >> 16;
    }
    nl += __popc(bl & lanemask_lt());
    ng += __popc(bg & lanemask_lt());
    int32_t id = s_id[t + 2 * PLOC_R];
    if (lower) {
        const int32_t a = id, b = s_id[j - (int32_t)base + 2 * PLOC_R];
        WNode mm;
        id = (int32_t)(cur.next_id + nl);
        merge(T, a, b, T.box[a], T.box[b], id, mm);
    }
    dst[i - ng] = id;
}

// All remaining passes in one block, the clusters' boxes and ids in shared memory (two copies in turn). Leaves
// the root in *root (-1: the passes did not get this far, or nothing merged).
struct TailSmem {
    float box[2][6 * TAIL_CLUSTERS];
    uint32_t cnt[2][TAIL_CLUSTERS];
    int32_t id[2][TAIL_CLUSTERS];
    int32_t nn[TAIL_CLUSTERS];
    uint32_t warp[TAIL_T / 32];
};
__global__ void __launch_bounds__(TAIL_T)
k_ploc_tail(Tree T, const Ploc* st, const int32_t* list0, const int32_t* list1, int32_t* root) {
    chain();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TailSmem& S = *reinterpret_cast<TailSmem*>(smem_raw);
    constexpr uint32_t W = TAIL_CLUSTERS, PER = TAIL_CLUSTERS / TAIL_T;
    const uint32_t t = threadIdx.x, lane = lane_id(), warp = t >> 5;
    uint32_t m = st->m, next_id = st->next_id, c = 0;
    if (m == 0u || m > TAIL_CLUSTERS) {
        if (t == 0) *root = -1;
        return;
    }
    const int32_t* src = st->src ? list1 : list0;
    for (uint32_t i = t; i < m; i += TAIL_T) {
        const int32_t id = src[i];
        const WNode w = T.box[id];
        S.id[0][i] = id;
        S.cnt[0][i] = __float_as_uint(w.lo.w);
        float* b = S.box[0];
        b[i] = w.lo.x, b[W + i] = w.lo.y, b[2 * W + i] = w.lo.z;
        b[3 * W + i] = w.hi.x, b[4 * W + i] = w.hi.y, b[5 * W + i] = w.hi.z;
    }
    __syncthreads();
    auto node = [&](uint32_t k, uint32_t i) {
        const float* b = S.box[k];
        WNode w;
        w.lo = make_float4(b[i], b[W + i], b[2 * W + i], __uint_as_float(S.cnt[k][i]));
        w.hi = make_float4(b[3 * W + i], b[4 * W + i], b[5 * W + i], 0.f);
        return w;
    };
    while (m > 1u) {
        for (uint32_t i = t; i < m; i += TAIL_T) S.nn[i] = nearest(S.box[c], W, 0, i, m);
        __syncthreads();
        // PER consecutive positions a thread: how many lower halves of a pair and how many removed ones
        uint32_t low = 0, gone = 0;
#pragma unroll
        for (uint32_t q = 0; q < PER; ++q) {
            const uint32_t i = t * PER + q;
            if (i >= m) continue;
            const int32_t j = S.nn[i];
            if (j >= 0 && S.nn[j] == (int32_t)i) {
                if ((int32_t)i < j) low |= 1u << q;
                else gone |= 1u << q;
            }
        }
        const uint32_t own = __popc(low) | (__popc(gone) << 16);
        uint32_t x = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= (uint32_t)d) x += y;
        }
        if (lane == 31) S.warp[warp] = x;
        __syncthreads();
        uint32_t before = 0, all = 0;
        {
            uint32_t v = S.warp[lane];  // TAIL_T / 32 == 32 warps
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= (uint32_t)d) v += y;
            }
            all = __shfl_sync(0xffffffffu, v, 31);
            before = warp ? __shfl_sync(0xffffffffu, v, (int)warp - 1) : 0u;
        }
        before += x - own;
        const uint32_t merges = all & 0xFFFFu;
        if (merges == 0u) break;
        uint32_t nl = before & 0xFFFFu, ng = before >> 16;
#pragma unroll
        for (uint32_t q = 0; q < PER; ++q) {
            const uint32_t i = t * PER + q;
            if (i >= m) continue;
            if ((gone >> q) & 1u) {
                ++ng;
                continue;
            }
            int32_t id = S.id[c][i];
            WNode w = node(c, i);
            if ((low >> q) & 1u) {
                const uint32_t j = (uint32_t)S.nn[i];
                const int32_t a = id;
                id = (int32_t)(next_id + nl++);
                WNode mm;
                merge(T, a, S.id[c][j], w, node(c, j), id, mm);
                w = mm;
            }
            const uint32_t k = i - ng;
            float* b = S.box[c ^ 1u];
            S.id[c ^ 1u][k] = id;
            S.cnt[c ^ 1u][k] = __float_as_uint(w.lo.w);
            b[k] = w.lo.x, b[W + k] = w.lo.y, b[2 * W + k] = w.lo.z;
            b[3 * W + k] = w.hi.x, b[4 * W + k] = w.hi.y, b[5 * W + k] = w.hi.z;
        }
        next_id += merges;
        m -= all >> 16;
        c ^= 1u;
        __syncthreads();  // the new list is whole (and the costs that a later merge reads are written)
    }
    if (t == 0) {
        *root = m == 1u ? S.id[c][0] : -1;
        if (m == 1u) T.up[S.id[c][0]] = make_int2(-1, 0);
    }
}

// Every triangle's depth-first position: the sum of what lies left of it on the way up.
__global__ void k_wide_tris(const float4* tris, uint32_t n, const int2* up,
                            const int32_t* root, uint32_t* first, float4* out) {
    chain();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || *root < 0) return;
    uint32_t f = 0;
    for (int2 u = ld_chain(up + k); u.x >= 0; u = ld_chain(up + u.x)) f += (uint32_t)u.y;
    first[k] = f;
    const uint64_t d = 3ull * f;
    out[d] = ld_chain(tris + 3ull * k);
    out[d + 1] = ld_chain(tris + 3ull * k + 1);
    out[d + 2] = ld_chain(tris + 3ull * k + 2);
}

// One breadth-first level of the collapse: the slots [base, base + count); `recs`: nodes (records) before it.
struct Bfs {
    uint32_t base, count, recs, pad;
};

__global__ void k_bfs_init(const int32_t* root, int32_t* item, Bfs* lv,
                           float4* boxes) {
    chain();
    item[0] = *root;
    lv[0] = Bfs{0u, *root >= 0 ? 1u : 0u, 0u, 0u};
    boxes[0] = boxes[1] = make_float4(0.f, 0.f, 0.f, 0.f);  // slot 0 is unused
}

// Every slot of level l: a node's children (its decomposition into the j slots its choice says, left parts
// first) take the next slots in order and the node the next record; a cluster has none. Slot 0 stands for the
// root, which has no slot of its own; a root that is a cluster is its own single child. Writes the slot's box
// and words (cluster: triangle range; node: its stack entry), rec_of[slot] for nodes, and rec_kids[record] =
// the stack entry of the record's children.
__global__ void __launch_bounds__(PT)
k_bfs_level(Tree T, const uint32_t* first, Bfs* lv, uint32_t l, int32_t* item, uint32_t* rec_of, uint32_t* rec_kids, float pad,
            float4* boxes, unsigned long long* status, uint32_t* ticket, uint32_t epoch, uint32_t* err) {
    chain();
    __shared__ uint32_t s_tile, s_kids[PT / 32], s_recs[PT / 32];
    __shared__ unsigned long long s_excl;
    const Bfs cur = lv[l];
    const uint32_t t = threadIdx.x, lane = lane_id(), warp = t >> 5;
    if (cur.count == 0u) {
        if (blockIdx.x == 0 && t == 0) lv[l + 1] = cur;
        return;
    }
    if (t == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile, tiles = (cur.count + PT - 1) / PT;
    if (tile >= tiles) return;
    const uint32_t i = tile * PT + t;
    const bool in = i < cur.count;
    const uint32_t slot = cur.base + i;
    int32_t kid[8];
    uint32_t m = 0;
    int32_t x = 0;
    if (in) {
        x = item[slot];
        const uint32_t cx = (uint32_t)x < T.n ? CH_CLUSTER : T.choice[x - T.n];
        if (cx & CH_CLUSTER) {
            if (slot == 0u) kid[m++] = x;
        } else {
            int32_t sy[8];
            uint32_t sk[8], top = 1;
            sy[0] = x;
            sk[0] = ((cx >> 21) & 7u) + 2u;
            while (top > 0) {
                --top;
                const int32_t y = sy[top];
                const uint32_t k = sk[top];
                if (k == 1u) {
                    kid[m++] = y;
                    continue;
                }
                // only a merged node has a finite cost of two slots or more
                const uint32_t si = (T.choice[y - T.n] >> (3u * (k - 2u))) & 7u;
                const int2 lr = T.ch[y - T.n];
                sy[top] = lr.y;  // the right part after the left one
                sk[top] = k - si;
                sy[top + 1] = lr.x;
                sk[top + 1] = si;
                top += 2;
            }
        }
    }
    uint32_t inc = m;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= (uint32_t)d) inc += y;
    }
    const uint32_t isn = __ballot_sync(0xffffffffu, m > 0u);
    if (lane == 31) {
        s_kids[warp] = inc;
        s_recs[warp] = __popc(isn);
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t ck = lane < PT / 32 ? s_kids[lane] : 0u, cr = lane < PT / 32 ? s_recs[lane] : 0u;
        ck = __reduce_add_sync(0xffffffffu, ck);
        cr = __reduce_add_sync(0xffffffffu, cr);
        const unsigned long long sum = (unsigned long long)ck | ((unsigned long long)cr << 24);
        const unsigned long long ex = look_back2(status, tile, sum, epoch, err);
        if (lane == 0) {
            s_excl = ex;
            if (tile == tiles - 1) {
                const unsigned long long all = ex + sum;
                // the root level's slot 0 is followed by slot 1, every level's end by the next one's start
                lv[l + 1] = ex == LB_FAILED ? Bfs{0u, 0u, 0u, 0u}
                                            : Bfs{cur.base + cur.count, (uint32_t)all & 0xFFFFFFu,
                                                  cur.recs + ((uint32_t)(all >> 24) & 0xFFFFFFu), 0u};
            }
        }
    }
    __syncthreads();
    if (s_excl == LB_FAILED || !in) return;
    uint32_t ko = (uint32_t)s_excl & 0xFFFFFFu, ro = (uint32_t)(s_excl >> 24) & 0xFFFFFFu;
    for (uint32_t w = 0; w < warp; ++w) {
        ko += s_kids[w];
        ro += s_recs[w];
    }
    const uint32_t f = cur.base + cur.count + ko + inc - m, r = cur.recs + ro + __popc(isn & lanemask_lt());
    const WNode w = T.box[x];
    uint32_t lw, hw;
    if (m == 0u) {  // a cluster
        lw = ld_chain(first + ((uint32_t)x < T.n ? x : T.left[x - T.n]));
        hw = CLUSTER_BIT | __float_as_uint(w.lo.w);
    } else {
        lw = (1u << 27) | ((m - 1u) << 24) | (f & 0xFFFFFFu);
        hw = m;
        rec_of[slot] = r;
        rec_kids[r] = lw;
        for (uint32_t q = 0; q < m; ++q) item[f + q] = kid[q];
    }
    if (slot == 0u) return;  // the root has no slot of its own
    boxes[2ull * slot] = make_float4(w.lo.x - pad, w.lo.y - pad, w.lo.z - pad, __uint_as_float(lw));
    boxes[2ull * slot + 1] = make_float4(w.hi.x + pad, w.hi.y + pad, w.hi.z + pad, __uint_as_float(hw));
}

// Traversal records: the slot tree laid out again for the rays-only kernel, one record per node (in slot
// order, so the root's children are record 0), REC_F4 float4 each: the eight children's padded boxes plane by
// plane (lo x, hi x, lo y, hi y, lo z, hi z: 8 floats each) and their eight stack entries. A ray picks the near
// and the far plane of each axis once per record from the sign of its direction, so a child's entry and exit
// distances need no min / max per axis. An unused child has the empty box (lo = +inf, hi = -inf, which every
// ray misses) and entry 0. A child's entry: a cluster's first triangle | (triangles - 1) << 23 (bit 31 clear;
// fewer than 2^23 triangles, at most 64 per cluster), or a node's REC_NODE | (children - 1) << 28 | record
// index (kernels.h). Eight lanes a record, one per child.
__global__ void k_rec_write(const float4* boxes, uint32_t recs, const uint32_t* rec_kids,
                            const uint32_t* rec_of, float4* out) {
    chain();
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t rec = g >> 3, c = g & 7u;
    if (rec >= recs) return;
    const uint32_t k = rec_kids[rec], n = ((k >> 24) & 7u) + 1u, slot = (k & 0xFFFFFFu) + c;
    const float inf = __int_as_float(0x7f800000);
    float4 b0 = make_float4(inf, inf, inf, 0.f), b1 = make_float4(-inf, -inf, -inf, 0.f);
    uint32_t entry = 0u;
    if (c < n) {
        b0 = boxes[2ull * slot];
        b1 = boxes[2ull * slot + 1];
        const uint32_t lw = __float_as_uint(b0.w), hw = __float_as_uint(b1.w);
        entry = (hw & CLUSTER_BIT) ? lw | ((hw - CLUSTER_BIT - 1u) << 23)
                                   : REC_NODE | (((lw >> 24) & 7u) << 28) | rec_of[slot];
    }
    float* r = reinterpret_cast<float*>(out + REC_F4 * (size_t)rec) + c;
    r[0] = b0.x, r[8] = b1.x;
    r[16] = b0.y, r[24] = b1.y;
    r[32] = b0.z, r[40] = b1.z;
    reinterpret_cast<uint32_t*>(r)[48] = entry;
}

// What the host reads of a build.
struct State {
    int32_t root, pad[3];
    Ploc ploc[PLOC_BUNCH + 1];
    Bfs bfs[BFS_BUNCH + 1];
};

struct Scratch {
    State* state = nullptr;  // root, ploc and bfs point into it
    Tree T;
    int32_t *list0, *list1, *root, *item;
    uint32_t *first, *rec_of, *rec_kids, *tickets;
    unsigned long long* status;
    Ploc* ploc;
    Bfs* bfs;
    size_t status_words;
};
size_t layout(uint32_t n, char* base, Scratch* out) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + off : nullptr;
        off += (bytes + 255) & ~size_t(255);
        return p;
    };
    Scratch s{};
    s.T.n = n;
    s.T.box = reinterpret_cast<WNode*>(take(sizeof(WNode) * 2ull * n));
    s.T.up = reinterpret_cast<int2*>(take(8ull * 2 * n));
    s.T.ch = reinterpret_cast<int2*>(take(8ull * n));
    s.T.f = reinterpret_cast<float4*>(take(32ull * n));
    s.T.choice = reinterpret_cast<uint32_t*>(take(4ull * n));
    s.T.left = reinterpret_cast<int32_t*>(take(4ull * n));
    s.first = reinterpret_cast<uint32_t*>(take(4ull * n));
    s.list0 = reinterpret_cast<int32_t*>(take(4ull * n));
    s.list1 = reinterpret_cast<int32_t*>(take(4ull * n));
    s.item = reinterpret_cast<int32_t*>(take(4ull * (2ull * n + 8)));
    s.rec_of = reinterpret_cast<uint32_t*>(take(4ull * (2ull * n + 8)));
    s.rec_kids = reinterpret_cast<uint32_t*>(take(4ull * (n + 8)));
    s.state = reinterpret_cast<State*>(take(sizeof(State)));
    if (s.state) s.root = &s.state->root, s.ploc = s.state->ploc, s.bfs = s.state->bfs;
    s.tickets = reinterpret_cast<uint32_t*>(take(4ull * (PLOC_BUNCH + BFS_BUNCH)));
    s.status_words = (2ull * n + 8 + PT - 1) / PT + 1;
    s.status = reinterpret_cast<unsigned long long*>(take(8 * s.status_words));
    if (out) *out = s;
    return off;
}

}  // namespace

size_t box_tree_scratch_bytes(uint32_t tri_count) { return layout(tri_count ? tri_count : 1, nullptr, nullptr); }

#define RSH_BT(call)                               \
    do {                                           \
        const cudaError_t e_ = (call);             \
        if (e_ != cudaSuccess) return e_;          \
    } while (0)

cudaError_t build_box_tree(ObjHierarchy& h, float pad, void* scratch, uint32_t* err, cudaStream_t s, void* host) {
    const uint32_t n = h.tri_count;
    h.wslots = 0;
    h.wroot = 0;
    if (n == 0) return cudaSuccess;
    if ((uint64_t)2 * n + 8 > (1ull << 24)) return cudaErrorInvalidValue;  // slots are 24-bit indices
    Scratch w;
    layout(n, static_cast<char*>(scratch), &w);
    w.T.cluster = h.cluster;
    auto blocks = [](uint64_t m) { return (uint32_t)((m + PT - 1) / PT); };
    uint32_t epoch = 0;
    auto clear = [&](bool all) -> cudaError_t {
        if (all) {
            epoch = 0;
            RSH_BT(cudaMemsetAsync(w.status, 0, 8 * w.status_words, s));
        }
        return cudaMemsetAsync(w.tickets, 0, 4ull * (PLOC_BUNCH + BFS_BUNCH), s);
    };
    RSH_BT(clear(true));
    RSH_BT(cudaFuncSetAttribute(k_ploc_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TailSmem)));
    // breadth-first levels; each has at most 8 times the slots of the one before it
    uint64_t most = 1;
    auto levels = [&]() {
        for (uint32_t l = 0; l < BFS_BUNCH; ++l) {
            launch_chained(true, k_bfs_level, blocks(most), PT, 0, s, w.T, w.first, w.bfs, l, w.item, w.rec_of,
                           w.rec_kids, pad, h.wboxes, w.status, w.tickets + PLOC_BUNCH + l, ++epoch, err);
            most = std::min<uint64_t>(most * 8, 2ull * n + 8);
        }
        note_launch(BFS_BUNCH);
        return cudaGetLastError();
    };
    static_assert(sizeof(State) <= BUILD_HOST_BYTES, "the state fits");
    State& st = *static_cast<State*>(host);
    auto read = [&]() -> cudaError_t {
        RSH_BT(cudaMemcpyAsync(&st, w.state, sizeof(st), cudaMemcpyDeviceToHost, s));
        return cudaStreamSynchronize(s);
    };
    // 1. PLOC passes, then the last ones in one block
    launch_chained(true, k_wide_leaves, blocks(n), PT, 0, s, h.tris, w.T, w.list0, w.ploc);
    note_launch();
    uint32_t m = n;
    for (;;) {
        // enough passes to get from m to the tail when each keeps 4/5 of its clusters (0.76 on a soup of spheres);
        // a pass too many costs its launch alone, one too few another round
        uint32_t passes = 0;
        for (uint64_t k = m; k > TAIL_CLUSTERS && passes < PLOC_BUNCH; k = k * 4 / 5) ++passes;
        for (uint32_t p = 0; p < passes; ++p)
            launch_chained(true, k_ploc_pass, blocks(m), PT_THREADS, 0, s, w.T, w.ploc, p, w.list0, w.list1, w.status,
                           w.tickets + p, ++epoch, err);
        launch_chained(true, k_ploc_tail, 1, TAIL_T, sizeof(TailSmem), s, w.T, w.ploc + passes, w.list0, w.list1,
                       w.root);
        note_launch(passes + 1);
        // 2. triangles in depth-first order, 3. the collapse, level by level: enqueued before the root is known to be
        // there (without one these kernels do nothing), for one read-back of all the build's state (a frame of 1001
        // moving objects 1.19 -> 1.16 ms)
        launch_chained(true, k_wide_tris, blocks(n), PT, 0, s, h.tris, n, w.T.up, w.root, w.first, h.wtris);
        launch_chained(true, k_bfs_init, 1, 1, 0, s, w.root, w.item, w.bfs, h.wboxes);
        note_launch(2);
        most = 1;
        RSH_BT(levels());
        RSH_BT(read());
        if (st.root >= 0) break;
        // a pass that merged nothing cannot happen (the closest pair is mutual); never loop forever
        const Ploc& end = st.ploc[passes];
        if (end.m <= TAIL_CLUSTERS || end.m >= m) return cudaErrorUnknown;
        m = end.m;
        RSH_BT(cudaMemcpyAsync(w.ploc, w.ploc + passes, sizeof(Ploc), cudaMemcpyDeviceToDevice, s));
        RSH_BT(clear(epoch + PLOC_BUNCH + BFS_BUNCH >= LB_EPOCHS));
    }
    const Bfs* lv = st.bfs;
    if (lv[1].count == 0 || lv[1].count > 8) return cudaErrorUnknown;  // the root always has children
    h.wroot = (1u << 27) | ((lv[1].count - 1u) << 24) | 1u;
    h.wnroot = REC_NODE | ((lv[1].count - 1u) << 28);
    while (lv[BFS_BUNCH].count != 0) {
        most = lv[BFS_BUNCH].count;
        RSH_BT(cudaMemcpyAsync(w.bfs, w.bfs + BFS_BUNCH, sizeof(Bfs), cudaMemcpyDeviceToDevice, s));
        RSH_BT(clear(epoch + BFS_BUNCH >= LB_EPOCHS));
        RSH_BT(levels());
        RSH_BT(read());
    }
    if (lv[BFS_BUNCH].base == 0) return cudaErrorUnknown;  // a look-back gave up
    h.wslots = lv[BFS_BUNCH].base;
    // 4. the traversal records
    const uint32_t recs = lv[BFS_BUNCH].recs;
    if (recs > h.wnode_cap) {
        cudaFree(h.wnodes);
        h.wnodes = nullptr;
        h.wnode_cap = 0;
        // an eighth more than this tree needs: a rebuild after objects moved rarely needs exactly as many
        const uint32_t cap = recs + recs / 8;
        RSH_BT(cudaMalloc(reinterpret_cast<void**>(&h.wnodes), sizeof(float4) * REC_F4 * (size_t)cap));
        h.wnode_cap = cap;
    }
    h.wnode_count = recs;
    launch_chained(true, k_rec_write, blocks(8ull * recs), PT, 0, s, h.wboxes, recs, w.rec_kids, w.rec_of, h.wnodes);
    note_launch();
    return cudaGetLastError();
}

}  // namespace rsh
