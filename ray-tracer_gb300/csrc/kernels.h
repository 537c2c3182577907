// Host-side launchers of the sm_103a kernels (one translation unit per stage). Internal to the library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/rsh.h"

// Device error word bits (bounded waits that gave up, buffer overflows).
#ifndef RSH_DEVERR_TIMEOUT
#define RSH_DEVERR_TIMEOUT 1u
#define RSH_DEVERR_OVERFLOW 2u
#endif

namespace rsh {

// Counts this library's kernel launches (rsh_kernel_launches).
void note_launch(unsigned n = 1);

// A kernel that may start while the one before it in the stream still runs; it waits itself
// (griddepcontrol.wait) before it touches what that one wrote. (The second of a pair of traversals reads nothing of
// the first's and waits at its end; what the first waited for, too, it gets through FusedArgs::ready.)
template <class... P, class... A>
inline cudaError_t launch_chained(bool chained, void (*kernel)(P...), uint32_t grid, uint32_t threads, size_t smem,
                           cudaStream_t s, A... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

struct HashP {
    float lo[3];
    float scale[3];
    uint32_t grid_bits, dir_log2, tag_bits, key_bits;
};
inline HashP to_hashp(const rsh_hash_params& h) {
    HashP p;
    for (int i = 0; i < 3; ++i) {
        p.lo[i] = h.lo[i];
        p.scale[i] = h.scale[i];
    }
    p.grid_bits = h.grid_bits;
    p.dir_log2 = h.dir_log2;
    p.tag_bits = h.tag_bits;
    p.key_bits = h.key_bits;
    return p;
}

struct LightsP {
    uint32_t count;
    uint32_t samples;  // shadow rays per light: 1, or 16 (soft shadows)
    float pos[8][3];
};

struct CameraP {
    float eye[3], dir[3], right[3], up[3];
};

// ---- raygen + hash (raygen.cu)
// Two ranges of words: zeroed, or copied from the first to the second.
struct Words2 {
    uint32_t *p[2], *to[2];
    uint32_t n[2];
};
// zero: words set to 0 beside it (a frame's counters: no memset of their own)
cudaError_t launch_raygen_primary(const CameraP& cam, uint32_t w, uint32_t h, rsh_ray* rays,
                                  uint32_t* pixel_of_ray, cudaStream_t s, const Words2& zero = Words2());
// What ray generation writes beside the rays for a batched call whose rays use packets: its keys (tag | (ray hash >>
// drop) or RSH_KEY_NONE), with the segment's results prefilled (flags 0 for an any-hit segment, hits RSH_HIT_NONE
// otherwise) and its ray count added to *count (one atomic per block).
struct RayOut {
    uint32_t* keys = nullptr;      // the batch's key array at the segment's first slot
    uint32_t tag = 0;
    uint32_t drop = 0;
    HashP hp{};                    // the segment scene's hash (tag 0)
    uint32_t* count = nullptr;     // null: the caller keys or counts the rays itself
    uint32_t* flags = nullptr;
    unsigned long long* hits = nullptr;
};
cudaError_t launch_raygen_shadow(const float4* spos, const float4* snrm, uint32_t w, uint32_t h,
                                 const LightsP& lights, float eps, const HashP& hp, rsh_ray* rays,
                                 uint32_t* keys, cudaStream_t s, const RayOut& out = RayOut());
cudaError_t launch_raygen_reflect(const float4* spos, const float4* snrm, const rsh_ray* prev,
                                  const float eye[3], uint32_t w, uint32_t h, float eps,
                                  float jitter, uint32_t seed, uint32_t bounce, const HashP& hp,
                                  rsh_ray* rays, uint32_t* keys, cudaStream_t s,
                                  const RayOut& out = RayOut());
cudaError_t launch_raygen_refract(const float4* spos, const float4* snrm, const rsh_ray* prev, const float eye[3],
                                  uint32_t w, uint32_t h, float eps, float eta, const HashP& hp, rsh_ray* rays,
                                  uint32_t* keys, cudaStream_t s);
cudaError_t launch_hash(const rsh_ray* rays, uint32_t n, const HashP& hp, uint32_t tag,
                        uint32_t* keys, cudaStream_t s);

// ---- trim + compress (compress.cu)
size_t compress_scratch_bytes(uint32_t n_slots);
cudaError_t launch_compress(const uint32_t* keys, uint32_t n_slots, uint32_t* trimmed_ids,
                            uint32_t* chunk_keys, uint32_t* chunk_bases, uint32_t* counts,
                            void* scratch, uint32_t* err, cudaStream_t s);
cudaError_t launch_chunk_sizes(const uint32_t* chunk_bases, const uint32_t* counts, uint32_t max_chunks,
                               uint32_t* chunk_sizes, cudaStream_t s);

// ---- onesweep radix sort (sort.cu)
size_t sort_scratch_bytes(uint32_t n_max, uint32_t key_bits);
size_t sort_selftest_scratch_bytes();
cudaError_t sort_selftest_timeout(void* scratch, uint32_t* err, uint32_t spin_limit, cudaStream_t s);
cudaError_t launch_sort_pairs(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                              uint32_t* vals_out, uint32_t n_max, const uint32_t* d_count,
                              uint32_t key_bits, void* scratch, uint32_t* err, cudaStream_t s,
                              bool keys_wanted = true);  // false: keys_out is used but does not receive the sorted keys

// ---- decompress (decompress.cu)
size_t decompress_scratch_bytes(uint32_t max_chunks);
// Batched layout target of decompression: ray k of the sorted order (segment tag = key >> tag_shift)
// is written to padded[k + seg_delta[tag]] instead of sorted_ids[k].
struct PaddedOut {
    const uint32_t* seg_delta;
    uint32_t tag_shift;
    uint32_t max_padded;
    uint32_t* padded;
};
cudaError_t launch_decompress(const uint32_t* sorted_chunk_keys, const uint32_t* sorted_chunk_vals,
                              const uint32_t* chunk_bases, const uint32_t* trimmed_ids,
                              const uint32_t* counts, uint32_t max_rays, uint32_t* sorted_keys,
                              uint32_t* sorted_ids, void* scratch, uint32_t* err, cudaStream_t s,
                              const PaddedOut* padded_out = nullptr);

// ---- ray-space hierarchy build (build.cu)
uint32_t hierarchy_capacity(uint32_t max_rays, uint32_t packet, uint32_t offsets[4]);
cudaError_t launch_build_rsh(const rsh_ray* rays, const uint32_t* sorted_ids, uint32_t max_rays,
                             const uint32_t* d_count, uint32_t packet, rsh_node* nodes,
                             cudaStream_t s);

// ---- object-sphere hierarchy (objh.cu)
struct ObjHierarchy {
    uint32_t tri_count = 0;
    uint32_t cluster = 8;
    uint32_t levels = 0;           // level 0 = clusters; levels-1 = top (<= 8 nodes)
    uint32_t level_off[16] = {};   // offsets into spheres
    uint32_t level_size[16] = {};
    float4* spheres = nullptr;     // all levels
    uint32_t* kids = nullptr;      // per level l (at level_off[l] + l): level_size[l] + 1 child-range starts
    float4* tris = nullptr;        // cluster order, 3 per triangle, v0.w = original id bits
    uint32_t* order = nullptr;     // cluster slot -> original triangle id
    float4* boxes = nullptr;       // per node, all levels like spheres: padded box lo, hi; lo.w / hi.w: child link
    // the single-ray box tree (wide.cu): 8-wide, mixed depth, 2 float4 per slot; triangles in its own
    // depth-first order (v0.w = original id bits); wroot = the root's stack entry
    float4* wboxes = nullptr;
    float4* wtris = nullptr;
    uint32_t wroot = 0;
    uint32_t wslots = 0;
    // the same tree as traversal records (14 float4 per node: child boxes plane by plane, child entries)
    float4* wnodes = nullptr;
    uint32_t wnode_count = 0;
    uint32_t wnode_cap = 0;        // records allocated
    uint32_t wnroot = 0;           // the root's entry in record form
};
// A traversal record of the box tree: REC_F4 float4 (the eight children's box planes lo x, hi x, lo y, hi y,
// lo z, hi z, 8 floats each, then their eight stack entries); a node's entry is REC_NODE | (children - 1)
// << 28 | record index, a cluster's its first triangle | (triangles - 1) << 23.
constexpr uint32_t REC_F4 = 14;
constexpr uint32_t REC_NODE = 0x80000000u;
// Builds the single-ray box tree from h.tris (Morton order) and h.cluster; boxes widened by `pad`. The scratch
// is the caller's (box_tree_scratch_bytes). Synchronises the stream.
size_t box_tree_scratch_bytes(uint32_t tri_count);
constexpr size_t BUILD_HOST_BYTES = 2048;
cudaError_t build_box_tree(ObjHierarchy& h, float pad, void* scratch, uint32_t* err, cudaStream_t s, void* host);
// Builds (or, for the same triangle count, rebuilds in place) the object hierarchy and the box tree; scratch of
// objh_scratch_bytes; host: BUILD_HOST_BYTES of pinned memory. The levels are built on `side`, a stream of the caller's that nothing else waits for.
// Synchronises both streams.
cudaError_t build_object_hierarchy(const float4* positions_dev, uint32_t tri_count, uint32_t cluster,
                                   const float lo[3], const float hi[3], ObjHierarchy& h,
                                   void* scratch, uint32_t* err, cudaStream_t s, cudaStream_t side, void* host);
size_t objh_scratch_bytes(uint32_t tri_count);
void free_object_hierarchy(ObjHierarchy& h);
size_t object_hierarchy_bytes(const ObjHierarchy& h);  // what its arrays take

// ---- traversal (traverse.cu)
struct TravArgs {
    const rsh_node* nodes;
    uint32_t node_off[4];       // level offsets of the ray hierarchy (from max_rays)
    uint32_t max_rays;
    const uint32_t* d_count;
    uint32_t packet;
    const float4* spheres;
    const uint32_t* kids;        // object-tree child ranges (level l at lvl_off[l] + l)
    uint32_t lvl_off[16];
    uint32_t lvl_size[16];
    uint32_t levels;
    unsigned long long* cand;
    unsigned long long capacity;
    unsigned long long* cand_count;
    uint32_t* work;              // [0] = next unit, [1] = resume unit (min failed)
    uint32_t unit_end;           // units >= unit_end are left for a later pass
    unsigned long long* node_tests;
    uint32_t* err;
};
cudaError_t launch_traverse(const TravArgs& a, cudaStream_t s);

// ---- intersection (intersect.cu)
struct IsectArgs {
    const float4* spheres;       // cluster spheres (object-hierarchy level 0)
    const uint32_t* kids;        // level 0 child ranges: cluster c holds triangles [kids[c], kids[c + 1])
    const float4* tris;
    uint32_t tri_count;
    uint32_t cluster;
    const rsh_ray* rays;
    const uint32_t* sorted_ids;
    uint32_t max_rays;
    const uint32_t* d_count;
    uint32_t packet;
    const unsigned long long* cand;
    const unsigned long long* cand_count;
    unsigned long long capacity;
    uint32_t* flags;
    unsigned long long* hits;
    unsigned long long* tri_tests;
};
cudaError_t launch_intersect(const IsectArgs& a, bool any_hit, cudaStream_t s);

// ---- fused persistent traversal + intersection (fused.cu)
struct FusedSeg {
    const float4* spheres;
    const uint32_t* kids;          // object-tree child ranges (level l at lvl_off[l] + l)
    const float4* tris;
    const float4* boxes;           // per node (like spheres): padded box lo, hi; lo.w / hi.w: child link
    const float4* wboxes;          // the single-ray box tree (wide.cu): slots (cluster boxes), triangles,
    const float4* wtris;           // traversal records and the root's record entry
    const float4* wnodes;
    uint32_t wnroot;
    uint32_t tri_count;
    uint32_t cluster;
    uint32_t levels;
    uint32_t lvl_off[16];
    uint32_t lvl_size[16];
    uint32_t unit_begin;           // first work unit of this segment
    uint32_t any_hit;
    uint32_t ray_level;            // object-tree level at and below which rays descend individually
    const rsh_ray* rays;           // the segment's own rays (slot - slot_base); read in place by the rays-only kernel
    uint32_t* flags;               // indexed by slot - slot_base
    unsigned long long* hits;
    uint32_t slot_base;            // subtracted from an id: ids of a sorted batch count over all segments
    // the rays-only kernel: the segment's ray slots in the order they are traced, n of them (null: every slot
    // 0 .. n - 1, and the kernel also writes the result of a slot without a ray)
    const uint32_t* ids;
    uint32_t n;
    uint32_t slots;                // the segment's ray slots: an id outside them is skipped
    const uint32_t* count;         // device count of ids (null: n); at most n
};
struct FusedArgs {
    const rsh_node* nodes;
    uint32_t node_off[4];
    uint32_t packet;
    uint32_t ray_level;            // packet kernel: the segments' highest switch level
    const rsh_ray* rays;
    const uint32_t* sorted_ids;    // packet kernel
    const FusedSeg* segs;          // device; rays-only: count already folded into n
    uint32_t nseg;
    uint32_t units_max;
    const uint32_t* d_units;       // device count of units
    uint32_t* work;
    uint32_t blocks_per_sm;        // CTAs per SM of the launch (0: as many as fit)
    uint32_t share_tail;           // rays-only kernel: a drained warp shares its last rays among its lanes
    unsigned long long* node_tests;
    unsigned long long* tri_tests;
    uint32_t* err;
    uint32_t warps;                    // set by the launch: warps that the GPU holds
    bool pixel_order;                  // rays of neighbouring pixels lie together
    uint32_t pair;                     // rays-only: 1, 2: the first / second of two launches that neither read
                                       // nor write what the other writes; the second may start while the first runs
    uint32_t wait;                     // rays-only: the launch is chained behind a kernel whose results it reads
    // a pair whose first launch waits for results that the second reads, too: the word by which the first passes them
    // on, and the value that says so (null: what both read was complete before the first started)
    uint32_t* ready;
    uint32_t ready_is;
    FusedSeg one;                      // launch_rays_one: the one segment (slot_base 0)
    uint32_t* valid;                   // rays-only: the rays traced are added to valid[0] and valid[1] (null: not)
    unsigned long long* cand_pairs;    // launch_rays_one: counts (ray, cluster) pairs tested (null: not counted)
};
cudaError_t launch_fused(const FusedArgs& a, cudaStream_t s);
// Rays alone from the root: the segments of the table, all of one kind / one segment, from the arguments.
cudaError_t launch_rays_segs(const FusedArgs& a, bool any_hit, cudaStream_t s);
cudaError_t launch_rays_one(const FusedArgs& a, cudaStream_t s);
// rays per work unit of the rays-only kernel (a multiple of 64, at most 256: job words hold 8 bits)
#ifndef RSH_RAYS_UNIT
#define RSH_RAYS_UNIT 64
#endif

// ---- resolve + shade (shade.cu)
cudaError_t launch_resolve(const float4* tris_orig_pos, const float4* tris_orig_nrm,
                           const uint32_t* mat_ids, const rsh_ray* rays, const unsigned long long* hits,
                           const uint32_t* pixel_of_ray, uint32_t n, float4* spos, float4* snrm,
                           cudaStream_t s);
struct ShadeArgs {
    const float4* spos;
    const float4* snrm;
    const rsh_material* materials;
    uint32_t material_count;
    const uint32_t* shadow;   // W*H*L*samples slots
    float4* accum;            // W*H rgb accumulators + weight in w
    uint32_t w, h;
    uint32_t lights;
    uint32_t samples;         // shadow samples per light (1, or 16 for soft shadows)
    rsh_light light[8];
    float eye[3];
    uint32_t bounce;
    const rsh_ray* incident;  // reflection rays that produced the surface (bounce>0), else null
};
cudaError_t launch_shade(const ShadeArgs& a, cudaStream_t s);
cudaError_t launch_pack_rgba(const float4* accum, uint32_t n, uint32_t* rgba, cudaStream_t s);

// ---- a frame's work between two traversals (bounce.cu)
struct BounceArgs {
    uint32_t w, h;
    const float4 *pos, *nrm;          // the scene's triangles, normals and material ids (original order)
    const uint32_t* mat;
    const rsh_ray* rays;              // the traced rays whose hits are the next surface: the primary rays (tile
    const unsigned long long* hits;   // order: tiles_x x tiles_y tiles) or reflection rays by pixel (tiles_x 0)
    uint32_t tiles_x, tiles_y;
    float4 *spos, *snrm;              // that surface (written; null: not)
    // its rays (ray generation)
    LightsP lights;
    float eps, jitter;
    uint32_t seed, bounce;
    float eye[3];
    rsh_ray *srays, *rrays;
    uint32_t *sflags, *sids, *scount, *rids, *rcount;
    unsigned long long* rhits;
    // shading of the surface before it (ShadeArgs: its surface, flags, bounce and incident rays), the image
    ShadeArgs sh;
    uint32_t* rgba;
    Words2 counters;                  // without gen: words copied to (pinned host) memory, the frame's counters
};
// shade: shade sh's surface first; gen: write the next surface's rays and lists, their results prefilled;
// final_image (without gen): shade the next surface too, unshadowed, and pack the image.
cudaError_t launch_bounce(const BounceArgs& a, bool shade, bool gen, bool final_image, cudaStream_t s);

// ---- object transforms and bounds (transform.cu)
cudaError_t launch_transform(const float4* pos_rest, const float4* nrm_rest, const uint32_t* obj, uint32_t tri_count,
                             uint32_t n_objects, const float* model, const float* normal, float4* pos, float4* nrm,
                             cudaStream_t s);
size_t bounds_scratch_bytes();
cudaError_t launch_bounds(const float4* pos, uint32_t tri_count, void* scratch, float* out6, cudaStream_t s);

// ---- misc (util kernels in raygen.cu)
cudaError_t launch_fill_u64(unsigned long long* p, unsigned long long v, size_t n, cudaStream_t s);

}  // namespace rsh
