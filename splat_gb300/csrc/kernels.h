// kernels.h -- host-side launchers shared by the translation units.
#pragma once

#include <atomic>
#include <string>

#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace splat {

// Kernels launched by this thread (for launch profiling).
extern thread_local int64_t g_launches;
// Launch-shape knobs, indexed by SPLAT_TUNE_*.
extern std::atomic<int32_t> g_tune[SPLAT_TUNE_KEYS];  // process-wide launch knobs (splat_set_tuning)

// Where a hit kernel reads its rays: the structure-of-arrays bounce state
// (count on the device) or the reference's AoS ADRay array.
struct RaySrc {
    const float* f;          // SoA planes (nullptr for AoS)
    const int32_t* ignore;
    int64_t cap;
    const splat_adray_t* aos;  // AoS rays (nullptr for SoA)
    const int64_t* d_count;    // active count on the device (SoA)
    int64_t n;                 // ray count when d_count is null
    unsigned long long* fetch; // zeroed work counter: warps take rays 32 at a time (nullptr: grid-stride)
    int32_t packet;            // four-wide BVH: packet_form of the launch (0 one ray per lane)
    const int32_t* perm;       // BVH hitters: the k-th ray traced is ray perm[k] (nullptr: ray k); results
                               // go to the ray's own index
    int32_t tile_h;            // packet and brute-force kernels, no perm: rays are a light grid of tile_h rows in
                               // column-major order; warps take 8 x 4 tiles of it (0: in order)
    int32_t few;               // the count on the device may be far below the launch's bound (later bounces):
                               // four-wide BVH launches prepare for kGroupRays rays or less
};

// First-bounce rays come from a grid, and a packet of them pays where their
// paths through the tree overlap: with few rays for the triangles a packet's
// 8 x 4 patch spans many leaves and its warp walks them all in turn.
// Measured on one GB300, us a one-bounce step, one lane a ray / packets, by
// rays per triangle:
//   displaced sphere, 81,922   0.4 148/272   0.8 152/229   1.6 183/204   3.2 226/215   12.8 481/349
//   displaced sphere, 20,482   1.6 116/132   3.2 122/120   6.4 136/123   12.8 174/135
//   sponge, 96,012             0.7  68/72    1.4  84/90    2.7 112/107   10.9 270/241
constexpr float kPacketRaysPerTri = 2.5f;
// A caller's records come in their own order, at best columns of a grid: a
// packet is a strip of 32 x 1.  Measured likewise, us a frame of two bounces
// from a light, or a camera pass, lane / packets:
//   light, sphere, 81,922    0.8 281/328   1.6 355/439   3.2 507/538   6.4 719/706   12.8 1172/1112
//   light, displaced, 20,482 3.2 270/273   6.3 323/319   12.8 458/427
//   light, sponge, 96,012    1.4 296/317   2.7 473/488   5.5 756/776   10.9 1306/1313  21.8 2376/2370
//   camera, sphere, 81,922   0.7 308/430   1.8 469/602   3.3 578/656
//   camera, displaced, 20,482  2.8 261/290   7.2 397/425   13 518/515
constexpr float kStripRaysPerTri = 6.0f;
// The fused camera pass's rays come in tiles again, but from one point towards
// the whole view; a frame of two bounces, lane / packets:
//   displaced, 81,922   2.8 363/396   3.6 412/404   6.3 458/462
//   displaced, 20,482   2.8 180/186   4.3 223/219   11.2 266/260
//   sphere, 20,482      4.3 218/207   8.8 240/230
constexpr float kCameraRaysPerTri = 3.2f;
__host__ __device__ inline bool packet_density(int64_t grid_rays, int64_t n_recs,
                                               float per_tri = kPacketRaysPerTri) {
    return (float)grid_rays >= per_tri * (float)n_recs;
}

// Which traversal a warp of four-wide BVH rays takes, from
// SPLAT_TUNE_BVH_PACKET and whether the rays are on their first bounce:
// 0 one ray per lane, 1 a packet, 2 / 3 a packet when the warp's rays are
// coherent by the loose / tight thresholds of packet_coherent (hitcore.cuh).
__host__ __device__ inline int packet_form(int mode, bool first_bounce) {
    switch (mode) {
        case 1: return first_bounce ? 1 : 0;
        case 2: return 1;
        case 3: return first_bounce ? 1 : 2;
        case 4: return first_bounce ? 1 : 3;
        case 5: return 2;
        default: return 0;
    }
}

// Flattened BVH2 node (Aila & Laine 2009 layout): the boxes of both children
// and their references.  ref >= 0: inner node index; ref < 0: leaf,
// ~ref = first << 4 | (count - 1) in the BVH-ordered hit-record array.
struct __align__(16) BvhNode {
    float4 x;  // c0.lo.x, c0.hi.x, c1.lo.x, c1.hi.x
    float4 y;
    float4 z;
    int4 c;    // ref0, ref1, 0, 0
};
static_assert(sizeof(BvhNode) == 64, "BvhNode layout");

// Four-wide node collapsed from the binary tree: child i's box in
// component i of the six float4s.  Slots i >= meta.x are empty boxes
// (lo = +inf, hi = -inf), which no ray enters, so traversal needs no count.
struct __align__(16) Bvh4Node {
    float4 lox, hix, loy, hiy, loz, hiz;
    int4 c;      // child refs (as BvhNode)
    int4 meta;   // x: number of children (2..4); root: y, z, w the tree's frame (frame_of)
};
static_assert(sizeof(Bvh4Node) == 128, "Bvh4Node layout");

// The frame a scene's BVH boxes are axis-aligned in, as rows of a matrix
// applied to world positions and directions.  A linear map keeps the t of
// every ray-box intersection, so traversal rotates each ray once (slab_ray)
// and tests triangles in world space; only how tightly the boxes fit changes
// (what turning a ray rounds is in its slack there).  The frame is the vector part of a unit quaternion with
// w >= 0, kept as float bits in the four-wide root's meta.y, z, w; all zero
// is the world frame.  Host build, refit and traversal derive the matrix
// with the same binary32 operations.
struct BvhFrame {
    float r[9];
    bool world;
};
__host__ __device__ __forceinline__ BvhFrame frame_of(float x, float y, float z) {
    BvhFrame f;
    f.world = x == 0.0f && y == 0.0f && z == 0.0f;
    const float w2 = 1.0f - ((x * x + y * y) + z * z);
    const float w = sqrtf(w2 > 0.0f ? w2 : 0.0f);
    f.r[0] = 1.0f - 2.0f * (y * y + z * z);
    f.r[1] = 2.0f * (x * y - z * w);
    f.r[2] = 2.0f * (x * z + y * w);
    f.r[3] = 2.0f * (x * y + z * w);
    f.r[4] = 1.0f - 2.0f * (x * x + z * z);
    f.r[5] = 2.0f * (y * z - x * w);
    f.r[6] = 2.0f * (x * z - y * w);
    f.r[7] = 2.0f * (y * z + x * w);
    f.r[8] = 1.0f - 2.0f * (x * x + y * y);
    return f;
}
__host__ __device__ __forceinline__ void to_frame(const BvhFrame& f, float& x, float& y, float& z) {
    if (f.world) return;
    const float a = (f.r[0] * x + f.r[1] * y) + f.r[2] * z;
    const float b = (f.r[3] * x + f.r[4] * y) + f.r[5] * z;
    const float c = (f.r[6] * x + f.r[7] * y) + f.r[8] * z;
    x = a;
    y = b;
    z = c;
}
#ifdef __CUDACC__
__device__ __forceinline__ BvhFrame root_frame(const Bvh4Node* root) {
    const int4 m = __ldg(&root->meta);
    return frame_of(__int_as_float(m.y), __int_as_float(m.z), __int_as_float(m.w));
}
#endif

struct Bvh4View {
    const Bvh4Node* nodes;
    const TriHit* tris;  // BVH order (shared with the binary tree)
};

constexpr int kLeafMax = 16;
constexpr int kBvhStack = 64;

struct BvhView {
    const BvhNode* nodes;
    const TriHit* tris;  // BVH order
    const Bvh4Node* root4;  // the four-wide tree over the same leaves: its root holds the frame
};

// The padded boxes of the brute-force records in one array: one per record,
// then one per 8 and one per 32 consecutive records.
struct BruteBoxes {
    const TriBox *box, *box8, *box32;
};
__host__ __device__ inline int64_t brute_box_count(int64_t n_recs) {
    return n_recs + (n_recs + 7) / 8 + (n_recs + 31) / 32;
}
__host__ __device__ inline BruteBoxes brute_boxes_of(const TriBox* all, int64_t n_recs) {
    return {all, all + n_recs, all + n_recs + (n_recs + 7) / 8};
}

// n records as `splits` ranges of per_split (whole tiles), of at least `least`
// records each where possible; wanted of them at most, one when there is none.
struct RecordSplit {
    int64_t splits, per_split;
};
__host__ __device__ inline RecordSplit split_records(int64_t n, int64_t wanted, int64_t least, int64_t tile) {
    const int64_t most = (n + least - 1) / least;
    int64_t s = wanted < most ? wanted : most;
    s = s < 1 ? 1 : (s > 65535 ? 65535 : s);
    int64_t per = (n + s - 1) / s;
    per = (per + tile - 1) / tile * tile;
    if (per < tile) per = tile;  // no records
    s = (n + per - 1) / per;
    return {s < 1 ? 1 : s, per};
}

// brute force over prepacked hit records (reference indices 2..T in any
// order), each behind its padded box
cudaError_t launch_hit_brute(const RaySrc& rays, int64_t cap, const TriHit* recs, const TriBox* boxes, int64_t n_recs,
                             int32_t* hit_idx, float* hit_t, uint64_t* tmp, int32_t* err, int sm_count,
                             cudaStream_t s);
// the same with the results left as packed (t, index) words, which the caller
// has reset to kNoHit
cudaError_t launch_hit_brute_packed(const RaySrc& rays, int64_t cap, const TriHit* recs, const TriBox* boxes,
                                    int64_t n_recs, uint64_t* packed, int32_t* err, int sm_count, cudaStream_t s);
// brute force over the reference's n_tris array (Tuple{Int32,Tri})
cudaError_t launch_hit_brute_ntris(const splat_adray_t* rays, int64_t n_rays, const splat_ntri_t* ntris,
                                   int64_t n_tris, uint64_t* tmp, int32_t* hit_idx, int sm_count, cudaStream_t s);
// splat_next_hit_brute_static: the same hitter with its scratch in a
// file-scope device array (no allocation); n_rays <= kStaticHitMaxRays
constexpr int64_t kStaticHitMaxRays = SPLAT_STATIC_HIT_MAX_RAYS;
cudaError_t launch_hit_brute_ntris_static(const splat_adray_t* rays, int64_t n_rays, const splat_ntri_t* ntris,
                                          int64_t n_tris, int32_t* hit_idx, int sm_count, cudaStream_t s);
cudaError_t launch_hit_bvh(const RaySrc& rays, int64_t cap, const BvhView& bvh, int32_t* hit_idx, float* hit_t,
                           int32_t* err, int sm_count, cudaStream_t s);
cudaError_t launch_hit_bvh4(const RaySrc& rays, int64_t cap, const Bvh4View& bvh, int32_t* hit_idx, float* hit_t,
                            int32_t* err, int sm_count, cudaStream_t s);
// traversal work counted while SPLAT_TUNE_COUNT_WORK is set (nodes, triangle
// pre-tests, full triangle tests, rays); synchronises s; reset clears them
cudaError_t read_hit_work(uint64_t out[4], bool reset, cudaStream_t s);
// grid of a work-counter traversal launch (one resident wave)
int resident_grid(const void* kernel, int64_t cap, int sm_count, int threads, int max_per_sm);
// one-launch bottom-up refit of the two-child and the four-wide tree.  links:
// parent per node, then number of inner children per node; flags: n2 + n4
// arrival counts.  The boxes are taken in the frame of the four-wide root.
struct RefitTrees {
    BvhNode* nodes2;
    Bvh4Node* nodes4;
    int64_t n2, n4;
    const int32_t *links2, *links4;
    unsigned* flags;
};
cudaError_t launch_refit_trees(const RefitTrees& t, const TriHit* recs, const splat_ftri_t* ftri,
                               const unsigned* scale, float pad_rel, cudaStream_t s);

// GPU BVH rebuild (lbvh.cu): linear BVH over Morton-sorted centroids, written
// as two-child and four-wide nodes with leaves of at most leaf_max triangles
constexpr int kLbvhLeaf = 4;
size_t lbvh_scratch_bytes(int64_t n_prims);
// The nodes (each in an array of at least n_tris - 2 of them, at its radix-tree
// index), with the records, boxes, order and scale launch_pack_hits would write.
struct LbvhOut {
    BvhNode* nodes2;
    Bvh4Node* nodes4;
    int32_t* order;
    TriHit* recs;
    TriBox* boxes;
    int32_t* bvh_pos;
    unsigned* scale;
};
cudaError_t launch_lbvh_build(const splat_ftri_t* ftri, int64_t n_tris, int leaf_max, void* scratch,
                              const LbvhOut& out, int sm_count, cudaStream_t s);

// Coherent ray order (lbvh.cu): a permutation of the d_count active rays of
// a SoA bounce buffer, grouped by (direction octant, BVH-order position of
// the triangle the ray leaves) with a counting sort over a key of key_bits
// (4..22) bits (the position's low bits dropped to fit).  Rays that leave
// neighbouring triangles in similar directions then share warps, so the
// traversal's lanes take similar paths.  bvh_pos[i]: BVH record position of
// reference index i (0 for indices outside 1..n_tris).  *perm_out points
// into scratch.
size_t ray_order_bytes(int64_t cap);
cudaError_t launch_ray_order(const float* soa_f, const int32_t* ignore, int64_t cap, const int64_t* d_count,
                             const int32_t* bvh_pos, int64_t n_tris, int key_bits, void* scratch,
                             const int32_t** perm_out, int sm_count, cudaStream_t s);

// The bucket offsets of that counting sort for keys counted elsewhere: cnt
// holds each bucket's size (buckets entries) and is scanned in place into
// offsets (sums: order_sums_count(buckets) words of scratch).
size_t order_sums_count(int64_t buckets);
cudaError_t launch_order_scan(uint32_t* cnt, int64_t buckets, uint32_t* sums, cudaStream_t s);

// scene packing / refit.  scale: device word holding max |vertex coordinate|
// (float bits), from which every padded box takes pad_abs = 1e-4 max(1, scale).
// order: reference index of each record; bvh_pos (optional, n_tris + 1
// entries): its inverse.
cudaError_t launch_pack_hits(const splat_ftri_t* ftri, int64_t n_tris, TriHit* recs, TriBox* boxes, unsigned* scale,
                             const int32_t* order, int32_t* bvh_pos, cudaStream_t s);


// generation and conversion
struct GenParams {
    splat_rect_light_t light;
    int64_t upscale;
    splat_lambda_mode_t lm;
    uint64_t seed;
    uint32_t light_index;
    int64_t ray_begin;
};
// clears the step's n_counts counters (counts[0] = n) and, when given, the
// packed hits of the first bounce
cudaError_t launch_generate_soa(const GenParams& g, int64_t n, RaySoA out, int64_t* counts, int n_counts,
                                uint64_t* packed, cudaStream_t s);
cudaError_t launch_generate_aos(const GenParams& g, int64_t n, splat_adray_t* out, cudaStream_t s);
// active rays to out (their number added to d_count), the others to idle
// (d_idle); ids are the rays' slots
cudaError_t launch_aos_to_soa(const splat_adray_t* in, int64_t n, RaySoA out, int64_t* d_count, RaySoA idle,
                              int64_t* d_idle, cudaStream_t s);
// *d_total = *d_count + *d_idle, with the idle rays' hit state (position,
// direction, ignored triangle, id) appended to rays [0, *d_count)
cudaError_t launch_append_idle(RaySoA rays, const int64_t* d_count, RaySoA idle, const int64_t* d_idle,
                               int64_t* d_total, int sm_count, cudaStream_t s);
// rays [0, *d_count) back to their records, and the hits of [0, *d_total) to
// their slots
cudaError_t launch_soa_to_aos(RaySoA in, const int64_t* d_count, const int64_t* d_total, const int32_t* hit,
                              splat_adray_t* out, int32_t* hit_out, int status, cudaStream_t s);

// evolve (+ compaction, + fused splat in trace mode)
struct SplatParams {
    void* map;
    int32_t accum;  // SPLAT_ACCUM_*
    float scale;    // 2^frac_bits
    int64_t w, h;
    int32_t n_lambda;  // 0: own wavelength
    int32_t n_delta;
    float spectrum[SPLAT_MAX_LAMBDA];
    float deltas[16];
};

struct EvolveArgs {
    RaySoA in, out;
    const int64_t* in_count;
    int64_t* out_count;
    const int32_t* hit_idx;
    const splat_ftri_t* tris;
    int64_t n_tris;         // hit indices outside 1..n_tris are reported and treated as misses
    int32_t* err;           // error word (bit 4: bad hit index)
    int64_t first_diffuse;
    splat_material_t material;
    uint64_t seed;
    uint32_t bounce;
    float force_rand;
    int32_t quirks;
    int32_t last;           // trace mode: last bounce, no optics
    splat_adray_t* aos;     // plugin mode: retired rays written back here
    int32_t* aos_hit;       // plugin mode: and the hit they retired with, by slot
    RaySoA splat_q;         // trace mode: final-evolved diffuse rays (ignore = hit triangle)
    int64_t* splat_count;
    const uint64_t* hit_packed;  // trace mode: hits as packed (t, index) words instead of hit_idx
    uint64_t* next_packed;       // trace mode: the survivors' words for the next bounce, reset here
    RaySoA sky_q;           // camera mode: rays that escaped, unchanged
    int64_t* sky_count;
    int32_t tile_h;         // > 0: the input is a light grid of tile_h rows in column order, taken in its
                            // 8 x 4 tiles (grid_tile_ray), so the survivors leave in tile order
};
cudaError_t launch_evolve_trace(const EvolveArgs& a, int64_t cap, int sm_count, cudaStream_t s);
// trace mode plus the escaped rays queued for the skydome (camera pass)
cudaError_t launch_evolve_camera(const EvolveArgs& a, int64_t cap, int sm_count, cudaStream_t s);
cudaError_t launch_evolve_plugin(const EvolveArgs& a, int64_t cap, int sm_count, cudaStream_t s);
// one evolve_ray broadcast on AoS rays (rndm: per-ray draws or null)
cudaError_t launch_evolve_aos(splat_adray_t* rays, int64_t n, const int32_t* hit_idx, const float* rndm,
                              const EvolveArgs& a, int sm_count, cudaStream_t s);
// partition!: ACTIVE rays first, in place; scratch: counts (3 int64), list (2 n int64)
cudaError_t launch_partition(splat_adray_t* rays, int64_t n, int64_t* counts, int64_t* list, int64_t* d_n_active,
                             int sm_count, cudaStream_t s);
cudaError_t launch_light_map(splat_adray_t* rays, int64_t n, const int32_t* hit_idx, const splat_ftri_t* tris,
                             int64_t n_tris, int32_t* err, const SplatParams& sp, int sm_count, cudaStream_t s);
// camera pass (shade.cu)
struct CameraParams {
    splat_camera_t cam;
    int64_t h, w;      // camera grid (image / upscale)
    uint64_t seed;
    float lambda;
    // of the whole grid: scale = h cos45 / fov_half_sin, p = 1 / scale, and the
    // products p right, p up and dir in double
    double scale, p, pr[3], pu[3], d[3];
};
struct ShadeParams {
    cudaTextureObject_t map_tex, sky_tex;
    int64_t map_w, map_h, sky_w, sky_h;
    int32_t has_sky;
    int32_t n_lambda;
    int32_t nd;          // upscale: nd x nd sub-samples (pixels) per camera ray
    int64_t cam_h;       // camera grid rows
    int64_t height;      // image rows
    float* rgb;          // image, column-major RGB float triples
    float deltas[16];    // upres(nd)
    float spectrum[SPLAT_MAX_LAMBDA];
    float retina[3][SPLAT_MAX_LAMBDA];
};
cudaError_t launch_camera_soa(const CameraParams& c, int64_t n, RaySoA out, int64_t* count, cudaStream_t s);
cudaError_t launch_camera_aos(const CameraParams& c, int64_t n, splat_adray_t* out, cudaStream_t s);
cudaError_t launch_shade_diffuse(const RaySoA& q, const int64_t* count, const splat_ftri_t* tris,
                                 const ShadeParams& p, int64_t cap, int sm_count, cudaStream_t s);
cudaError_t launch_shade_sky(const RaySoA& q, const int64_t* count, const ShadeParams& p, int64_t cap, int sm_count,
                             cudaStream_t s);
cudaError_t launch_shade_aos(splat_adray_t* rays, int64_t n, const int32_t* hit_idx, const splat_ftri_t* tris,
                             int64_t n_tris, int32_t* err, const ShadeParams& p, int sm_count, cudaStream_t s);
cudaError_t launch_image_accumulate(float* out, const float* rgb, int64_t n, int32_t k, int sm_count,
                                    cudaStream_t s);
cudaError_t launch_map_to_array(const int32_t* map, int64_t w, int64_t h, int64_t planes, float inv_scale,
                                cudaSurfaceObject_t surf, cudaStream_t s);

// A whole trace step of at most kSmallStepRays rays in one launch (step.cu):
// nodes4 null is the brute-force hitter; ea gives scene, material and draws
// (its queues are unused).  stats accumulate, as the last splat leaves them.
constexpr int64_t kSmallStepRays = 12288;
// by brute force: of at most kSmallStepBruteRecs records, above
// kSmallStepBruteRays rays of kSmallStepFewRecs
constexpr int64_t kSmallStepBruteRays = 8192, kSmallStepBruteRecs = 1024, kSmallStepFewRecs = 128;
cudaError_t launch_small_step(const GenParams& gen, int64_t n, const Bvh4Node* nodes4, const TriHit* recs,
                              const TriBox* boxes, int64_t n_recs, const EvolveArgs& ea, int32_t depth,
                              const SplatParams& sp, splat_trace_stats_t* stats, cudaStream_t s);

// light-map splat of the queued diffuse rays [*begin, *end) (begin null: from
// 0).  The step's last splat also adds up its statistics: rays[b], the rays
// entering bounce b + 1, for depth bounces, *end the diffuse rays, and the
// scene's error word.
struct SplatRange {
    const int64_t *begin, *end;
    const int64_t* rays;  // null: not the last
    int depth;
    const int32_t* err;
};
cudaError_t launch_splat(const RaySoA& q, const SplatRange& rg, const splat_ftri_t* tris, const SplatParams& sp,
                         splat_trace_stats_t* stats, int sm_count, cudaStream_t s);
// *dst = *src in stream order (a queue-length snapshot)
cudaError_t launch_copy_count(const int64_t* src, int64_t* dst, cudaStream_t s);
cudaError_t launch_unpack_hits(const uint64_t* tmp, int64_t n, const int64_t* d_count, int32_t* hit_idx,
                               float* hit_t, cudaStream_t s);

// ---------------------------------------------------------------------------
// batch engine (batch.cu)
// ---------------------------------------------------------------------------
struct BatchSceneRef {
    const splat_ftri_t* ftri;
    const TriHit* brute;
    const TriBox* brute_boxes;
    const Bvh4Node* nodes4;
    const TriHit* bvh_tris;
    int64_t n_recs, n_tris, first_diffuse;
    const int32_t* bvh_pos;  // BVH record position of each reference index (nullptr: none)
};

// Ray order of the batch engine: bucket keys over every item of the table,
// (item's key base + BVH position of the triangle left >> pos_shift) x 8 +
// direction octant, at most 2^kBatchOrderBits buckets.
constexpr int kBatchOrderBits = 24;

struct BatchTickArgs {
    void* items;  // device item table
    int n_slots;
    int tick;
    void* fresh;  // device FreshList
    RaySoA cur, next, queue;
    int64_t* cur_count;
    int64_t* next_count;
    int64_t* queue_count;
    int64_t fresh_rays;  // rays generated this tick (known on the host)
    int64_t cap_rays;    // bound on the rays active this tick
    int32_t* hit_idx;
    int32_t* err;
    int sm_count;
    bool any_brute;      // some item in flight uses the brute-force hitter (or has no BVH)
    int material_kind;   // material kind shared by every item in flight, -1 when mixed
    unsigned long long* fetch;  // zeroed work counter of this tick's hit kernel
    // ray order before the hit kernel (order_buckets > 0): keys and perm of
    // cap_rays entries, bucket counts (order_buckets) and their scan's sums
    int64_t order_buckets;
    uint32_t* order_keys;
    uint32_t* order_cnt;
    uint32_t* order_sums;
    int32_t* order_perm;
};

cudaError_t launch_batch_tick(const BatchTickArgs& a, cudaStream_t s);

// A whole pass (ticks t0 .. t0 + n_ticks - 1 of items that all start at t0)
// as one persistent cooperative launch over 1/share of the GPU's resident
// blocks; every counter below is zeroed by the caller before the launch.
constexpr int kMaxPassTicks = 8;
struct BatchPassArgs {
    void* items;
    void* fresh;
    int n_slots, t0, n_ticks;
    int material_kind;   // shared by every item, -1 when mixed
    RaySoA a, b, queue;  // a: the first tick's rays
    int64_t* count;      // count[i]: rays entering tick t0 + i (n_ticks + 1 slots)
    int64_t* qcount;     // queue entries so far
    int64_t* qmark;      // qmark[i]: queue length before tick i's evolve (n_ticks slots)
    unsigned long long* fetch;        // per-tick traversal work counters (n_ticks)
    unsigned long long* splat_fetch;  // per-tick splat work counters (n_ticks)
    unsigned* bar;       // grid-wait arrivals
    int32_t* hit_idx;
    int32_t* err;
    int packet_mode;     // SPLAT_TUNE_BVH_PACKET when the pass was launched
};
cudaError_t launch_batch_pass(const BatchPassArgs& a, int share, int sm_count, cudaStream_t s);
// the two halves of a tick: reserve, generate, hit, evolve; and the splat of the tick's queue
cudaError_t launch_batch_trace(const BatchTickArgs& a, cudaStream_t s);
cudaError_t launch_batch_splat(const BatchTickArgs& a, cudaStream_t s);
// sets splat_last_error() of the calling thread and returns code (api.cu)
splat_status_t set_error(splat_status_t code, const std::string& msg);
size_t batch_item_bytes();
size_t batch_fresh_bytes();
void batch_fill_item(void* dst, const BatchSceneRef& sc, const GenParams& gen, int64_t n_rays, int32_t depth,
                     int32_t hitter, int32_t start_tick, int32_t quirks, float force_rand,
                     const splat_material_t& material, const SplatParams& sp);
void batch_clear_item(void* dst);
// Assigns every used item of a host item table its ray-order key base (items
// in slot order, each (n_tris >> shift) + 1 positions, one shift for all,
// the smallest that fits 8 x positions in 2^max_bits buckets); returns the
// number of buckets.
int64_t batch_assign_order_keys(void* items, const uint8_t* used, int32_t n_slots, int max_bits);
void batch_set_seed(void* dst, uint64_t seed);

}  // namespace splat
