// hit.cu -- nearest-hit kernels.
//
// Semantics (src/hitters.jl:24-30, src/tracer.jl:45-59): for every ray, the
// lexicographic minimum of (t, index) over the triangles with
// in_triangle(o + d t) && t > 0 && index != ignore_tri; (Inf, 1) when none.
// All kernels evaluate the reference's test with the same binary32
// operations, so t and the index are bit-identical to the CPU restatement.
//
// * hit_brute_kernel: all records, behind merged boxes over 32 and 8 of them.
//   The tiles that some ray of the block enters are staged through shared
//   memory by TMA bulk copies (cp.async.bulk + mbarrier, two-stage ring, no
//   multicast); each thread keeps a ray in registers and its running argmin.
//   Record ranges split over blockIdx.y merge with a packed 64-bit atomicMin
//   (src/atomic_argmin.jl).
// * hit_ntris_kernel: the same rule over the reference's n_tris array, with a
//   block's tile of records sorted and boxed on the fly; of few records
//   (hit_ntris_direct_kernel) without boxes.
// * hit_bvh_kernel: one thread per ray walks the flattened BVH2 with a short
//   per-thread stack; boxes are padded, and widened by the ray's slack, so
//   every triangle whose test can succeed is visited, and the same
//   lexicographic rule makes the result identical to brute force.
#include <algorithm>
#include <cstdio>
#include <mutex>
#include <unordered_map>

#include "hitcore.cuh"

namespace splat {

thread_local int64_t g_launches = 0;
std::atomic<int32_t> g_tune[SPLAT_TUNE_KEYS] = {4, 16, 8, 8, 0, 1, 2, 0, 2, 0, 0, 64, 0, 0};

// ---------------------------------------------------------------------------
// PTX helpers: mbarrier + bulk copy (sm_90+ async proxy)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after kWaitLimit polls (each poll may suspend the
// thread for a hardware-chosen time), so a lost copy cannot hang the GPU.
constexpr uint32_t kWaitLimit = 1u << 24;
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t phase, uint32_t limit = kWaitLimit) {
    for (uint32_t it = 0; it < limit; ++it)
        if (mbar_try_wait(bar, phase)) return true;
    return false;
}
// Polls of the stalled wait that SPLAT_TUNE_TEST_WAIT_STALL injects.
constexpr uint32_t kStallPolls = 64;

// ---------------------------------------------------------------------------
// brute force, TMA-staged tiles
// ---------------------------------------------------------------------------
constexpr int kBruteThreads = 256;  // the n_tris drop-in kernel
constexpr int kTile = 256;  // records per tile of the n_tris drop-in kernel
// Two stages of the ring: with four an SM holds half as many of the blocks of
// 128 (2^20 scattered records on 1,282 triangles 1.14 against 1.11 ms, a frame
// of 2^20 rays on 5,122 triangles 1.30 against 1.24 ms).
constexpr int kStages = 2;

// Every pair of a ray and a triangle is decided, but not one at a time: the
// records are kept in a spatial order (the BVH's, or along a Morton curve
// where the scene has none), their padded boxes are merged over 8 and over 32
// consecutive records (box8, box32), and a box that no ray of a warp enters
// at or before its best hit rules out its records as the record's own box
// would.  The block first tests its rays against the merged boxes of a run of
// kBruteRun tiles and lists the tiles some ray needs; only those are copied.
// In them every lane marks the groups of 8 its ray enters, then goes over its
// own groups and, in each, over the records it may enter: lanes look at
// different records.  (All lanes over every group that some lane enters is as
// good while a warp's rays are neighbours, and slower than one box test a pair
// where they are strangers: 2^20 scattered records on 1,282 triangles 1.37 ms
// with one box test a pair, 1.50 ms so, 1.11 with the lanes' own groups.)
// Ties take the smaller reference index, so the order does not show.  2^16
// rays, 20,482 triangles, depth 3: 3.87 -> 0.29 ms a frame (one GB300;
// before, one box test a pair).  The merged boxes alone, over the
// mesh's own order, gain nothing: a subdivided sphere lists neighbouring
// triangles far apart.
//
// TILE: hit records per stage of the ring (SPLAT_TUNE_BRUTE_TILE: 32, 64 or
// 128); the ring holds kStages x TILE x 116 bytes of shared memory.
constexpr int kBruteRun = 512;
// One ray a lane in blocks of 128: a block's tiles are then those of a small
// patch, and blocks over empty parts of the scene end early without holding
// others up (two rays a lane in blocks of 256: 515 against 450 us a frame of
// 2^16 rays).
constexpr int kScanThreads = 128;

// The groups of 8 that a tile of cnt records has, as bits.
__device__ __forceinline__ uint32_t group_bits(int cnt) {
    const int groups = (cnt + 7) / 8;
    return groups >= 32 ? 0xffffffffu : (1u << groups) - 1u;
}
// Which of the 8 boxes of a group a lane's ray may enter, as bits.  Lanes look
// at different groups, and where groups lie 256 bytes apart, equal boxes of all
// of them are in the same banks: there a lane starts at box g of its group g.
__device__ __forceinline__ uint32_t box_bits(const TriBox* box, int g, const float inv[3], const float oinv[3],
                                             float best) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int q = (i + g) & 7;
        m |= (enters(box[q].lo, box[q].hi, inv, oinv, best) ? 1u : 0u) << q;
    }
    return m;
}

template <bool AOS, int TILE>
__global__ void __launch_bounds__(kScanThreads) hit_brute_kernel(RaySrc src, const TriHit* __restrict__ recs,
                                                                  BruteBoxes boxes,
                                                                  int64_t n_recs, int64_t per_split,
                                                                  int32_t* __restrict__ hit_idx,
                                                                  float* __restrict__ hit_t,
                                                                  unsigned long long* __restrict__ tmp,
                                                                  int32_t* err, int stall_tile) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    TriHit* tiles = reinterpret_cast<TriHit*>(smem_raw);
    TriBox* btiles = reinterpret_cast<TriBox*>(smem_raw + (size_t)kStages * TILE * sizeof(TriHit));
    TriBox* gtiles = btiles + kStages * TILE;
    constexpr int kWarps = kScanThreads / 32;
    __shared__ uint32_t s_need[kWarps][kBruteRun / 32];  // per warp: the run's tiles its rays may need
    __shared__ int16_t s_list[kBruteRun];                // the tiles some warp needs, in order
    __shared__ int s_n;
    __shared__ __align__(8) uint64_t bars[kStages];
    // stall_tile >= 0 (test only): the wait for that tile polls `stall`, a
    // barrier that no copy and no thread ever completes, kStallPolls times,
    // so the block takes the failure path below with its copies in flight
    __shared__ __align__(8) uint64_t stall;

    const int64_t n = src.d_count ? *src.d_count : src.n;
    const int64_t ray0 = (int64_t)blockIdx.x * kScanThreads;
    if (ray0 >= n) return;
    const int64_t tb = (int64_t)blockIdx.y * per_split;
    const int64_t te = min(n_recs, tb + per_split);
    if (tb >= te) return;
    const int n_tiles = (int)((te - tb + TILE - 1) / TILE);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;

    // a warp's rays are consecutive; a first bounce takes them in 8 x 4 tiles
    // of the light grid, so that a block's rays are a patch of it (613 -> 515
    // us a frame of 2^16 rays: as columns of the grid its warps need different
    // tiles and wait for one another at every one)
    const int64_t at = ray0 + threadIdx.x;
    const int64_t k = src.tile_h > 0 && at < n && n < (int64_t(1) << 32)
                          ? (int64_t)grid_tile_ray((uint32_t)at, (uint32_t)src.tile_h, (uint32_t)n)
                          : at;
    const HitRay ray = k < n ? load_hit_ray<AOS>(src, k) : HitRay{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0};
    // an idle lane's ray enters no box
    float best = k < n ? __int_as_float(0x7f800000) : -__int_as_float(0x7f800000);
    int32_t bi = 1;
    // slab-test terms of the padded-box pre-test
    const float inv[3] = {safe_inv(ray.dx), safe_inv(ray.dy), safe_inv(ray.dz)};
    const float oinv[3] = {ray.ox * inv[0], ray.oy * inv[1], ray.oz * inv[2]};

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(&bars[s], 1);
        mbar_init(&stall, 1);
        fence_mbar_init();
    }
    __syncthreads();

    // the it-th tile of the launch is tile kt of the range
    auto issue = [&](int it, int kt) {
        const int s = it % kStages;
        const int64_t first = tb + (int64_t)kt * TILE;
        const uint32_t cnt = (uint32_t)min((int64_t)TILE, te - first);
        const uint32_t bytes = cnt * (uint32_t)sizeof(TriHit), bbytes = cnt * (uint32_t)sizeof(TriBox);
        const uint32_t gbytes = (cnt + 7) / 8 * (uint32_t)sizeof(TriBox);
        mbar_arrive_expect_tx(&bars[s], bytes + bbytes + gbytes);
        bulk_g2s(tiles + s * TILE, recs + first, bytes, &bars[s]);
        bulk_g2s(btiles + s * TILE, boxes.box + first, bbytes, &bars[s]);
        bulk_g2s(gtiles + s * (TILE / 8), boxes.box8 + first / 8, gbytes, &bars[s]);
    };

    const int64_t last32 = (te - 1) / 32;
    int done = 0;    // tiles consumed so far
    int issued = 0;  // tiles issued so far (thread 0)
    bool failed = false;
    for (int run = 0; run < n_tiles && !failed; run += kBruteRun) {
        const int run_tiles = min(kBruteRun, n_tiles - run);
        // the run's tiles that a ray of this warp may need
        for (int t0 = 0; t0 < run_tiles; t0 += 32) {
            uint32_t bits = 0;
            const int m = min(32, run_tiles - t0);
#pragma unroll 4
            for (int t = 0; t < m; ++t) {
                const int64_t b0 = (tb + (int64_t)(run + t0 + t) * TILE) / 32;
                bool need = false;
#pragma unroll
                for (int i = 0; i < TILE / 32; ++i) {
                    const TriBox* bx = boxes.box32 + min(b0 + i, last32);
                    const float4 lo = __ldg(&bx->lo), hi = __ldg(&bx->hi);
                    need |= enters(lo, hi, inv, oinv, best);
                }
                bits |= (__any_sync(0xffffffffu, need) ? 1u : 0u) << t;
            }
            if (lane == 0) s_need[wid][t0 / 32] = bits;
        }
        __syncthreads();
        if (wid == 0) {
            int cnt = 0;
            for (int t0 = 0; t0 < run_tiles; t0 += 32) {
                uint32_t any = 0;
#pragma unroll
                for (int w = 0; w < kWarps; ++w) any |= s_need[w][t0 / 32];
                if (any >> lane & 1u) s_list[cnt + __popc(any & ((1u << lane) - 1u))] = (int16_t)(t0 + lane);
                cnt += __popc(any);
            }
            if (lane == 0) s_n = cnt;
        }
        __syncthreads();
        const int n_list = s_n;
        if (threadIdx.x == 0) {
            if (run > 0) fence_proxy_async();
            for (int j = 0; j < min(kStages, n_list); ++j) issue(issued++, run + s_list[j]);
        }
        for (int j = 0; j < n_list; ++j) {
            const int s = done % kStages;
            const uint32_t ph = (uint32_t)(done / kStages) & 1u;
            const int rel = s_list[j], kt = run + rel;
            const bool ok =
                kt == stall_tile ? mbar_wait_bounded(&stall, 0u, kStallPolls) : mbar_wait_bounded(&bars[s], ph);
            if (__syncthreads_or(!ok)) {
                failed = true;
                break;
            }
            const int cnt = (int)min((int64_t)TILE, te - (tb + (int64_t)kt * TILE));
            const TriHit* tile = tiles + s * TILE;
            const TriBox* btile = btiles + s * TILE;
            const TriBox* gtile = gtiles + s * (TILE / 8);
            if (s_need[wid][rel / 32] >> (rel & 31) & 1u) {
                // each lane's groups of 8, then its records in them
                uint32_t gm = 0;
#pragma unroll
                for (int g = 0; g < TILE / 8; ++g)
                    gm |= (enters(gtile[g].lo, gtile[g].hi, inv, oinv, best) ? 1u : 0u) << g;
                gm &= group_bits(cnt);
                for (; gm; gm &= gm - 1) {
                    const int g = __ffs(gm) - 1;
                    uint32_t m = box_bits(btile + g * 8, g, inv, oinv, best);
                    if (g * 8 + 8 > cnt) m &= (1u << (cnt - g * 8)) - 1u;
                    for (; m; m &= m - 1) {
                        const TriHit& h = tile[g * 8 + __ffs(m) - 1];
                        float num, den;
                        if (!tri_candidate(h.n_nv, ray, best, num, den)) continue;
                        const float4 q1 = h.a_idx;
                        const int32_t idx = __float_as_int(q1.w);
                        bool inside;
                        const float t = tri_t_from(num, den, q1, h.e0, h.e1, h.inv, ray, inside);
                        if (inside & (t > 0.0f) & (idx != ray.ig) & ((t < best) | ((t == best) & (idx < bi)))) {
                            best = t;
                            bi = idx;
                        }
                    }
                }
            }
            ++done;
            __syncthreads();
            if (threadIdx.x == 0 && j + kStages < n_list) {
                fence_proxy_async();
                issue(issued++, run + s_list[j + kStages]);
            }
        }
    }
    if (failed) {
        if (threadIdx.x == 0) {
            atomicOr(err, 1);
            // drain this block's copies still in flight (bounded) before exit
            for (int it = done; it < issued; ++it)
                (void)mbar_wait_bounded(&bars[it % kStages], (uint32_t)(it / kStages) & 1u);
        }
        return;
    }

    if (k >= n) return;
    if (tmp) {
        if (bi != 1) atomicMin(tmp + k, (unsigned long long)pack_argmin(best, (uint32_t)bi));
    } else {
        hit_idx[k] = bi;
        if (hit_t) hit_t[k] = best;
    }
}

__global__ void fill_u64_kernel(unsigned long long* p, int64_t n, const int64_t* d_count, unsigned long long v) {
    const int64_t m = d_count ? *d_count : n;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        p[k] = v;
}

__global__ void unpack_hits_kernel(const unsigned long long* tmp, int64_t n, const int64_t* d_count,
                                   int32_t* hit_idx, float* hit_t) {
    const int64_t m = d_count ? *d_count : n;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t v = tmp[k];
        hit_idx[k] = (int32_t)(uint32_t)(v & 0xffffffffull);
        if (hit_t) hit_t[k] = monotonic_f32((uint32_t)(v >> 32));
    }
}

__global__ void miss_kernel(int64_t n, const int64_t* d_count, int32_t* hit_idx, float* hit_t) {
    const int64_t m = d_count ? *d_count : n;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        hit_idx[k] = 1;
        if (hit_t) hit_t[k] = __int_as_float(0x7f800000);
    }
}

static int grid_for(int64_t n, int threads, int sm_count, int per_sm) {
    int64_t b = (n + threads - 1) / threads;
    int64_t cap = (int64_t)sm_count * per_sm;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

cudaError_t launch_unpack_hits(const uint64_t* tmp, int64_t n, const int64_t* d_count, int32_t* hit_idx,
                               float* hit_t, cudaStream_t s) {
    unpack_hits_kernel<<<grid_for(n, 256, 152, 8), 256, 0, s>>>((const unsigned long long*)tmp, n, d_count, hit_idx,
                                                                hit_t);
    ++g_launches;
    return cudaGetLastError();
}


template <int TILE>
static void launch_brute_tiles(dim3 grid, cudaStream_t s, const RaySrc& rays, const TriHit* recs, const BruteBoxes& boxes,
                               int64_t n_recs, int64_t per_split, int32_t* hit_idx, float* hit_t,
                               unsigned long long* tmp, int32_t* err, int stall_tile) {
    const size_t smem = (size_t)kStages * (TILE * (sizeof(TriHit) + sizeof(TriBox)) + TILE / 8 * sizeof(TriBox));
    static bool configured = false;  // rings above 48 KB need the opt-in
    if (!configured) {
        cudaFuncSetAttribute(hit_brute_kernel<true, TILE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(hit_brute_kernel<false, TILE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
        configured = true;
    }
    if (rays.aos)
        hit_brute_kernel<true, TILE><<<grid, kScanThreads, smem, s>>>(rays, recs, boxes, n_recs, per_split,
                                                                             hit_idx, hit_t, tmp, err, stall_tile);
    else
        hit_brute_kernel<false, TILE><<<grid, kScanThreads, smem, s>>>(rays, recs, boxes, n_recs, per_split,
                                                                              hit_idx, hit_t, tmp, err, stall_tile);
}

// packed: tmp holds kNoHit already and keeps the results.
static cudaError_t brute_launch(const RaySrc& rays, int64_t cap, const TriHit* recs, const TriBox* all_boxes,
                                int64_t n_recs, int32_t* hit_idx, float* hit_t, uint64_t* tmp, bool packed,
                                int32_t* err, int sm_count, cudaStream_t s) {
    if (cap <= 0) return cudaSuccess;
    const BruteBoxes boxes = brute_boxes_of(all_boxes, n_recs);
    const int tile = g_tune[SPLAT_TUNE_BRUTE_TILE].load();
    const int64_t rays_per_block = kScanThreads;
    const int64_t ray_blocks = (cap + rays_per_block - 1) / rays_per_block;
    // split the triangle range so the grid covers the GPU several times over
    // (kScanSplit blocks of 128 for each of the knob's: 2^16 rays, 20,482
    // triangles, 450 / 418 / 411 / 382 us a frame with 1 / 2 / 4 / 8), down to
    // one tile a block (1,024 rays, 322 triangles: 180 -> 129 us a frame)
    constexpr int64_t kScanSplit = 8;
    const int stall_tile = g_tune[SPLAT_TUNE_TEST_WAIT_STALL] - 1;
    const int64_t least = (stall_tile >= 0 ? 4 : 1) * (int64_t)tile;  // the stall wants a block's later tiles
    int64_t wanted = (kScanSplit * sm_count * g_tune[SPLAT_TUNE_BRUTE_BLOCKS_PER_SM] + ray_blocks - 1) / ray_blocks;
    if (tmp == nullptr) wanted = 1;
    const auto [splits, per_split] = split_records(n_recs, wanted, least, tile);
    const bool use_tmp = packed || splits > 1;
    if (use_tmp && !packed) {
        fill_u64_kernel<<<grid_for(cap, 256, sm_count, 8), 256, 0, s>>>((unsigned long long*)tmp, cap, rays.d_count,
                                                                        (unsigned long long)kNoHit);
        ++g_launches;
    }
    dim3 grid((unsigned)ray_blocks, (unsigned)splits);
    if (n_recs > 0) {
        unsigned long long* t = use_tmp ? (unsigned long long*)tmp : nullptr;
        if (tile == 32)
            launch_brute_tiles<32>(grid, s, rays, recs, boxes, n_recs, per_split, hit_idx, hit_t, t, err, stall_tile);
        else if (tile == 128)
            launch_brute_tiles<128>(grid, s, rays, recs, boxes, n_recs, per_split, hit_idx, hit_t, t, err, stall_tile);
        else
            launch_brute_tiles<64>(grid, s, rays, recs, boxes, n_recs, per_split, hit_idx, hit_t, t, err, stall_tile);
        ++g_launches;
    } else if (!packed) {
        // no triangles: every ray misses
        miss_kernel<<<grid_for(cap, 256, sm_count, 8), 256, 0, s>>>(cap, rays.d_count, hit_idx, hit_t);
        ++g_launches;
        return cudaGetLastError();
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (use_tmp && !packed) return launch_unpack_hits(tmp, cap, rays.d_count, hit_idx, hit_t, s);
    return cudaSuccess;
}

cudaError_t launch_hit_brute(const RaySrc& rays, int64_t cap, const TriHit* recs, const TriBox* boxes, int64_t n_recs,
                             int32_t* hit_idx, float* hit_t, uint64_t* tmp, int32_t* err, int sm_count,
                             cudaStream_t s) {
    return brute_launch(rays, cap, recs, boxes, n_recs, hit_idx, hit_t, tmp, false, err, sm_count, s);
}

cudaError_t launch_hit_brute_packed(const RaySrc& rays, int64_t cap, const TriHit* recs, const TriBox* boxes,
                                    int64_t n_recs, uint64_t* packed, int32_t* err, int sm_count, cudaStream_t s) {
    return brute_launch(rays, cap, recs, boxes, n_recs, nullptr, nullptr, packed, true, err, sm_count, s);
}

// ---------------------------------------------------------------------------
// brute force over the reference's n_tris array (next_hit_kernel6 drop-in)
// ---------------------------------------------------------------------------
// Box of a caller's record outside which no point can be accepted, or all of
// space where that is not sure.  Acceptance looks at the point's barycentrics
// alone, so the box holds only for a plane normal that is the triangle's own
// (an accepted point then lies in the triangle's plane) and for a triangle
// that is no sliver (whose barycentrics' rounding moves points across its
// edges): |n . edge| <= 2.5e-4 |n| |edge| for both edges at a (measured by the
// edge, not by the diagonal: a needle's short edge may be the normal's own
// direction) and sin^2 of the corner at a >= 1e-2.  The normal then leans by
// at most 5e-3, an accepted point is at most 2.5e-4 of an edge off the
// triangle's plane, and all accepted points leave the triangle by less than
// half the padding, 1e-3 of the diagonal plus 1e-4 max(1, largest
// coordinate), as long as the ray starts within kNtrisReach of that scale and
// its direction is one that the box test keeps (plain_direction).  A record
// without a normal (the sentinel) accepts nothing: an empty box.
constexpr float kNtrisReach = 100.0f;
// The box test raises components below 1e-30 to that (safe_inv), which moves a
// point at distance t |d| by t 1e-30: nothing at 300 scales while |d| >= 1e-20.
// From 1e30 on inverses are close to the subnormal ones.  A zero direction
// accepts nothing, and idle lanes have one.
__device__ __forceinline__ bool plain_direction(float dx, float dy, float dz) {
    const float m = fmaxf(fmaxf(fabsf(dx), fabsf(dy)), fabsf(dz));
    return (m >= 1.0e-20f && m <= 1.0e30f) || m == 0.0f;
}
__device__ __forceinline__ TriBox ntris_box(const TriHit& h, F3 a, F3 b, F3 c, float& scale) {
    const float inf = __int_as_float(0x7f800000);
    const F3 n = {h.n_nv.x, h.n_nv.y, h.n_nv.z}, e0 = {h.e0.x, h.e0.y, h.e0.z}, e1 = {h.e1.x, h.e1.y, h.e1.z};
    const float lx = fminf(fminf(a.x, b.x), c.x), ly = fminf(fminf(a.y, b.y), c.y), lz = fminf(fminf(a.z, b.z), c.z);
    const float hx = fmaxf(fmaxf(a.x, b.x), c.x), hy = fmaxf(fmaxf(a.y, b.y), c.y), hz = fmaxf(fmaxf(a.z, b.z), c.z);
    const float dx = hx - lx, dy = hy - ly, dz = hz - lz;
    const float diag = sqrtf(dx * dx + dy * dy + dz * dz);
    scale = fmaxf(1.0f, fmaxf(fmaxf(fmaxf(fabsf(lx), fabsf(hx)), fmaxf(fabsf(ly), fabsf(hy))),
                              fmaxf(fabsf(lz), fabsf(hz))));
    const float lean = 2.5e-4f * sqrtf(dot(n, n));
    const bool own =
        fabsf(dot(n, e0)) <= lean * sqrtf(h.e0.w) && fabsf(dot(n, e1)) <= lean * sqrtf(h.e1.w) && diag < inf;
    const bool wide = h.inv.y * (h.e0.w * h.e1.w) <= 1.0e2f && h.inv.y > 0.0f;
    if (n.x == 0.0f && n.y == 0.0f && n.z == 0.0f)
        return TriBox{make_float4(inf, inf, inf, 0.f), make_float4(-inf, -inf, -inf, 0.f)};
    if (!(own && wide)) return TriBox{make_float4(-inf, -inf, -inf, 0.f), make_float4(inf, inf, inf, 0.f)};
    const float pad = 1.0e-4f * scale + 1.0e-3f * diag;
    return TriBox{make_float4(lx - pad, ly - pad, lz - pad, 0.f), make_float4(hx + pad, hy + pad, hz + pad, 0.f)};
}

// Ascending order of the block's 256 keys, one a thread (bitonic; strides
// below a warp by shuffle, the others through shared memory).
__device__ __forceinline__ uint32_t block_sort256(uint32_t key, uint32_t* s_key) {
    const int i = threadIdx.x;
#pragma unroll
    for (int k = 2; k <= 256; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j; j >>= 1) {
            uint32_t other;
            if (j >= 32) {
                __syncthreads();
                s_key[i] = key;
                __syncthreads();
                other = s_key[i ^ j];
            } else {
                other = __shfl_xor_sync(0xffffffffu, key, j);
            }
            const bool up = (i & k) == 0, low = (i & j) == 0;
            key = (low == up) ? min(key, other) : max(key, other);
        }
    }
    return key;
}

__device__ __forceinline__ uint32_t spread8(uint32_t x) {  // 8 bits, two zeros between
    x = (x | (x << 8)) & 0x0000f00fu;
    x = (x | (x << 4)) & 0x000c30c3u;
    return (x | (x << 2)) & 0x00249249u;
}

// A tile of 256 of the caller's records is packed, given boxes (ntris_box) and
// put along a Morton curve of its own box, so that boxes merged over 8 and 32
// of them are small whatever order the array has; a warp passes by those over
// 32 that none of its rays enters, and every lane goes over the groups of 8 of
// its own ray as in hit_brute_kernel (a warp with a ray too far out for the
// boxes tests every triangle).  Equal distances take the earlier record, as
// over the array's order: pos is the record's place in its tile.  Scattered /
// gridded rays, us a call (a division and the full test for every pair; all
// lanes over every group that some lane enters, two rays a lane; now):
//   322 triangles, 2^16 rays    71 / 76         106 / 56      59 / 46
//   1,282, 2^16                 206             190           112
//   5,122, 300,000              3,026 / 3,374   2,170 / 634   1,175 / 663
// Boxes of 8 records; the padding puts equal ones of different groups into
// different banks.
struct TriBox8 {
    TriBox b[8];
    float4 pad;
};

__global__ void __launch_bounds__(kBruteThreads) hit_ntris_kernel(const splat_adray_t* __restrict__ rays,
                                                                   int64_t n_rays, const splat_ntri_t* __restrict__ nt,
                                                                   int64_t n_tris, int64_t per_split,
                                                                   unsigned long long* __restrict__ tmp) {
    static_assert(kTile == kBruteThreads && kTile == 256, "a record a thread");
    constexpr int kWarps = kBruteThreads / 32;
    __shared__ TriHit tile[kTile];  // inv.z: pos
    __shared__ __align__(16) TriBox8 box[kTile / 8];
    __shared__ TriBox box8[kTile / 8], box32[kTile / 32];
    __shared__ float s_ext[kWarps][7];
    __shared__ uint32_t s_key[kTile];
    __shared__ float s_scale;
    const float inf = __int_as_float(0x7f800000);
    RaySrc src{};
    src.aos = rays;
    src.n = n_rays;
    const int64_t tb = (int64_t)blockIdx.y * per_split;
    const int64_t te = min(n_tris, tb + per_split);
    if (tb >= te) return;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t k = (int64_t)blockIdx.x * kBruteThreads + tid;
    const HitRay ray = k < n_rays ? load_hit_ray<true>(src, k) : HitRay{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0};
    float best = k < n_rays ? inf : -inf;  // an idle lane's ray enters no box
    int32_t bi = 1;
    const float inv[3] = {safe_inv(ray.dx), safe_inv(ray.dy), safe_inv(ray.dz)};
    const float oinv[3] = {ray.ox * inv[0], ray.oy * inv[1], ray.oz * inv[2]};
    // largest |origin coordinate| over the warp; infinite: some direction is not plain
    float reach = fmaxf(fmaxf(fabsf(ray.ox), fabsf(ray.oy)), fabsf(ray.oz));
    if (!plain_direction(ray.dx, ray.dy, ray.dz)) reach = inf;
    reach = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(reach)));
    for (int64_t base = tb; base < te; base += kTile) {
        const int cnt = (int)min((int64_t)kTile, te - base);
        TriHit h;
        TriBox m{make_float4(inf, inf, inf, 0.f), make_float4(-inf, -inf, -inf, 0.f)};
        float scale = inf, c[3] = {0.f, 0.f, 0.f}, lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
        if (tid < cnt) {
            const splat_ntri_t& q = nt[base + tid];
            const F3 v0 = f3(q.v[1]), v1 = f3(q.v[2]), v2 = f3(q.v[3]);
            h = pack_one(q.idx, f3(q.v[0]), v0, v1, v2);
            h.inv.z = __int_as_float(tid);
            m = ntris_box(h, v0, v1, v2, scale);
            c[0] = v0.x;
            c[1] = v0.y;
            c[2] = v0.z;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (!(fabsf(c[a]) < inf)) c[a] = 0.0f;
                lo[a] = hi[a] = c[a];
            }
        }
        // the tile's extent and smallest scale
        for (int o = 16; o; o >>= 1) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
                hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
            }
            scale = fminf(scale, __shfl_xor_sync(0xffffffffu, scale, o));
        }
        if (lane == 0) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                s_ext[wid][a] = lo[a];
                s_ext[wid][3 + a] = hi[a];
            }
            s_ext[wid][6] = scale;
        }
        __syncthreads();
        uint32_t code = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            float l = inf, u = -inf;
            for (int w = 0; w < kWarps; ++w) {
                l = fminf(l, s_ext[w][a]);
                u = fmaxf(u, s_ext[w][3 + a]);
            }
            const float f = u > l ? (c[a] - l) * (256.0f / (u - l)) : 0.0f;
            code |= spread8((uint32_t)fminf(fmaxf(f, 0.0f), 255.0f)) << a;
        }
        if (tid == 0) {
            float w = inf;
            for (int i = 0; i < kWarps; ++i) w = fminf(w, s_ext[i][6]);
            s_scale = w;
        }
        // sorted: the record that goes to slot tid; its owner learns the slot
        const uint32_t key = block_sort256(tid < cnt ? (code << 8) | (uint32_t)tid : 0xffffff00u | (uint32_t)tid, s_key);
        __syncthreads();
        s_key[key & 255u] = (uint32_t)tid;
        __syncthreads();
        const int slot = (int)s_key[tid];
        if (tid < cnt) tile[slot] = h;
        box[slot >> 3].b[slot & 7] = m;
        __syncthreads();
        m = box[tid >> 3].b[tid & 7];
        for (int o = 1; o < 32; o <<= 1) {
            m.lo.x = fminf(m.lo.x, __shfl_xor_sync(0xffffffffu, m.lo.x, o));
            m.lo.y = fminf(m.lo.y, __shfl_xor_sync(0xffffffffu, m.lo.y, o));
            m.lo.z = fminf(m.lo.z, __shfl_xor_sync(0xffffffffu, m.lo.z, o));
            m.hi.x = fmaxf(m.hi.x, __shfl_xor_sync(0xffffffffu, m.hi.x, o));
            m.hi.y = fmaxf(m.hi.y, __shfl_xor_sync(0xffffffffu, m.hi.y, o));
            m.hi.z = fmaxf(m.hi.z, __shfl_xor_sync(0xffffffffu, m.hi.z, o));
            if (o == 4 && (lane & 7) == 0) box8[tid / 8] = m;
        }
        if (lane == 0) box32[wid] = m;
        __syncthreads();
        // (a NaN origin drops out of reach: its ray passes no triangle's test)
        const bool all = !(reach <= kNtrisReach * s_scale);
        int32_t bpos = -1;  // a best hit from an earlier tile wins ties
        uint32_t gm = 0;
#pragma unroll 1
        for (int part = 0; part * 32 < cnt; ++part) {
            const bool some = all || enters(box32[part].lo, box32[part].hi, inv, oinv, best);
            if (!__any_sync(0xffffffffu, some)) continue;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const TriBox& b = box8[part * 4 + g];
                gm |= (all || enters(b.lo, b.hi, inv, oinv, best) ? 1u : 0u) << (part * 4 + g);
            }
        }
#pragma unroll 1
        for (gm &= group_bits(cnt); gm; gm &= gm - 1) {
            const int g = __ffs(gm) - 1;
            uint32_t m = all ? 0xffu : box_bits(box[g].b, 0, inv, oinv, best);
            if (g * 8 + 8 > cnt) m &= (1u << (cnt - g * 8)) - 1u;
#pragma unroll 1
            for (; m; m &= m - 1) {
                const TriHit& h = tile[g * 8 + __ffs(m) - 1];
                float num, den;
                if (!tri_candidate(h.n_nv, ray, best, num, den)) continue;
                const float4 q1 = h.a_idx, q4 = h.inv;
                const int32_t idx = __float_as_int(q1.w), pos = __float_as_int(q4.z);
                bool inside;
                const float t = tri_t_from(num, den, q1, h.e0, h.e1, q4, ray, inside);
                // next_hit_kernel6 (src/hitters.jl:183) has no i != 1 test: the
                // sentinel's t is NaN and fails t > 0.
                if (inside & (t > 0.0f) & (idx != ray.ig) & ((t < best) | ((t == best) & (pos < bpos)))) {
                    best = t;
                    bi = idx;
                    bpos = pos;
                }
            }
        }
        __syncthreads();
    }
    if (k < n_rays && bi != 1) atomicMin(tmp + k, (unsigned long long)pack_argmin(best, (uint32_t)bi));
}

// Up to kNtrisDirect records: every one against every ray, for the boxes and
// their order take longer to make than they save.  us a call, boxes / none:
//   42 triangles    2^20 rays 150 / 124   300,000 of a grid 58 / 58
//   82              246 / 209             70 / 77
//   128             244 / 309             73 / 107
constexpr int kNtrisDirect = 96;
__global__ void __launch_bounds__(kBruteThreads) hit_ntris_direct_kernel(const splat_adray_t* __restrict__ rays,
                                                                          int64_t n_rays,
                                                                          const splat_ntri_t* __restrict__ nt,
                                                                          int n_tris,
                                                                          unsigned long long* __restrict__ tmp) {
    __shared__ TriHit tile[kNtrisDirect];
    RaySrc src{};
    src.aos = rays;
    src.n = n_rays;
    const int tid = threadIdx.x;
    const int64_t k = (int64_t)blockIdx.x * kBruteThreads + tid;
    const HitRay ray = k < n_rays ? load_hit_ray<true>(src, k) : HitRay{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0};
    float best = __int_as_float(0x7f800000);
    int32_t bi = 1;
    if (tid < n_tris) {
        const splat_ntri_t& q = nt[tid];
        tile[tid] = pack_one(q.idx, f3(q.v[0]), f3(q.v[1]), f3(q.v[2]), f3(q.v[3]));
    }
    __syncthreads();
#pragma unroll 2
    for (int j = 0; j < n_tris; ++j) {
        float num, den;
        if (!tri_candidate(tile[j].n_nv, ray, best, num, den)) continue;
        const float4 q1 = tile[j].a_idx;
        const int32_t idx = __float_as_int(q1.w);
        bool inside;
        const float t = tri_t_from(num, den, q1, tile[j].e0, tile[j].e1, tile[j].inv, ray, inside);
        if (inside & (t > 0.0f) & (idx != ray.ig) & (t < best)) {
            best = t;
            bi = idx;
        }
    }
    if (k < n_rays && bi != 1) atomicMin(tmp + k, (unsigned long long)pack_argmin(best, (uint32_t)bi));
}

cudaError_t launch_hit_brute_ntris(const splat_adray_t* rays, int64_t n_rays, const splat_ntri_t* ntris,
                                   int64_t n_tris, uint64_t* tmp, int32_t* hit_idx, int sm_count, cudaStream_t s) {
    if (n_rays <= 0) return cudaSuccess;
    fill_u64_kernel<<<grid_for(n_rays, 256, sm_count, 8), 256, 0, s>>>((unsigned long long*)tmp, n_rays, nullptr,
                                                                       (unsigned long long)kNoHit);
    ++g_launches;
    const int64_t rays_per_block = kBruteThreads;
    const int64_t ray_blocks = (n_rays + rays_per_block - 1) / rays_per_block;
    const int64_t wanted = ((int64_t)sm_count * 4 + ray_blocks - 1) / ray_blocks;
    const auto [splits, per_split] = split_records(n_tris, wanted, kTile, kTile);
    if (n_tris > kNtrisDirect) {
        dim3 grid((unsigned)ray_blocks, (unsigned)splits);
        hit_ntris_kernel<<<grid, kBruteThreads, 0, s>>>(rays, n_rays, ntris, n_tris, per_split,
                                                         (unsigned long long*)tmp);
        ++g_launches;
    } else if (n_tris > 0) {
        hit_ntris_direct_kernel<<<(unsigned)ray_blocks, kBruteThreads, 0, s>>>(rays, n_rays, ntris, (int)n_tris,
                                                                               (unsigned long long*)tmp);
        ++g_launches;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_unpack_hits(tmp, n_rays, nullptr, hit_idx, nullptr, s);
}

// ---------------------------------------------------------------------------
// brute force over n_tris with library-held scratch (no allocation)
// ---------------------------------------------------------------------------
// The packed (t, index) words of splat_next_hit_brute_static live here rather
// than in caller memory.  Every GPU that loads the library holds this array
// until the process exits; all calls share it.
static __device__ __align__(256) unsigned long long g_static_hit_tmp[kStaticHitMaxRays];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
void* g_static_ptr[kMaxDevices] = {nullptr};

// Device address of g_static_hit_tmp on the current device, looked up once
// per device (host code only has a host-side stand-in for the symbol).
cudaError_t static_hit_scratch(unsigned long long** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (g_static_ptr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_hit_tmp);
        if (e != cudaSuccess) return e;
        g_static_ptr[dev] = p;
    }
    *out = reinterpret_cast<unsigned long long*>(g_static_ptr[dev]);
    return cudaSuccess;
}
}  // namespace

cudaError_t launch_hit_brute_ntris_static(const splat_adray_t* rays, int64_t n_rays, const splat_ntri_t* ntris,
                                          int64_t n_tris, int32_t* hit_idx, int sm_count, cudaStream_t s) {
    unsigned long long* tmp = nullptr;
    cudaError_t e = static_hit_scratch(&tmp);
    if (e != cudaSuccess) return e;
    // launch_hit_brute_ntris first resets the n_rays words it uses to (Inf, 1)
    return launch_hit_brute_ntris(rays, n_rays, ntris, n_tris, reinterpret_cast<uint64_t*>(tmp), hit_idx, sm_count,
                                  s);
}

// ---------------------------------------------------------------------------
// BVH traversal
// ---------------------------------------------------------------------------
constexpr int kBvhThreads = 128;

// Grid of a work-counter launch: as many blocks as stay resident together
// (capped by a blocks-per-SM knob and by the work), so the launch is one
// wave that drains the counter.
int resident_grid(const void* kernel, int64_t cap, int sm_count, int threads, int max_per_sm) {
    static std::mutex mu;
    static std::unordered_map<const void*, int> occ;
    int per_sm = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = occ.find(kernel);
        if (it == occ.end()) {
            int nb = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, 0) != cudaSuccess || nb < 1)
                nb = 4;
            it = occ.emplace(kernel, nb).first;
        }
        per_sm = it->second;
    }
    if (per_sm > max_per_sm) per_sm = max_per_sm;
    return grid_for(cap, threads, sm_count, per_sm);
}

template <bool AOS>
__global__ void __launch_bounds__(kBvhThreads) hit_bvh_kernel(RaySrc src, BvhView bvh, int32_t* __restrict__ hit_idx,
                                                              float* __restrict__ hit_t, int32_t* err) {
    const int64_t n = src.d_count ? *src.d_count : src.n;
    int2 stack[kBvhStack];  // (ref, entry distance bits)
    for_each_ray(n, src.fetch, [&](int64_t kk) {
        const int64_t k = src.perm ? (int64_t)src.perm[kk] : kk;
        const HitRay r = load_hit_ray<AOS>(src, k);
        const SlabRay sr = slab_ray(r, bvh.root4);
        // the near plane of an axis by the sign of the inverse direction, as in node4_slabs
        const bool sx = sr.ix < 0.0f, sy = sr.iy < 0.0f, sz = sr.iz < 0.0f;
        float best = __int_as_float(0x7f800000);
        int32_t bi = 1;
        int sp = 0;
        int ref = 0;
        while (true) {
            if (ref >= 0) {
                const BvhNode* nd = bvh.nodes + ref;
                const float4 bx = __ldg(&nd->x);
                const float4 by = __ldg(&nd->y);
                const float4 bz = __ldg(&nd->z);
                const int4 c = __ldg(&nd->c);
                const float a0 = fmaf(sx ? bx.y : bx.x, sr.ix, sr.nx), b0 = fmaf(sx ? bx.x : bx.y, sr.ix, sr.fx);
                const float a1 = fmaf(sy ? by.y : by.x, sr.iy, sr.ny), b1 = fmaf(sy ? by.x : by.y, sr.iy, sr.fy);
                const float a2 = fmaf(sz ? bz.y : bz.x, sr.iz, sr.nz), b2 = fmaf(sz ? bz.x : bz.y, sr.iz, sr.fz);
                const float tmin0 = fmaxf(fmaxf(a0, a1), a2), tmax0 = fminf(fminf(b0, b1), b2);
                const float e0 = fmaf(sx ? bx.w : bx.z, sr.ix, sr.nx), f0 = fmaf(sx ? bx.z : bx.w, sr.ix, sr.fx);
                const float e1 = fmaf(sy ? by.w : by.z, sr.iy, sr.ny), f1 = fmaf(sy ? by.z : by.w, sr.iy, sr.fy);
                const float e2 = fmaf(sz ? bz.w : bz.z, sr.iz, sr.nz), f2 = fmaf(sz ? bz.z : bz.w, sr.iz, sr.fz);
                const float tmin1 = fmaxf(fmaxf(e0, e1), e2), tmax1 = fminf(fminf(f0, f1), f2);
                const bool h0 = (tmin0 <= tmax0) & (tmax0 >= 0.0f) & (tmin0 <= best);
                const bool h1 = (tmin1 <= tmax1) & (tmax1 >= 0.0f) & (tmin1 <= best);
                if (h0 && h1) {
                    int near_ref = c.x, far_ref = c.y;
                    float far_t = tmin1;
                    if (tmin1 < tmin0) {
                        near_ref = c.y;
                        far_ref = c.x;
                        far_t = tmin0;
                    }
                    if (sp < kBvhStack) {
                        stack[sp++] = make_int2(far_ref, __float_as_int(far_t));
                    } else {
                        atomicOr(err, 2);
                    }
                    ref = near_ref;
                    continue;
                }
                if (h0) {
                    ref = c.x;
                    continue;
                }
                if (h1) {
                    ref = c.y;
                    continue;
                }
            } else {
                const int enc = ~ref;
                const int first = enc >> 4;
                const int count = (enc & 15) + 1;
                for (int j = 0; j < count; ++j) {
                    const TriHit* h = bvh.tris + first + j;
                    float num, den;
                    if (!tri_candidate(__ldg(&h->n_nv), r, best, num, den)) continue;
                    const float4 q1 = __ldg(&h->a_idx);
                    const int32_t idx = __float_as_int(q1.w);
                    bool inside;
                    const float t = tri_t_from(num, den, q1, __ldg(&h->e0), __ldg(&h->e1), __ldg(&h->inv), r, inside);
                    if (inside & (t > 0.0f) & (idx != r.ig) & ((t < best) | ((t == best) & (idx < bi)))) {
                        best = t;
                        bi = idx;
                    }
                }
            }
            bool found = false;
            while (sp > 0) {
                const int2 e = stack[--sp];
                if (__int_as_float(e.y) <= best) {
                    ref = e.x;
                    found = true;
                    break;
                }
            }
            if (!found) break;
        }
        hit_idx[k] = bi;
        if (hit_t) hit_t[k] = best;
    });
}

// A caller's records come without a work counter and in no order, and a long
// ray holds up the rays that its warp takes after it: they get four times the
// blocks of the knob, so that most warps take one turn.  982,000 scattered
// rays on a sphere, two-wide tree: 351 -> 306 us; 350,000 records, four calls
// of the caller's bounce loop, four-wide: 660 -> 647 us.
constexpr int kAosGrid = 4;

cudaError_t launch_hit_bvh(const RaySrc& rays, int64_t cap, const BvhView& bvh, int32_t* hit_idx, float* hit_t,
                           int32_t* err, int sm_count, cudaStream_t s) {
    if (cap <= 0) return cudaSuccess;
    const int grid = rays.fetch ? resident_grid(reinterpret_cast<const void*>(hit_bvh_kernel<false>), cap, sm_count,
                                                kBvhThreads, g_tune[SPLAT_TUNE_BVH_BLOCKS_PER_SM])
                                : grid_for(cap, kBvhThreads, sm_count,
                                           (rays.aos ? kAosGrid : 1) * g_tune[SPLAT_TUNE_BVH_BLOCKS_PER_SM]);
    if (rays.aos)
        hit_bvh_kernel<true><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t, err);
    else
        hit_bvh_kernel<false><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t, err);
    ++g_launches;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// four-wide BVH traversal
// ---------------------------------------------------------------------------
// One thread per ray.  A node fetch (128 bytes) tests four child boxes; the
// hit children are sorted by entry distance, the nearest is visited next and
// the others are pushed farthest first together with their entry distance,
// so a popped entry that lies beyond the current best hit is skipped.
// Traversal work of the counting kernels (SPLAT_TUNE_COUNT_WORK): nodes
// visited, triangle pre-tests, full triangle tests, rays traced.  Every GPU
// that loads the library holds these four words; splat_hit_work reads and
// clears them.
__device__ unsigned long long g_hit_work[4];

__device__ __forceinline__ void flush_work(const WorkCount& wc, uint32_t rays) {
    unsigned long long v[4] = {wc.nodes, wc.pre, wc.full, rays};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        for (int o = 16; o; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        if ((threadIdx.x & 31) == 0 && v[i]) atomicAdd(&g_hit_work[i], v[i]);
    }
}

template <bool AOS, bool COUNT>
__global__ void __launch_bounds__(kBvhThreads) hit_bvh4_kernel(RaySrc src, Bvh4View bvh,
                                                               int32_t* __restrict__ hit_idx,
                                                               float* __restrict__ hit_t, int32_t* err) {
    const int64_t n = src.d_count ? *src.d_count : src.n;
    if (src.few && n <= kGroupRays) return;  // the group kernel's
    int2 stack[kBvhStack];
    WorkCount wc{0u, 0u, 0u};
    uint32_t rays = 0;
    for_each_ray(n, src.fetch, [&](int64_t kk) {
        const int64_t k = src.perm ? (int64_t)src.perm[kk] : kk;
        const HitRay r = load_hit_ray<AOS>(src, k);
        float best;
        int32_t bi;
        bvh4_closest(r, bvh, stack, err, best, bi, COUNT ? &wc : nullptr);
        if (COUNT) ++rays;
        hit_idx[k] = bi;
        if (hit_t) hit_t[k] = best;
    });
    if (COUNT) flush_work(wc, rays);
}


// Few rays: a warp or eight lanes a ray (bvh4_group_loop).  Seven blocks share
// an SM at 72 registers, so that kGroupRays rays of eight lanes, 1,024 blocks,
// are one wave: 16,000 records on 81,922 triangles 45 us, 56 at six blocks.
template <bool AOS>
__global__ void __launch_bounds__(kBvhThreads, 7) hit_bvh4_group_kernel(RaySrc src, Bvh4View bvh,
                                                                     int32_t* __restrict__ hit_idx,
                                                                     float* __restrict__ hit_t, int32_t* err) {
    __shared__ int2 s_stack[kBvhThreads / 32][kGroupStackWarp];
    const int64_t n = src.d_count ? *src.d_count : src.n;
    if (n > kGroupRays) return;
    auto ray_of = [&](int64_t kk) { return src.perm ? (int64_t)src.perm[kk] : kk; };
    bvh4_groups(
        (int)n, src.fetch, s_stack[threadIdx.x >> 5], err,
        [&](int kk) { return load_hit_ray<AOS>(src, ray_of(kk)); }, bvh,
        [&](int kk, float best, int32_t bi) {
            const int64_t k = ray_of(kk);
            hit_idx[k] = bi;
            if (hit_t) hit_t[k] = best;
        });
}

// The per-ray form with finished lanes refilled from the work counter.
template <bool AOS>
__global__ void __launch_bounds__(kBvhThreads) hit_bvh4_refill_kernel(RaySrc src, Bvh4View bvh,
                                                                      int32_t* __restrict__ hit_idx,
                                                                      float* __restrict__ hit_t, int32_t* err,
                                                                      int refill_min) {
    const int64_t n = src.d_count ? *src.d_count : src.n;
    auto ray_of = [&](int64_t k) { return src.perm ? (int64_t)src.perm[k] : k; };
    bvh4_refill_loop(
        n, src.fetch, refill_min, err, [&](int64_t k) { return load_hit_ray<AOS>(src, ray_of(k)); },
        [&](int64_t) { return bvh; },
        [&](int64_t k, float best, int32_t bi) {
            const int64_t kk = ray_of(k);
            hit_idx[kk] = bi;
            if (hit_t) hit_t[kk] = best;
        });
}

// Packet form: each warp traverses its 32 rays together (bvh4_closest_packet)
// on a shared-memory stack.  ADAPT: per warp, packets only when its rays are
// coherent by packet_coherent's thresholds of `form` (2 loose, 3 tight);
// otherwise one ray per lane.  Rays are taken through src.perm when set, or,
// with src.tile_h set (a first bounce: the light grid's columns in order),
// in 8 x 4 tiles of the grid (grid_tile_ray), so a warp holds a compact
// patch of rays.
template <bool AOS, bool ADAPT, bool COUNT = false>
__global__ void __launch_bounds__(kBvhThreads) hit_bvh4_packet_kernel(RaySrc src, Bvh4View bvh,
                                                                      int32_t* __restrict__ hit_idx,
                                                                      float* __restrict__ hit_t, int32_t* err,
                                                                      int form) {
    WorkCount wc{0u, 0u, 0u};
    uint32_t rays = 0;
    __shared__ int2 s_stack[kBvhThreads / 32][kPacketStack];
    int2* stack = s_stack[threadIdx.x >> 5];
    const int64_t n = src.d_count ? *src.d_count : src.n;
    const int lane = threadIdx.x & 31;
    const float extent = ADAPT ? bvh4_extent(bvh.nodes) : 0.0f;
    int2 lane_stack[ADAPT ? kBvhStack : 1];
    for_each_warp_batch(n, src.fetch, [&](int64_t base) {
        const bool valid = base + lane < n;
        const int64_t kk = valid ? base + lane : base;
        int64_t k = src.perm ? (int64_t)src.perm[kk] : kk;
        if (!src.perm && src.tile_h > 0 && n < (int64_t(1) << 32))  // 8 x 4 tiles of the grid
            k = (int64_t)grid_tile_ray((uint32_t)kk, (uint32_t)src.tile_h, (uint32_t)n);
        const HitRay r = load_hit_ray<AOS>(src, k);
        float best;
        int32_t bi;
        const bool packet = !ADAPT || packet_coherent(r, form, extent);
        if (packet) {
            bvh4_closest_packet(r, valid, bvh, stack, err, best, bi, COUNT ? &wc : nullptr);
        } else if (ADAPT && valid) {
            bvh4_closest(r, bvh, lane_stack, err, best, bi, COUNT ? &wc : nullptr);
        }
        if (valid) {
            if (COUNT) ++rays;
            hit_idx[k] = bi;
            if (hit_t) hit_t[k] = best;
        }
    });
    if (COUNT) flush_work(wc, rays);
}

// The traversal kernels use no shared memory: give the whole L1/shared
// array to L1, where the upper BVH levels and hot hit records live.
template <class K>
static void prefer_l1(K kernel) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
}

template <bool COUNT>
static void launch_bvh4_form(const RaySrc& rays, int64_t cap, const Bvh4View& bvh, int32_t* hit_idx, float* hit_t,
                             int32_t* err, int sm_count, cudaStream_t s) {
    const int knob = g_tune[SPLAT_TUNE_BVH_BLOCKS_PER_SM];
    auto grid_of = [&](const void* k) {
        return rays.fetch ? resident_grid(k, cap, sm_count, kBvhThreads, knob) : grid_for(cap, kBvhThreads, sm_count, knob);
    };
    if (rays.packet) {
        // packet_form: 1 every warp; 2, 3 per warp by ray spread (loose, tight)
        const int form = rays.packet;
        if (form == 1) {
            const int grid = grid_of(reinterpret_cast<const void*>(hit_bvh4_packet_kernel<false, false, COUNT>));
            if (rays.aos)
                hit_bvh4_packet_kernel<true, false, COUNT><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t, err,
                                                                                       form);
            else
                hit_bvh4_packet_kernel<false, false, COUNT><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t,
                                                                                        err, form);
        } else {
            const int grid = grid_of(reinterpret_cast<const void*>(hit_bvh4_packet_kernel<false, true, COUNT>));
            if (rays.aos)
                hit_bvh4_packet_kernel<true, true, COUNT><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t, err,
                                                                                      form);
            else
                hit_bvh4_packet_kernel<false, true, COUNT><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t, err,
                                                                                       form);
        }
        return;
    }
    if (!COUNT && rays.fetch && g_tune[SPLAT_TUNE_BVH_REFILL] > 0) {
        const int grid = resident_grid(reinterpret_cast<const void*>(hit_bvh4_refill_kernel<false>), cap, sm_count,
                                       kBvhThreads, knob);
        const int m = g_tune[SPLAT_TUNE_BVH_REFILL];
        if (rays.aos)
            hit_bvh4_refill_kernel<true><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t, err, m);
        else
            hit_bvh4_refill_kernel<false><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t, err, m);
        return;
    }
    const int grid = rays.aos && !rays.fetch ? grid_for(cap, kBvhThreads, sm_count, kAosGrid * knob)
                                             : grid_of(reinterpret_cast<const void*>(hit_bvh4_kernel<false, COUNT>));
    if (rays.aos)
        hit_bvh4_kernel<true, COUNT><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t, err);
    else
        hit_bvh4_kernel<false, COUNT><<<grid, kBvhThreads, 0, s>>>(rays, bvh, hit_idx, hit_t, err);
}

cudaError_t launch_hit_bvh4(const RaySrc& rays, int64_t cap, const Bvh4View& bvh, int32_t* hit_idx, float* hit_t,
                            int32_t* err, int sm_count, cudaStream_t s) {
    if (cap <= 0) return cudaSuccess;
    static bool configured = false;
    if (!configured) {
        prefer_l1(hit_bvh4_kernel<true, false>);
        prefer_l1(hit_bvh4_kernel<false, false>);
        prefer_l1(hit_bvh4_kernel<true, true>);
        prefer_l1(hit_bvh4_kernel<false, true>);
        prefer_l1(hit_bvh4_refill_kernel<true>);
        prefer_l1(hit_bvh4_refill_kernel<false>);
        prefer_l1(hit_bvh_kernel<true>);
        prefer_l1(hit_bvh_kernel<false>);
        configured = true;
    }
    RaySrc src = rays;
    src.few = 0;  // set below where the group kernel is launched too
    if (g_tune[SPLAT_TUNE_COUNT_WORK]) {
        // the counting forms take every ray: the group kernel does not count
        launch_bvh4_form<true>(src, cap, bvh, hit_idx, hit_t, err, sm_count, s);
        ++g_launches;
        return cudaGetLastError();
    }
    // Few rays go to the group kernel.  Their number is known here when it is
    // the launch's bound; otherwise, where few are likely (few), both kernels
    // are launched and the count on the device picks the one that works.
    // Packet and refill forms that were asked for by their knobs stay.
    const bool groups = g_tune[SPLAT_TUNE_BVH_REFILL] == 0 && g_tune[SPLAT_TUNE_BVH_PACKET] <= 1;
    src.few = groups && rays.few && rays.packet == 0 ? 1 : 0;
    const bool only = groups && cap <= kGroupRays;
    if (only || src.few) {
        const int64_t lanes = cap <= kGroupWarpRays ? 32 * cap : std::max(32 * kGroupWarpRays, 8 * std::min(cap, kGroupRays));
        const int grid = resident_grid(reinterpret_cast<const void*>(hit_bvh4_group_kernel<false>), lanes, sm_count,
                                       kBvhThreads, 256);
        if (rays.aos)
            hit_bvh4_group_kernel<true><<<grid, kBvhThreads, 0, s>>>(src, bvh, hit_idx, hit_t, err);
        else
            hit_bvh4_group_kernel<false><<<grid, kBvhThreads, 0, s>>>(src, bvh, hit_idx, hit_t, err);
        ++g_launches;
        if (only) return cudaGetLastError();
    }
    launch_bvh4_form<false>(src, cap, bvh, hit_idx, hit_t, err, sm_count, s);
    ++g_launches;
    return cudaGetLastError();
}

cudaError_t read_hit_work(uint64_t out[4], bool reset, cudaStream_t s) {
    cudaError_t e = cudaMemcpyFromSymbolAsync(out, g_hit_work, 4 * sizeof(unsigned long long), 0,
                                              cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    if (reset) {
        static const unsigned long long zero[4] = {0ull, 0ull, 0ull, 0ull};
        if ((e = cudaMemcpyToSymbolAsync(g_hit_work, zero, sizeof(zero), 0, cudaMemcpyHostToDevice, s)) != cudaSuccess)
            return e;
        e = cudaStreamSynchronize(s);
    }
    return e;
}

// ---------------------------------------------------------------------------
// scene packing and BVH refit
// ---------------------------------------------------------------------------
// max |vertex coordinate| of the hit triangles (float bits; NaN skipped).
__global__ void scene_scale_kernel(const splat_ftri_t* __restrict__ ftri, int64_t n_tris, unsigned* scale) {
    unsigned m = 0u;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j + 1 < n_tris;
         j += (int64_t)gridDim.x * blockDim.x) {
        const float* p = ftri[j + 1].v[1];
        for (int v = 0; v < 9; ++v) {
            const float x = fabsf(p[v]);
            if (x == x) m = max(m, __float_as_uint(x));
        }
    }
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(scale, m);
}

__global__ void pack_hits_kernel(const splat_ftri_t* __restrict__ ftri, int64_t n_tris, TriHit* recs, TriBox* boxes,
                                 const unsigned* __restrict__ scale, const int32_t* __restrict__ order,
                                 int32_t* bvh_pos) {
    const float pad_abs = pad_abs_of_scale(__uint_as_float(*scale));
    const float inf = __int_as_float(0x7f800000);
    const int lane = threadIdx.x & 31;
    const BruteBoxes bb = brute_boxes_of(boxes, n_tris - 1);
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; base + 1 < n_tris;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = base + lane;
        float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
        if (j + 1 < n_tris) {
            const int32_t idx = order[j];  // every reference index but the sentinel's
            const float* p = ftri[idx - 1].v[0];
            recs[j] = pack_one(idx, f3(p), f3(p + 3), f3(p + 6), f3(p + 9));
            padded_box(p + 3, pad_abs, 1.0e-3f, lo, hi);
            boxes[j] = TriBox{make_float4(lo[0], lo[1], lo[2], 0.0f), make_float4(hi[0], hi[1], hi[2], 0.0f)};
            if (bvh_pos) bvh_pos[idx] = (int32_t)j;
        }
        merge_boxes(bb, j, j + 1 < n_tris, lo, hi);
    }
    if (bvh_pos && blockIdx.x == 0 && threadIdx.x == 0) {
        bvh_pos[0] = 0;
        bvh_pos[1] = 0;  // the sentinel
    }
}

cudaError_t launch_pack_hits(const splat_ftri_t* ftri, int64_t n_tris, TriHit* recs, TriBox* boxes, unsigned* scale,
                             const int32_t* order, int32_t* bvh_pos, cudaStream_t s) {
    if (n_tris <= 1) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(scale, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    scene_scale_kernel<<<grid_for(n_tris, 256, 152, 8), 256, 0, s>>>(ftri, n_tris, scale);
    pack_hits_kernel<<<grid_for(n_tris, 256, 152, 8), 256, 0, s>>>(ftri, n_tris, recs, boxes, scale, order, bvh_pos);
    g_launches += 2;
    return cudaGetLastError();
}

__device__ __forceinline__ void leaf_box(int ref, const TriHit* recs, const splat_ftri_t* ftri, const BvhFrame& fr,
                                         float pad_abs, float pad_rel, float lo[3], float hi[3]) {
    const int enc = ~ref;
    const int first = enc >> 4, count = (enc & 15) + 1;
    for (int j = 0; j < count; ++j) {
        const int32_t idx = __float_as_int(recs[first + j].a_idx.w);
        const float* q = ftri[idx - 1].v[1];
        float p[9];
        for (int v = 0; v < 9; ++v) p[v] = q[v];
        for (int v = 0; v < 3; ++v) to_frame(fr, p[3 * v], p[3 * v + 1], p[3 * v + 2]);
        float tl[3], th[3];
        for (int a = 0; a < 3; ++a) {
            tl[a] = fminf(fminf(p[a], p[3 + a]), p[6 + a]);
            th[a] = fmaxf(fmaxf(p[a], p[3 + a]), p[6 + a]);
        }
        const float dx = th[0] - tl[0], dy = th[1] - tl[1], dz = th[2] - tl[2];
        const float pad = pad_abs + pad_rel * sqrtf(dx * dx + dy * dy + dz * dz);
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], tl[a] - pad);
            hi[a] = fmaxf(hi[a], th[a] + pad);
        }
    }
}

// One-launch refit: the threads of the nodes whose children are all leaves
// start; each node's box union is written by the last of its inner children
// to finish (atomic arrival count against its number of inner children), so
// the tree is refit bottom-up without a launch per level.  links[q] =
// parent of node q (-1: root), links[n + q] = its number of inner children.
// Child nodes written by other threads are read through L2 (__ldcg).
__device__ __forceinline__ float4 ldcg4(const float4* p) { return __ldcg(p); }

__device__ __forceinline__ void refit2_node(BvhNode* nodes, int q, const TriHit* recs, const splat_ftri_t* ftri,
                                            const BvhFrame& fr, float pad_abs, float pad_rel) {
    const int4 c = nodes[q].c;
    float l[2][3], h[2][3];
    const int refs[2] = {c.x, c.y};
    for (int i = 0; i < 2; ++i) {
        for (int a = 0; a < 3; ++a) {
            l[i][a] = __int_as_float(0x7f800000);
            h[i][a] = -__int_as_float(0x7f800000);
        }
        if (refs[i] >= 0) {
            const float4 x = ldcg4(&nodes[refs[i]].x), y = ldcg4(&nodes[refs[i]].y), z = ldcg4(&nodes[refs[i]].z);
            l[i][0] = fminf(x.x, x.z);
            h[i][0] = fmaxf(x.y, x.w);
            l[i][1] = fminf(y.x, y.z);
            h[i][1] = fmaxf(y.y, y.w);
            l[i][2] = fminf(z.x, z.z);
            h[i][2] = fmaxf(z.y, z.w);
        } else {
            leaf_box(refs[i], recs, ftri, fr, pad_abs, pad_rel, l[i], h[i]);
        }
    }
    nodes[q].x = make_float4(l[0][0], h[0][0], l[1][0], h[1][0]);
    nodes[q].y = make_float4(l[0][1], h[0][1], l[1][1], h[1][1]);
    nodes[q].z = make_float4(l[0][2], h[0][2], l[1][2], h[1][2]);
}

__device__ __forceinline__ void refit4_node(Bvh4Node* nodes, int q, const TriHit* recs, const splat_ftri_t* ftri,
                                            const BvhFrame& fr, float pad_abs, float pad_rel) {
    const int nc = nodes[q].meta.x;
    const int4 c = nodes[q].c;
    const int refs[4] = {c.x, c.y, c.z, c.w};
    float lo[3][4], hi[3][4];
    for (int i = 0; i < 4; ++i) {
        float l[3] = {__int_as_float(0x7f800000), __int_as_float(0x7f800000), __int_as_float(0x7f800000)};
        float h[3] = {-l[0], -l[0], -l[0]};
        if (i < nc) {
            if (refs[i] >= 0) {
                const Bvh4Node* ch = nodes + refs[i];
                const float4 lx = ldcg4(&ch->lox), hx = ldcg4(&ch->hix), ly = ldcg4(&ch->loy), hy = ldcg4(&ch->hiy);
                const float4 lz = ldcg4(&ch->loz), hz = ldcg4(&ch->hiz);
                const int cn = __ldcg(&ch->meta.x);
                for (int j = 0; j < cn; ++j) {
                    l[0] = fminf(l[0], comp(lx, j));
                    h[0] = fmaxf(h[0], comp(hx, j));
                    l[1] = fminf(l[1], comp(ly, j));
                    h[1] = fmaxf(h[1], comp(hy, j));
                    l[2] = fminf(l[2], comp(lz, j));
                    h[2] = fmaxf(h[2], comp(hz, j));
                }
            } else {
                leaf_box(refs[i], recs, ftri, fr, pad_abs, pad_rel, l, h);
            }
        }
        for (int a = 0; a < 3; ++a) {
            lo[a][i] = l[a];
            hi[a][i] = h[a];
        }
    }
    Bvh4Node& nd = nodes[q];
    nd.lox = make_float4(lo[0][0], lo[0][1], lo[0][2], lo[0][3]);
    nd.hix = make_float4(hi[0][0], hi[0][1], hi[0][2], hi[0][3]);
    nd.loy = make_float4(lo[1][0], lo[1][1], lo[1][2], lo[1][3]);
    nd.hiy = make_float4(hi[1][0], hi[1][1], hi[1][2], hi[1][3]);
    nd.loz = make_float4(lo[2][0], lo[2][1], lo[2][2], lo[2][3]);
    nd.hiz = make_float4(hi[2][0], hi[2][1], hi[2][2], hi[2][3]);
}

template <bool WIDE, class Node>
__device__ __forceinline__ void refit_from(Node* nodes, int64_t n_nodes, int64_t q0, const int32_t* __restrict__ links,
                                           unsigned* flags, const TriHit* recs, const splat_ftri_t* ftri,
                                           const BvhFrame& fr, float pad_abs, float pad_rel) {
    if (links[n_nodes + q0] != 0) return;  // has inner children: reached by its last child
    int q = (int)q0;
    for (int64_t guard = 0; guard < n_nodes; ++guard) {
        if constexpr (WIDE) refit4_node(nodes, q, recs, ftri, fr, pad_abs, pad_rel);
        else refit2_node(nodes, q, recs, ftri, fr, pad_abs, pad_rel);
        const int p = links[q];
        if (p < 0) return;
        __threadfence();
        if ((int)atomicAdd(&flags[p], 1u) + 1 < links[n_nodes + p]) return;
        __threadfence();
        q = p;
    }
}

// Both trees in one launch, side by side: each climb waits on an atomic a
// level, so the two take as long as the deeper one (an update of the
// 96,012-triangle sponge: 157 -> 104 us).
__global__ void __launch_bounds__(128) refit_trees_kernel(RefitTrees t, const TriHit* __restrict__ recs,
                                                          const splat_ftri_t* __restrict__ ftri,
                                                          const unsigned* __restrict__ scale, float pad_rel) {
    const float pad_abs = pad_abs_of_scale(__uint_as_float(*scale));
    const BvhFrame fr = root_frame(t.nodes4);  // a refit writes no meta
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < t.n2 + t.n4;
         q += (int64_t)gridDim.x * blockDim.x) {
        if (q < t.n2)
            refit_from<false>(t.nodes2, t.n2, q, t.links2, t.flags, recs, ftri, fr, pad_abs, pad_rel);
        else
            refit_from<true>(t.nodes4, t.n4, q - t.n2, t.links4, t.flags + t.n2, recs, ftri, fr, pad_abs, pad_rel);
    }
}

cudaError_t launch_refit_trees(const RefitTrees& t, const TriHit* recs, const splat_ftri_t* ftri,
                               const unsigned* scale, float pad_rel, cudaStream_t s) {
    const int64_t n = t.n2 + t.n4;
    if (n <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(t.flags, 0, sizeof(unsigned) * (size_t)n, s);
    if (e != cudaSuccess) return e;
    refit_trees_kernel<<<grid_for(n, 128, 152, 16), 128, 0, s>>>(t, recs, ftri, scale, pad_rel);
    ++g_launches;
    return cudaGetLastError();
}

}  // namespace splat
