// evolve.cu -- evolve_ray over the active rays of one bounce, with the ray
// compaction (warp ballot + block scan, one atomic per block) fused in.  In
// trace mode the diffuse rays' final_evolution is fused in as well and the
// result is compacted into a splat queue for the splat launches.
//
// Reference: evolve_ray src/tracer.jl:181-201, partition! src/partition.jl
// (semantics: the active rays, in any order, and their count),
// final_evolution src/ray_imagers.jl:4-37, atomic_spectrum_kernel2
// src/ray_imagers.jl:78-113.  Each ray's Fresnel draw is keyed by its id, so
// results do not depend on the order compaction leaves the rays in.
//
// Splat: one lane per queued ray walks the ray's n_lambda x N x N samples.
// Fixed-point maps add round(intensity * 2^frac_bits) with integer atomics
// (runs of samples on one texel are summed in a register first), which makes
// the map independent of ray order and bit-exact run to run.  Float maps use
// plain float atomics, as the reference does.
#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "optics.cuh"

namespace splat {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kEvolveThreads = 256;

__device__ __forceinline__ void add_stats(splat_trace_stats_t* st, int diffuse, int samples) {
    if (!st) return;
    const int d = __reduce_add_sync(kFull, diffuse);
    const int s = __reduce_add_sync(kFull, samples);
    if (lane_id() == 0) {
        if (d) atomicAdd(reinterpret_cast<unsigned long long*>(&st->diffuse), (unsigned long long)d);
        if (s) atomicAdd(reinterpret_cast<unsigned long long*>(&st->samples), (unsigned long long)s);
    }
}

// TRACE: diffuse rays are final-evolved and splatted here, misses dropped, the
// last bounce skips the optics.  PLUGIN: retired rays are written back to the
// caller's AoS array with their status, as run_evolution! leaves them.
// MODE 0: plugin (retired rays written back to the caller's AoS array);
// 1: trace (diffuse rays final-evolved into the splat queue, escaped rays
// dropped); 2: camera (as trace, escaped rays queued unchanged for the sky).
// MK >= 0: the material kind, fixed at compile time so that only that
// material's optics is inlined (smaller code, no per-evaluation switch).
// PACKED: hits come as packed (t, index) words, and the survivors' words are
// reset for the next bounce.
template <int MODE, int MK, bool PACKED = false>
__global__ void __launch_bounds__(kEvolveThreads) evolve_kernel(EvolveArgs A) {
    constexpr bool TRACE = MODE != 0;
    constexpr bool SKY = MODE == 2;
    // double-buffered by iteration parity: iteration i + 2 writes a buffer
    // only after every thread has passed both barriers of iteration i + 1,
    // so no third barrier is needed at the end of an iteration
    __shared__ int s_warp2[2][kEvolveThreads / 32];
    __shared__ int s_wdif2[2][kEvolveThreads / 32];
    __shared__ int s_wsky2[2][kEvolveThreads / 32];
    __shared__ unsigned long long s_base2[2], s_dbase2[2], s_sbase2[2];
    const int64_t n = *A.in_count;
    const int lane = lane_id();
    const int wid = threadIdx.x >> 5;
    const bool quirks = A.quirks != 0;
    int par = 0;
    for (int64_t base = (int64_t)blockIdx.x * kEvolveThreads; base < n;
         base += (int64_t)gridDim.x * kEvolveThreads, par ^= 1) {
        int* s_warp = s_warp2[par];
        int* s_wdif = s_wdif2[par];
        int* s_wsky = s_wsky2[par];
        unsigned long long& s_base = s_base2[par];
        unsigned long long& s_dbase = s_dbase2[par];
        unsigned long long& s_sbase = s_sbase2[par];
        int64_t k = base + threadIdx.x;
        bool keep = false, dif = false, sky = false;
        RayState r, o;
        uint32_t id = 0;
        int32_t ih = 1;
        if (k < n) {
            if (A.tile_h > 0 && n < (int64_t(1) << 32))
                k = (int64_t)grid_tile_ray((uint32_t)k, (uint32_t)A.tile_h, (uint32_t)n);
            r = load_ray(A.in, k);
            id = A.in.id[k];
            EvolveView v{A.tris, A.n_tris, A.err, A.first_diffuse, A.material, A.seed, A.bounce,
                         A.force_rand, quirks, A.last != 0};
            if (MK >= 0) v.material.kind = MK;
            const int32_t hit = PACKED ? (int32_t)(uint32_t)A.hit_packed[k] : A.hit_idx[k];
            const int fate = evolve_one<TRACE>(r, hit, id, v, o, ih);
            keep = fate == kFateKeep;
            dif = fate == kFateDiffuse;
            sky = SKY && fate == kFateInfinity;
            if (!TRACE && fate != kFateKeep) {
                // the state written back is the one this hit was found for
                ray_to_aos(A.aos[id], r, fate == kFateDiffuse ? kStatusDiffuse : kStatusInfinity);
                A.aos_hit[id] = A.hit_idx[k];
            }
        }
        // compaction of the survivors (and, tracing, of the diffuse rays into
        // the splat queue and of the escaped ones into the sky queue): ballot
        // -> block scan -> one atomic per block and queue
        const unsigned kb = __ballot_sync(kFull, keep);
        const unsigned db = TRACE ? __ballot_sync(kFull, dif) : 0u;
        const unsigned sb = SKY ? __ballot_sync(kFull, sky) : 0u;
        if (lane == 0) {
            s_warp[wid] = __popc(kb);
            s_wdif[wid] = __popc(db);
            s_wsky[wid] = __popc(sb);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0, dtot = 0, stot = 0;
            for (int w = 0; w < kEvolveThreads / 32; ++w) {
                const int c = s_warp[w], d = s_wdif[w], e = s_wsky[w];
                s_warp[w] = tot;
                s_wdif[w] = dtot;
                s_wsky[w] = stot;
                tot += c;
                dtot += d;
                stot += e;
            }
            s_base = tot ? atomicAdd(reinterpret_cast<unsigned long long*>(A.out_count), (unsigned long long)tot) : 0ull;
            s_dbase = dtot ? atomicAdd(reinterpret_cast<unsigned long long*>(A.splat_count), (unsigned long long)dtot)
                           : 0ull;
            if (SKY)
                s_sbase = stot ? atomicAdd(reinterpret_cast<unsigned long long*>(A.sky_count), (unsigned long long)stot)
                               : 0ull;
        }
        __syncthreads();
        const unsigned below = (1u << lane) - 1u;
        if (keep) {
            const int64_t p = (int64_t)s_base + s_warp[wid] + __popc(kb & below);
            store_ray(A.out, p, o, id);
            if (PACKED) A.next_packed[p] = kNoHit;
        } else if (TRACE && dif) {
            store_ray(A.splat_q, (int64_t)s_dbase + s_wdif[wid] + __popc(db & below), o, id);
        } else if (SKY && sky) {
            store_ray(A.sky_q, (int64_t)s_sbase + s_wsky[wid] + __popc(sb & below), r, id);
        }
    }
}

// The two evolve kernels hold two blocks per SM, so the knob's default of 8 is
// halved to two full waves that go over the rays in turn; blocks beyond those
// start one by one as others end (2^18 rays through run_evolution 618 -> 608
// us, the Menger step of 2^22 7.04 -> 7.02 ms, others within 1 %).
static int evolve_grid_waves(int64_t cap, int sm_count) {
    int64_t b = (cap + kEvolveThreads - 1) / kEvolveThreads;
    const int64_t lim = (int64_t)sm_count * ((g_tune[SPLAT_TUNE_EVOLVE_BLOCKS_PER_SM] + 1) / 2);
    if (b > lim) b = lim;
    return (int)(b < 1 ? 1 : b);
}

static int evolve_grid(int64_t cap, int sm_count) {
    int64_t b = (cap + kEvolveThreads - 1) / kEvolveThreads;
    const int64_t lim = (int64_t)sm_count * g_tune[SPLAT_TUNE_EVOLVE_BLOCKS_PER_SM];
    if (b > lim) b = lim;
    return (int)(b < 1 ? 1 : b);
}

template <int MODE, bool PACKED = false>
static cudaError_t launch_evolve_mode(const EvolveArgs& a, int64_t cap, int sm_count, cudaStream_t s) {
    if (cap <= 0) return cudaSuccess;
    const int grid = evolve_grid_waves(cap, sm_count);
    switch (a.material.kind) {
        case SPLAT_MATERIAL_LINEAR_REF: evolve_kernel<MODE, SPLAT_MATERIAL_LINEAR_REF, PACKED><<<grid, kEvolveThreads, 0, s>>>(a); break;
        case SPLAT_MATERIAL_CAUCHY: evolve_kernel<MODE, SPLAT_MATERIAL_CAUCHY, PACKED><<<grid, kEvolveThreads, 0, s>>>(a); break;
        case SPLAT_MATERIAL_SELLMEIER: evolve_kernel<MODE, SPLAT_MATERIAL_SELLMEIER, PACKED><<<grid, kEvolveThreads, 0, s>>>(a); break;
        default: evolve_kernel<MODE, -1, PACKED><<<grid, kEvolveThreads, 0, s>>>(a); break;
    }
    ++g_launches;
    return cudaGetLastError();
}

cudaError_t launch_evolve_trace(const EvolveArgs& a, int64_t cap, int sm_count, cudaStream_t s) {
    return a.hit_packed ? launch_evolve_mode<1, true>(a, cap, sm_count, s) : launch_evolve_mode<1>(a, cap, sm_count, s);
}

cudaError_t launch_evolve_camera(const EvolveArgs& a, int64_t cap, int sm_count, cudaStream_t s) {
    return launch_evolve_mode<2>(a, cap, sm_count, s);
}

cudaError_t launch_evolve_plugin(const EvolveArgs& a, int64_t cap, int sm_count, cudaStream_t s) {
    return launch_evolve_mode<0>(a, cap, sm_count, s);
}

// A warp with at most this many records to change reads and writes those in
// place: moving all 32 for them is wasted traffic.  2^20 records, one evolve,
// us: 3 % active 118 all moved, 97 so; 10 % 130, 107; 20 % 129, 112; a third,
// the line, 129, 136.
constexpr int kSparseRecords = 12;

// evolve_ray broadcast (src/tracer.jl:181-201: `rays .= evolve_ray.(rays,
// hit_idx, tri_view, rndm, first_diffuse)`) on the caller's AoS rays: every
// ACTIVE ray evolves in place with its hit index and its Fresnel draw
// rndm[k] (the reference's rand! output; without an array, Philox(seed) at
// (k, 0, 1, bounce), or force_rand when >= 0); a ray that hits a diffuse
// triangle or nothing only changes status; other rays are untouched.
__global__ void __launch_bounds__(kEvolveThreads) evolve_aos_kernel(splat_adray_t* rays, int64_t n,
                                                                    const int32_t* __restrict__ hit_idx,
                                                                    const float* __restrict__ rndm, EvolveArgs A) {
    __shared__ AosTile s_tile[kEvolveThreads / 32];
    AosTile& tile = s_tile[threadIdx.x >> 5];
    const bool quirks = A.quirks != 0;
    const int lane = lane_id();
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = base + lane;
        // the status first: a warp of retired rays moves nothing
        const bool act = k < n && rays[k].status == kStatusActive;
        const unsigned m = __ballot_sync(kFull, act);
        if (m == 0) continue;
        const bool dense = __popc(m) > kSparseRecords;
        if (dense) aos_tile_load(tile, rays, base, n);
        if (act) {
            splat_adray_t& a = dense ? aos_tile_ray(tile) : rays[k];
            const RayState r = ray_from_aos(a);
            const EvolveView v{A.tris, A.n_tris, A.err, A.first_diffuse, A.material, A.seed, A.bounce,
                               rndm ? rndm[k] : A.force_rand, quirks, false};
            RayState o;
            int32_t ih;
            const int fate = evolve_one<false>(r, hit_idx[k], (uint32_t)k, v, o, ih);
            if (fate == kFateKeep) ray_to_aos(a, o, kStatusActive);
            else if (fate == kFateDiffuse) a.status = (uint8_t)kStatusDiffuse;
            else if (fate == kFateInfinity) a.status = (uint8_t)kStatusInfinity;
        }
        if (dense) aos_tile_store(tile, rays, base, n);
    }
}

cudaError_t launch_evolve_aos(splat_adray_t* rays, int64_t n, const int32_t* hit_idx, const float* rndm,
                              const EvolveArgs& a, int sm_count, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    evolve_aos_kernel<<<evolve_grid_waves(n, sm_count), kEvolveThreads, 0, s>>>(rays, n, hit_idx, rndm, a);
    ++g_launches;
    return cudaGetLastError();
}

// partition! (src/partition.jl:10-132): the ACTIVE rays first, in no
// particular order (the reference's blocks claim offsets atomically too).
// In place: with A active rays, every retired record below position A trades
// places with an active one at or above A, so only misplaced records move
// (a scatter into a second array and the copy back moved each record four
// times).  counts[0] = A, counts[1] = records to move up, counts[2] = to move
// down (equal); list: the positions of both, n entries each.  350,000 rays,
// a tenth of them retired: 71 us and a copy of the array -> 26 us (ncu, one
// GB300).
__global__ void __launch_bounds__(kEvolveThreads) partition_count_kernel(const splat_adray_t* __restrict__ rays,
                                                                         int64_t n, int64_t* counts) {
    int64_t mine = 0;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        mine += rays[k].status == kStatusActive ? 1 : 0;
    __shared__ int s_sum[kEvolveThreads / 32];
    const int w = __reduce_add_sync(kFull, (int)mine);
    if (lane_id() == 0) s_sum[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < kEvolveThreads / 32; ++i) t += (unsigned long long)s_sum[i];
        if (t) atomicAdd(reinterpret_cast<unsigned long long*>(&counts[0]), t);
    }
}

__global__ void __launch_bounds__(kEvolveThreads) partition_list_kernel(const splat_adray_t* __restrict__ rays,
                                                                        int64_t n, int64_t* counts, int64_t* list) {
    const int64_t n_active = counts[0];
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane_id(); base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = base + lane_id();
        const bool act = k < n && rays[k].status == kStatusActive;
        const bool hole = k < n_active && !act;        // n_active <= n
        const bool mover = act && k >= n_active;
        const unsigned below = (1u << lane_id()) - 1u;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const bool mine = side ? mover : hole;
            const unsigned m = __ballot_sync(kFull, mine);
            if (m == 0) continue;
            unsigned long long p = 0;
            if (lane_id() == 0)
                p = atomicAdd(reinterpret_cast<unsigned long long*>(&counts[1 + side]), (unsigned long long)__popc(m));
            p = __shfl_sync(kFull, p, 0);
            if (mine) list[side * n + (int64_t)p + __popc(m & below)] = k;
        }
    }
}

// Trades the j-th hole's record with the j-th mover's, one 8-byte word a
// thread; writes the result count.
__global__ void __launch_bounds__(kEvolveThreads) partition_swap_kernel(splat_adray_t* rays, int64_t n,
                                                                        const int64_t* __restrict__ counts,
                                                                        const int64_t* __restrict__ list,
                                                                        int64_t* d_n_active) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *d_n_active = counts[0];
    const int64_t words = counts[1] * kAosWords;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < words; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = t / kAosWords, w = t - j * kAosWords;
        uint64_t* a = reinterpret_cast<uint64_t*>(rays + list[j]) + w;
        uint64_t* b = reinterpret_cast<uint64_t*>(rays + list[n + j]) + w;
        const uint64_t x = *a, y = *b;
        *a = y;
        *b = x;
    }
}

cudaError_t launch_partition(splat_adray_t* rays, int64_t n, int64_t* counts, int64_t* list, int64_t* d_n_active,
                             int sm_count, cudaStream_t s) {
    if (n <= 0) return cudaMemsetAsync(d_n_active, 0, sizeof(int64_t), s);
    cudaError_t e = cudaMemsetAsync(counts, 0, 3 * sizeof(int64_t), s);
    if (e != cudaSuccess) return e;
    partition_count_kernel<<<evolve_grid(n, sm_count), kEvolveThreads, 0, s>>>(rays, n, counts);
    partition_list_kernel<<<evolve_grid(n, sm_count), kEvolveThreads, 0, s>>>(rays, n, counts, list);
    partition_swap_kernel<<<evolve_grid(n, sm_count), kEvolveThreads, 0, s>>>(rays, n, counts, list, d_n_active);
    g_launches += 3;
    return cudaGetLastError();
}

// go(N, ACCUM) with the splat's sample count, 1, 2 or 0 (any), and map type as
// compile-time constants.
template <class Go>
static void by_form(const SplatParams& sp, const Go& go) {
    auto typed = [&](auto nd) {
        if (sp.accum == SPLAT_ACCUM_I32)
            go(nd, std::integral_constant<int, SPLAT_ACCUM_I32>{});
        else
            go(nd, std::integral_constant<int, SPLAT_ACCUM_F32>{});
    };
    if (sp.n_delta == 2)
        typed(std::integral_constant<int, 2>{});
    else if (sp.n_delta == 1)
        typed(std::integral_constant<int, 1>{});
    else
        typed(std::integral_constant<int, 0>{});
}

// continuum_light_map2! on the caller's AoS rays: final_evolution in place,
// then the splat, one lane per diffuse ray walking all its planes as in
// splat_kernel.  The block's diffuse rays are compacted through shared memory
// between the two (their records' tile slots are reused: a ray's float planes
// and triangle index, 28 words of its 34), so warps splat with all lanes
// busy.  What it was bound by before: one ray at a time per warp, its 27
// values and triangle broadcast to the lanes that held its samples.  2^18
// rays, 12 planes, 2 x 2 offsets: 311.7 -> 137.6 us (ncu, one GB300).  A block
// of 128 for every 128 records, four at a time per SM: the whole frame of
// those rays takes 632 us with blocks of 256 that go over the records in two
// or more turns, and 617 so; 592 instead of 599 with a kernel per sample count
// and map type.  A block with few diffuse rays spreads each ray's planes over
// 2, 4, ... threads (2^20 records, 8 planes, 2 x 2: 1 % diffuse 166 -> 67 us,
// 10 % 216 -> 89, 35 % 228 -> 157), and a warp with few of them leaves the
// other records where they are (kSparseRecords).
constexpr int kMapThreads = 128;

template <int ND, int ACCUM>
__global__ void __launch_bounds__(kMapThreads, 4) light_map_kernel(splat_adray_t* rays, int64_t n,
                                                                   const int32_t* __restrict__ hit_idx,
                                                                   const splat_ftri_t* __restrict__ tris,
                                                                   int64_t n_tris, int32_t* err, SplatParams sp) {
    constexpr int kWarps = kMapThreads / 32;
    __shared__ AosTile s_tile[kWarps];
    __shared__ int s_cnt[kWarps];
    float* pool = reinterpret_cast<float*>(s_tile);  // [plane][kMapThreads], kPlanes + 1 planes
    static_assert(sizeof(s_tile) >= sizeof(float) * (kPlanes + 1) * kMapThreads, "pool fits the tiles");
    const int lane = lane_id(), wid = threadIdx.x >> 5;
    AosTile& tile = s_tile[wid];
    const DirectSink<SplatParams, ACCUM> sink{sp};
    const int planes = sp.n_lambda > 0 ? sp.n_lambda : 1;
    for (int64_t base = (int64_t)blockIdx.x * kMapThreads; base < n; base += (int64_t)gridDim.x * kMapThreads) {
        const int64_t wbase = base + 32 * wid, k = wbase + lane;
        bool dif = false;
        RayState o;
        int32_t ih = 1;
        const bool want = k < n && rays[k].status == kStatusDiffuse;
        const unsigned wm = __ballot_sync(kFull, want);
        if (wm) {
            const bool dense = __popc(wm) > kSparseRecords;
            if (dense) aos_tile_load(tile, rays, wbase, n);
            if (want) {
                const int32_t i = hit_idx[k];
                if (i >= 1 && i <= n_tris) {
                    splat_adray_t& a = dense ? aos_tile_ray(tile) : rays[k];
                    const RayState r = ray_from_aos(a);
                    const Tri T = load_tri(tris, i);
                    HitDerivs h;
                    ih = get_hit_ad(r, i, T, h);
                    final_evolution(r, h, ih, o);
                    ray_to_aos(a, o, kStatusDiffuse);
                    dif = true;
                } else {
                    atomicOr(err, 16);
                }
            }
            if (dense) aos_tile_store(tile, rays, wbase, n);
        }
        const unsigned db = __ballot_sync(kFull, dif);
        if (lane == 0) s_cnt[wid] = __popc(db);
        __syncthreads();  // every warp is done with its tile
        int before = 0, total = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const int c = s_cnt[w];
            before += w < wid ? c : 0;
            total += c;
        }
        const RaySoA q{pool, nullptr, nullptr, nullptr, kMapThreads};
        if (dif) {
            const int p = before + __popc(db & ((1u << lane) - 1u));
            st3(q.f, q.cap, 0, p, o.pos);
            st3(q.f, q.cap, 3, p, o.dir);
            st3(q.f, q.cap, 6, p, o.dpl);
            st3(q.f, q.cap, 9, p, o.dpx);
            st3(q.f, q.cap, 12, p, o.dpy);
            st3(q.f, q.cap, 15, p, o.ddl);
            st3(q.f, q.cap, 18, p, o.ddx);
            st3(q.f, q.cap, 21, p, o.ddy);
            q.f[24 * q.cap + p] = o.lam;
            q.f[25 * q.cap + p] = o.x;
            q.f[26 * q.cap + p] = o.y;
            q.f[27 * q.cap + p] = __int_as_float(ih);
        }
        __syncthreads();
        // few rays: 2, 4, ... threads a ray, each with every 2nd, 4th, ... plane
        int spread = 0;
        while (total << (spread + 1) <= kMapThreads && 1 << spread < planes) ++spread;
        const int p = threadIdx.x >> spread;
        if (p < total) {
            RayState s;
            s.pos = ld3(q.f, q.cap, 0, p);
            s.dir = ld3(q.f, q.cap, 3, p);
            s.dpl = ld3(q.f, q.cap, 6, p);
            s.dpx = ld3(q.f, q.cap, 9, p);
            s.dpy = ld3(q.f, q.cap, 12, p);
            s.ddl = ld3(q.f, q.cap, 15, p);
            s.ddx = ld3(q.f, q.cap, 18, p);
            s.ddy = ld3(q.f, q.cap, 21, p);
            s.lam = q.f[24 * q.cap + p];
            s.x = q.f[25 * q.cap + p];
            s.y = q.f[26 * q.cap + p];
            const Tri T = load_tri(tris, __float_as_int(q.f[27 * q.cap + p]));
            const TriUV quv = tri_uv(T);
            for (int il = threadIdx.x & ((1 << spread) - 1); il < planes; il += 1 << spread)
                (void)splat_ray_plane_n<ND>(sp, s, T, quv, il, sink);
        }
        __syncthreads();  // the tiles are free again
    }
}

cudaError_t launch_light_map(splat_adray_t* rays, int64_t n, const int32_t* hit_idx, const splat_ftri_t* tris,
                             int64_t n_tris, int32_t* err, const SplatParams& sp, int sm_count, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int64_t b = std::min<int64_t>((n + kMapThreads - 1) / kMapThreads, (int64_t)sm_count * 64);
    by_form(sp, [&](auto nd, auto accum) {
        light_map_kernel<decltype(nd)::value, decltype(accum)::value>
            <<<(int)b, kMapThreads, 0, s>>>(rays, n, hit_idx, tris, n_tris, err, sp);
    });
    ++g_launches;
    return cudaGetLastError();
}

// The step's counters into its statistics, by the last splat (rg.rays set):
// every bounce is done by then.  They accumulate: a step run as several ray
// ranges adds each range's counts into statistics cleared once.
__device__ __forceinline__ void splat_stats(const SplatRange& rg, splat_trace_stats_t* st) {
    if (!rg.rays || !st || blockIdx.x != 0) return;
    const int i = threadIdx.x;
    if (i < rg.depth)
        atomicAdd(reinterpret_cast<unsigned long long*>(&st->rays_per_bounce[i]), (unsigned long long)rg.rays[i]);
    else if (i == 8)
        atomicAdd(reinterpret_cast<unsigned long long*>(&st->diffuse), (unsigned long long)*rg.end);
    else if (i == 9 && *rg.err)
        atomicOr(reinterpret_cast<unsigned long long*>(&st->error), (unsigned long long)(uint32_t)*rg.err);
}

// Queued diffuse rays -> light map, one lane per ray walking all its planes
// (each plane's N x N sub-samples in the reference's order, x offset
// fastest; runs of samples on the same texel add in a register before one
// atomic).  Integer maps are bit-exact; float maps change only the order of
// additions, which float atomics never fix anyway.
// Instruction issue bounds it (splat_ray_plane_n).  96 registers at 20 warps
// per SM: 24 warps at 80 registers spill more, 16 at 128 hide less latency
// and made the step of 2^20 rays, 2 x 2 samples and 16 planes 2 % longer.  One
// kernel for each of 1 x 1, 2 x 2 and other samples and each map type leaves
// more registers to the one that runs: that step 1.263 -> 1.258 ms, the water
// surface 515 -> 511 us.
constexpr int kSplatThreads = 128;
template <int ND, int ACCUM>
__global__ void __launch_bounds__(kSplatThreads, 5) splat_kernel(RaySoA q, SplatRange rg,
                                                                 const splat_ftri_t* __restrict__ tris,
                                                                 SplatParams sp, splat_trace_stats_t* st) {
    const int64_t k0 = rg.begin ? *rg.begin : 0;
    const int64_t n = *rg.end;
    splat_stats(rg, st);
    const int planes = sp.n_lambda > 0 ? sp.n_lambda : 1;
    const DirectSink<SplatParams, ACCUM> sink{sp};
    int done = 0;
    for (int64_t k = k0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        const RayState r = load_ray(q, k);
        const Tri T = load_tri(tris, r.ignore);
        const TriUV quv = tri_uv(T);
        for (int il = 0; il < planes; ++il) done += splat_ray_plane_n<ND>(sp, r, T, quv, il, sink);
    }
    add_stats(st, 0, done);
}

// The same splat through the block's shared texel table: the block takes
// 256 queued rays at a time and, plane by plane, sums their samples per
// texel before one map atomic per distinct texel.
__global__ void __launch_bounds__(256, 2) splat_agg_kernel(RaySoA q, SplatRange rg,
                                                           const splat_ftri_t* __restrict__ tris, SplatParams sp,
                                                           splat_trace_stats_t* st) {
    __shared__ int32_t s_key[kAggSlots], s_val[kAggSlots];
    const int64_t k0 = rg.begin ? *rg.begin : 0;
    const int64_t n = *rg.end;
    splat_stats(rg, st);
    const int planes = sp.n_lambda > 0 ? sp.n_lambda : 1;
    const TableSink sink{sp, s_key, s_val};
    table_clear(s_key, s_val);
    __syncthreads();
    int done = 0;
    for (int64_t base = k0 + (int64_t)blockIdx.x * blockDim.x; base < n; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = base + threadIdx.x;
        const bool live = k < n;
        RayState r;
        Tri T;
        TriUV quv;
        if (live) {
            r = load_ray(q, k);
            T = load_tri(tris, r.ignore);
            quv = tri_uv(T);
        }
        for (int il = 0; il < planes; ++il) {
            if (live) done += splat_ray_plane(sp, r, T, quv, il, sink);
            __syncthreads();
            table_flush(sp, s_key, s_val);
            __syncthreads();
        }
    }
    add_stats(st, 0, done);
}

cudaError_t launch_splat(const RaySoA& q, const SplatRange& rg, const splat_ftri_t* tris, const SplatParams& sp,
                         splat_trace_stats_t* stats, int sm_count, cudaStream_t s) {
    if (q.cap <= 0) return cudaSuccess;
    const bool agg = g_tune[SPLAT_TUNE_SPLAT_AGGREGATE] != 0;
    const int threads = agg ? 256 : kSplatThreads;
    int64_t b = (q.cap + threads - 1) / threads;
    // the knob counts 160 threads a block for the one without a table: its
    // default of 8 is two full waves of 10 blocks of 128 (1.287 ms; 8 blocks
    // 1.299, 16 blocks 1.292, and 521, 521, 529 us for the water surface)
    int64_t lim = (int64_t)sm_count * g_tune[SPLAT_TUNE_SPLAT_BLOCKS_PER_SM];
    if (!agg) lim = lim * 160 / kSplatThreads;
    if (b > lim) b = lim;
    if (agg)
        splat_agg_kernel<<<(int)b, threads, 0, s>>>(q, rg, tris, sp, stats);
    else
        by_form(sp, [&](auto nd, auto accum) {
            splat_kernel<decltype(nd)::value, decltype(accum)::value>
                <<<(int)b, threads, 0, s>>>(q, rg, tris, sp, stats);
        });
    ++g_launches;
    return cudaGetLastError();
}

__global__ void copy_count_kernel(const int64_t* src, int64_t* dst) { *dst = *src; }

cudaError_t launch_copy_count(const int64_t* src, int64_t* dst, cudaStream_t s) {
    copy_count_kernel<<<1, 1, 0, s>>>(src, dst);
    ++g_launches;
    return cudaGetLastError();
}

// Also clears the step's n_counts counters, counts[0] the rays, and the packed
// hits of the first bounce (packed, optional).
__global__ void generate_soa_kernel(GenParams g, int64_t n, RaySoA out, int64_t* counts, int n_counts,
                                    unsigned long long* packed) {
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < n_counts; i += blockDim.x) counts[i] = i == 0 ? n : 0;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t kid = g.ray_begin + k;
        store_ray(out, k, gen_ray(g, kid), (uint32_t)kid);
        if (packed) packed[k] = kNoHit;
    }
}

__global__ void __launch_bounds__(256) generate_aos_kernel(GenParams g, int64_t n, splat_adray_t* out) {
    __shared__ AosTile s_tile[256 / 32];
    AosTile& tile = s_tile[threadIdx.x >> 5];
    const int lane = lane_id();
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = base + lane;
        if (k < n) {
            const RayState r = gen_ray(g, g.ray_begin + k);
            splat_adray_t a;
            memset(&a, 0, sizeof(a));
            ray_to_aos(a, r, kStatusActive);
            a.dest = 0;
            aos_tile_ray(tile) = a;
        }
        aos_tile_store(tile, out, base, n);
        __syncwarp();
    }
}

cudaError_t launch_generate_soa(const GenParams& g, int64_t n, RaySoA out, int64_t* counts, int n_counts,
                                uint64_t* packed, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    generate_soa_kernel<<<evolve_grid(n, 152), 256, 0, s>>>(g, n, out, counts, n_counts,
                                                            reinterpret_cast<unsigned long long*>(packed));
    ++g_launches;
    return cudaGetLastError();
}

cudaError_t launch_generate_aos(const GenParams& g, int64_t n, splat_adray_t* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    generate_aos_kernel<<<evolve_grid(n, 152), 256, 0, s>>>(g, n, out);
    ++g_launches;
    return cudaGetLastError();
}

// AoS rays -> SoA (id = slot), the active ones to out and the others to idle,
// compacted with one atomic per warp and target
__global__ void __launch_bounds__(256) aos_to_soa_kernel(const splat_adray_t* in, int64_t n, RaySoA out,
                                                         int64_t* d_count, RaySoA idle, int64_t* d_idle) {
    __shared__ AosTile s_tile[256 / 32];
    AosTile& tile = s_tile[threadIdx.x >> 5];
    const int lane = lane_id();
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = base + lane;
        aos_tile_load(tile, in, base, n);
        const splat_adray_t& a = aos_tile_ray(tile);
        const bool act = k < n && a.status == kStatusActive;
        const unsigned valid = __ballot_sync(kFull, k < n);
        const unsigned b = __ballot_sync(kFull, act);
        unsigned long long wbase = 0, ibase = 0;
        if (lane == 0 && b)
            wbase = atomicAdd(reinterpret_cast<unsigned long long*>(d_count), (unsigned long long)__popc(b));
        if (lane == 0 && b != valid)
            ibase = atomicAdd(reinterpret_cast<unsigned long long*>(d_idle), (unsigned long long)__popc(valid & ~b));
        wbase = __shfl_sync(kFull, wbase, 0);
        ibase = __shfl_sync(kFull, ibase, 0);
        const unsigned below = (1u << lane) - 1u;
        if (act)
            store_ray(out, (int64_t)wbase + __popc(b & below), ray_from_aos(a), (uint32_t)k);
        else if (k < n)
            store_ray(idle, (int64_t)ibase + __popc(valid & ~b & below), ray_from_aos(a), (uint32_t)k);
    }
}

__global__ void append_idle_kernel(RaySoA rays, const int64_t* d_count, RaySoA idle, const int64_t* d_idle,
                                   int64_t* d_total) {
    const int64_t m = *d_count, z = *d_idle;
    if (blockIdx.x == 0 && threadIdx.x == 0) *d_total = m + z;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < z; j += (int64_t)gridDim.x * blockDim.x) {
        st3(rays.f, rays.cap, 0, m + j, ld3(idle.f, idle.cap, 0, j));
        st3(rays.f, rays.cap, 3, m + j, ld3(idle.f, idle.cap, 3, j));
        rays.ignore[m + j] = idle.ignore[j];
        rays.id[m + j] = idle.id[j];
    }
}

__global__ void soa_to_aos_kernel(RaySoA in, const int64_t* d_count, const int64_t* d_total,
                                  const int32_t* __restrict__ hit, splat_adray_t* out, int32_t* hit_out, int status) {
    const int64_t m = *d_count, n = *d_total;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t id = in.id[k];
        hit_out[id] = hit[k];
        if (k < m) ray_to_aos(out[id], load_ray(in, k), status);
    }
}

cudaError_t launch_aos_to_soa(const splat_adray_t* in, int64_t n, RaySoA out, int64_t* d_count, RaySoA idle,
                              int64_t* d_idle, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    aos_to_soa_kernel<<<evolve_grid(n, 152), 256, 0, s>>>(in, n, out, d_count, idle, d_idle);
    ++g_launches;
    return cudaGetLastError();
}

cudaError_t launch_append_idle(RaySoA rays, const int64_t* d_count, RaySoA idle, const int64_t* d_idle,
                               int64_t* d_total, int sm_count, cudaStream_t s) {
    append_idle_kernel<<<sm_count, 256, 0, s>>>(rays, d_count, idle, d_idle, d_total);
    ++g_launches;
    return cudaGetLastError();
}

cudaError_t launch_soa_to_aos(RaySoA in, const int64_t* d_count, const int64_t* d_total, const int32_t* hit,
                              splat_adray_t* out, int32_t* hit_out, int status, cudaStream_t s) {
    if (in.cap <= 0) return cudaSuccess;
    soa_to_aos_kernel<<<evolve_grid(in.cap, 152), 256, 0, s>>>(in, d_count, d_total, hit, out, hit_out, status);
    ++g_launches;
    return cudaGetLastError();
}

}  // namespace splat
