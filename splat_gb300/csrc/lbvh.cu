// lbvh.cu -- BVH rebuild on the GPU for scenes whose geometry changes every
// frame (the reference rebuilds its bounding volumes on the host each frame,
// src/scenes/splash_scene.jl:41, src/bv.jl:68-121).
//
// A linear BVH: triangle centroids are quantised to 10 bits per axis and
// ordered by their Morton code (a stable least-significant-digit radix sort,
// 8 bits per pass); the binary radix tree over the sorted codes is built with
// one thread per inner node (Karras, "Maximizing Parallelism in the
// Construction of BVHs, Octrees, and k-d Trees", HPG 2012, codes made unique
// by appending the sorted position).  A node's box is that of a range of the
// sorted triangles, read off prefix and suffix boxes of runs of 32 and of
// 1,024 of them (RangeBoxes), so no pass climbs the tree.  Subtrees of at
// most `leaf_max` triangles become leaves (their triangles are contiguous in
// sorted order), and the tree is written in the traversal formats the host
// builder produces: two-child nodes and, for the inner nodes at even depth,
// four-wide nodes (each takes its children, or its grandchildren through an
// odd-depth inner child), both at the radix tree's own indices.  Boxes are padded exactly as the host builder pads
// them, so traversal results equal brute force bit for bit.
#include "hitcore.cuh"

namespace splat {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 4;
constexpr int kTile = kSortThreads * kSortItems;  // 1024 keys per tile

__host__ __device__ __forceinline__ int64_t n_tiles_of(int64_t n) { return (n + kTile - 1) / kTile; }

// -------------------------------------------------------------- scan (u32)
// In-place exclusive scan of a[0, m): tiles of 1024 scanned in shared memory,
// the tile sums scanned by one block, then added back.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
    __shared__ uint32_t warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (warp == 0) {
        uint32_t w = lane < nw ? warp_sum[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) warp_sum[lane] = w;
    }
    __syncthreads();
    const uint32_t before = warp ? warp_sum[warp - 1] : 0u;
    if (total) *total = warp_sum[nw - 1];
    __syncthreads();
    return before + x - v;
}

__global__ void scan_tiles_kernel(uint32_t* a, int64_t m, uint32_t* sums) {
    const int64_t base = (int64_t)blockIdx.x * kTile + (int64_t)threadIdx.x * kSortItems;
    uint32_t v[kSortItems];
    uint32_t s = 0;
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        v[j] = base + j < m ? a[base + j] : 0u;
        s += v[j];
    }
    uint32_t tot;
    uint32_t off = block_exclusive_scan(s, &tot);
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        if (base + j < m) a[base + j] = off;
        off += v[j];
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void scan_sums_kernel(uint32_t* sums, int64_t n) {
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int64_t base = 0; base < n; base += blockDim.x) {
        const int64_t i = base + threadIdx.x;
        const uint32_t v = i < n ? sums[i] : 0u;
        uint32_t tot;
        const uint32_t off = block_exclusive_scan(v, &tot);
        if (i < n) sums[i] = carry + off;
        __syncthreads();
        if (threadIdx.x == 0) carry += tot;
        __syncthreads();
    }
}

__global__ void scan_add_kernel(uint32_t* a, int64_t m, const uint32_t* sums) {
    const uint32_t add = sums[blockIdx.x];
    const int64_t base = (int64_t)blockIdx.x * kTile;
    for (int j = threadIdx.x; j < kTile; j += blockDim.x)
        if (base + j < m) a[base + j] += add;
}

cudaError_t scan_u32(uint32_t* a, int64_t m, uint32_t* sums, cudaStream_t s) {
    const int64_t tiles = n_tiles_of(m);
    scan_tiles_kernel<<<(unsigned)tiles, kSortThreads, 0, s>>>(a, m, sums);
    scan_sums_kernel<<<1, 1024, 0, s>>>(sums, tiles);
    scan_add_kernel<<<(unsigned)tiles, kSortThreads, 0, s>>>(a, m, sums);
    g_launches += 3;
    return cudaGetLastError();
}

// ------------------------------------------------------------ radix sort
// Digit histogram of one tile.  Up to kInlineTiles tiles it is stored tile by
// tile and the scatter blocks sum it up themselves; beyond, digit-major
// (hist[d * tiles + tile]), and an exclusive scan of the whole array makes it
// the place of the tile's first key with digit d.  (Three scan launches a
// pass were half of an 80,000-triangle sort; summing costs a block `tiles`
// rows of 1 KB.)
constexpr int64_t kInlineTiles = 256;

__device__ __forceinline__ void store_hist(uint32_t* hist, int64_t tiles, const uint32_t* cnt) {
    const int64_t d = threadIdx.x;
    hist[tiles <= kInlineTiles ? blockIdx.x * 256 + d : d * tiles + blockIdx.x] = cnt[d];
}

__global__ void radix_hist_kernel(const uint32_t* __restrict__ keys, int64_t n, int shift, uint32_t* hist,
                                  int64_t tiles) {
    __shared__ uint32_t cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kTile;
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const int64_t i = base + j * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    store_hist(hist, tiles, cnt);
}

// Stable scatter: a key's rank among the tile's keys with its digit is the
// count in the tile's earlier passes of the block, in earlier warps of this
// pass, and in earlier lanes of its warp (__match_any_sync peers).
__global__ void radix_scatter_kernel(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals, int64_t n,
                                     int shift, const uint32_t* __restrict__ hist, int64_t tiles, uint32_t* keys_out,
                                     uint32_t* vals_out) {
    __shared__ uint32_t s_run[256];  // where the digit's next key goes
    __shared__ __align__(16) uint32_t s_warp[kSortThreads / 32][256];
    static_assert(kSortThreads == 256, "the sums' four quarters of 64 threads");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        const int64_t d = threadIdx.x;
        uint32_t at = 0;
        if (tiles <= kInlineTiles) {
            // each quarter of the block sums every fourth tile, four digits a
            // thread, to have few loads in a row
            uint4 all = make_uint4(0u, 0u, 0u, 0u), before = all;
            const uint4* rows = reinterpret_cast<const uint4*>(hist);
            const int q = threadIdx.x >> 6, c4 = threadIdx.x & 63;
#pragma unroll 8
            for (int64_t t = q; t < tiles; t += 4) {
                const uint4 c = rows[t * 64 + c4];
                all.x += c.x;
                all.y += c.y;
                all.z += c.z;
                all.w += c.w;
                if (t < blockIdx.x) {
                    before.x += c.x;
                    before.y += c.y;
                    before.z += c.z;
                    before.w += c.w;
                }
            }
            reinterpret_cast<uint4*>(s_warp[q])[c4] = all;
            reinterpret_cast<uint4*>(s_warp[4 + q])[c4] = before;
            __syncthreads();
            const uint32_t a = (s_warp[0][d] + s_warp[1][d]) + (s_warp[2][d] + s_warp[3][d]);
            const uint32_t b = (s_warp[4][d] + s_warp[5][d]) + (s_warp[6][d] + s_warp[7][d]);
            at = block_exclusive_scan(a, nullptr) + b;
        } else {
            at = hist[d * tiles + blockIdx.x];
        }
        s_run[d] = at;
    }
    for (int w = 0; w < kSortThreads / 32; ++w) s_warp[w][threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kTile;
    const unsigned below = (1u << lane) - 1u;
    for (int j = 0; j < kSortItems; ++j) {
        const int64_t i = base + j * kSortThreads + threadIdx.x;
        const bool valid = i < n;
        const uint32_t key = valid ? keys[i] : 0u;
        const uint32_t d = valid ? (key >> shift) & 255u : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int rank = __popc(peers & below);
        if (valid && rank == 0) s_warp[warp][d] = (uint32_t)__popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t before = s_run[d];
            for (int w = 0; w < warp; ++w) before += s_warp[w][d];
            const uint32_t pos = before + (uint32_t)rank;
            keys_out[pos] = key;
            vals_out[pos] = vals[i];
        }
        __syncthreads();
        uint32_t add = 0;
        for (int w = 0; w < kSortThreads / 32; ++w) {
            add += s_warp[w][threadIdx.x];
            s_warp[w][threadIdx.x] = 0;
        }
        s_run[threadIdx.x] += add;
        __syncthreads();
    }
}

// --------------------------------------------------------- Morton codes
// bounds, all maxima over zeros: [0..2] complement of the centroid min, [3..5]
// centroid max (order-preserving u32), [6] max |vertex coordinate| (float
// bits, NaN skipped).
__device__ __forceinline__ float tri_centroid(const float* p, int a) {
    const float l = fminf(fminf(p[a], p[3 + a]), p[6 + a]);
    const float h = fmaxf(fmaxf(p[a], p[3 + a]), p[6 + a]);
    const float c = 0.5f * (l + h);
    return isfinite(c) ? c : 0.0f;
}

__global__ void __launch_bounds__(256) lbvh_bounds_kernel(const splat_ftri_t* __restrict__ ftri, int64_t np,
                                                          uint32_t* bounds) {
    uint32_t v[7] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < np; k += (int64_t)gridDim.x * blockDim.x) {
        const float* p = ftri[k + 1].v[1];
        for (int a = 0; a < 3; ++a) {
            const uint32_t u = monotonic_u32(tri_centroid(p, a));
            v[a] = max(v[a], ~u);
            v[3 + a] = max(v[3 + a], u);
        }
        for (int i = 0; i < 9; ++i) {
            const float x = fabsf(p[i]);
            if (x == x) v[6] = max(v[6], __float_as_uint(x));
        }
    }
    // one atomic a block and word (one a warp: 15 us for 80,000 triangles, of
    // which 10 in line at the seven words)
    __shared__ uint32_t s_v[8][7];
    for (int i = 0; i < 7; ++i) {
        const uint32_t w = __reduce_max_sync(0xffffffffu, v[i]);
        if ((threadIdx.x & 31) == 0) s_v[threadIdx.x >> 5][i] = w;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        uint32_t m = 0u;
        for (int w = 0; w < 8; ++w) m = max(m, s_v[w][threadIdx.x]);
        atomicMax(&bounds[threadIdx.x], m);
    }
}

__device__ __forceinline__ uint32_t spread10(uint32_t x) {
    x &= 0x3ffu;
    x = (x | (x << 16)) & 0x030000ffu;
    x = (x | (x << 8)) & 0x0300f00fu;
    x = (x | (x << 4)) & 0x030c30c3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// Codes of a tile's triangles and the histogram of their first digit.
__global__ void __launch_bounds__(kSortThreads) lbvh_morton_kernel(const splat_ftri_t* __restrict__ ftri, int64_t np,
                                                                   const uint32_t* bounds, uint32_t* keys,
                                                                   uint32_t* vals, uint32_t* hist, int64_t tiles) {
    __shared__ uint32_t cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    float lo[3], ext[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = monotonic_f32(~bounds[a]);
        ext[a] = monotonic_f32(bounds[3 + a]) - lo[a];
    }
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const int64_t k = (int64_t)blockIdx.x * kTile + j * kSortThreads + threadIdx.x;
        if (k >= np) continue;
        const float* p = ftri[k + 1].v[1];
        uint32_t q[3];
        for (int a = 0; a < 3; ++a) {
            const float f = ext[a] > 0.0f ? (tri_centroid(p, a) - lo[a]) / ext[a] : 0.5f;
            q[a] = (uint32_t)fminf(fmaxf(f * 1024.0f, 0.0f), 1023.0f);
        }
        const uint32_t key = (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]);
        keys[k] = key;
        vals[k] = (uint32_t)k;
        atomicAdd(&cnt[key & 255u], 1u);
    }
    __syncthreads();
    store_hist(hist, tiles, cnt);
}

// -------------------------------------------------------- range boxes
// Boxes over ranges of the sorted triangles, two levels deep: tab[j][k] is the
// box of triangles k .. k + 2^j - 1 (as far as their run of 32 goes; tab[0] the
// triangles' own padded boxes); pre1[k] / suf1[k] the box from the start of its
// run to k, and from k to the run's end; pre2 / suf2 the same over runs, within
// groups of 32 runs.  Minimum and maximum are idempotent: a range within a run
// is two boxes of the table, a longer one a suffix, what lies between, and a
// prefix.
struct RangeBoxes {
    TriBox *tab[5], *pre1, *suf1, *pre2, *suf2;
};

__device__ __forceinline__ TriBox empty_box() {
    const float inf = __int_as_float(0x7f800000);
    return TriBox{make_float4(inf, inf, inf, 0.f), make_float4(-inf, -inf, -inf, 0.f)};
}
__device__ __forceinline__ void grow(TriBox& b, const TriBox& o) {
    b.lo.x = fminf(b.lo.x, o.lo.x);
    b.lo.y = fminf(b.lo.y, o.lo.y);
    b.lo.z = fminf(b.lo.z, o.lo.z);
    b.hi.x = fmaxf(b.hi.x, o.hi.x);
    b.hi.y = fmaxf(b.hi.y, o.hi.y);
    b.hi.z = fmaxf(b.hi.z, o.hi.z);
}
template <bool UP>
__device__ __forceinline__ TriBox shifted(const TriBox& b, int o) {
    auto sh = [&](float x) {
        return UP ? __shfl_up_sync(0xffffffffu, x, o) : __shfl_down_sync(0xffffffffu, x, o);
    };
    return TriBox{make_float4(sh(b.lo.x), sh(b.lo.y), sh(b.lo.z), 0.f), make_float4(sh(b.hi.x), sh(b.hi.y), sh(b.hi.z), 0.f)};
}
// Inclusive prefix and suffix boxes over the warp's lanes.
__device__ __forceinline__ void warp_scan_boxes(const TriBox& b, TriBox& pre, TriBox& suf) {
    const int lane = threadIdx.x & 31;
    pre = suf = b;
    for (int o = 1; o < 32; o <<= 1) {
        const TriBox u = shifted<true>(pre, o), d = shifted<false>(suf, o);
        if (lane >= o) grow(pre, u);
        if (lane + o < 32) grow(suf, d);
    }
}

// Run r's prefix and suffix within its group (whole warps call).
__device__ __forceinline__ void range_boxes_level2(const RangeBoxes& rb, int64_t n, int64_t r) {
    const int64_t runs = (n + 31) / 32;
    const TriBox b = r < runs ? rb.pre1[min(32 * r + 31, n - 1)] : empty_box();
    TriBox pre, suf;
    warp_scan_boxes(b, pre, suf);
    if (r < runs) {
        rb.pre2[r] = pre;
        rb.suf2[r] = suf;
    }
}

// Box of sorted triangles f .. l.
__device__ __forceinline__ TriBox range_box(const RangeBoxes& rb, int32_t f, int32_t l) {
    TriBox b = empty_box();
    if (f >> 5 == l >> 5) {
        if ((f & 31) == 0) return rb.pre1[l];
        const int j = 31 - __clz(l - f + 1);  // at most 31 triangles: j <= 4
        b = rb.tab[j][f];
        grow(b, rb.tab[j][l + 1 - (1 << j)]);
        return b;
    }
    b = rb.suf1[f];
    grow(b, rb.pre1[l]);
    const int32_t r0 = (f >> 5) + 1, r1 = (l >> 5) - 1;  // whole runs between
    if (r0 > r1) return b;
    if (r0 >> 5 == r1 >> 5) {
        if ((r0 & 31) == 0) {
            grow(b, rb.pre2[r1]);
            return b;
        }
        for (int32_t r = r0; r <= r1; ++r) grow(b, rb.pre1[32 * r + 31]);
        return b;
    }
    grow(b, rb.suf2[r0]);
    grow(b, rb.pre2[r1]);
    for (int32_t g = (r0 >> 5) + 1; g < r1 >> 5; ++g) grow(b, rb.pre2[32 * g + 31]);
    return b;
}

// Everything of sorted triangle k that the tree's shape does not decide: its
// reference index, hit record and boxes (as pack_hits_kernel writes them),
// and the first level of the range boxes.
__global__ void __launch_bounds__(256) lbvh_leaves_kernel(const splat_ftri_t* __restrict__ ftri,
                                                          const uint32_t* __restrict__ vals, int64_t n,
                                                          const uint32_t* __restrict__ bounds, RangeBoxes rb,
                                                          int32_t* order, TriHit* recs, TriBox* boxes,
                                                          int32_t* bvh_pos, unsigned* scale) {
    const float pad_abs = pad_abs_of_scale(__uint_as_float(bounds[6]));
    const BruteBoxes bb = brute_boxes_of(boxes, n);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *scale = bounds[6];
        bvh_pos[0] = 0;
        bvh_pos[1] = 0;  // the sentinel
    }
    const int lane = threadIdx.x & 31;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = base + lane;
        const float inf = __int_as_float(0x7f800000);
        float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
        if (k < n) {
            const int32_t idx = (int32_t)vals[k] + 2;
            const float* p = ftri[idx - 1].v[0];
            order[k] = idx;
            bvh_pos[idx] = (int32_t)k;
            recs[k] = pack_one(idx, f3(p), f3(p + 3), f3(p + 6), f3(p + 9));
            padded_box(p + 3, pad_abs, 1.0e-3f, lo, hi);
        }
        const TriBox b{make_float4(lo[0], lo[1], lo[2], 0.0f), make_float4(hi[0], hi[1], hi[2], 0.0f)};
        TriBox pre, suf;
        warp_scan_boxes(b, pre, suf);
        TriBox w = b;
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            if (k < n) rb.tab[j][k] = w;
            const TriBox d = shifted<false>(w, 1 << j);
            if (lane + (1 << j) < 32) grow(w, d);
        }
        if (k < n) {
            boxes[k] = b;
            rb.pre1[k] = pre;
            rb.suf1[k] = suf;
        }
        merge_boxes(bb, k, k < n, lo, hi);
    }
}

// ------------------------------------------------------- radix tree
// delta(i, j): common prefix length of the unique 64-bit codes (code, position).
__device__ __forceinline__ int delta(const uint32_t* keys, int64_t n, int64_t i, int64_t j) {
    if (j < 0 || j >= n) return -1;
    const uint64_t a = ((uint64_t)keys[i] << 32) | (uint64_t)i;
    const uint64_t b = ((uint64_t)keys[j] << 32) | (uint64_t)j;
    return __clzll((long long)(a ^ b));
}

// Inner node i of n - 1: its key range [first, last], split and children
// (>= 0 inner node, < 0 leaf ~k for sorted triangle k), and the inner nodes'
// parents.  The first box_blocks blocks of the launch make the second level of
// the range boxes meanwhile.
__global__ void __launch_bounds__(256) lbvh_tree_kernel(const uint32_t* __restrict__ keys, int64_t n, int32_t* parent,
                                                        int32_t* lch, int32_t* rch, int32_t* first, int32_t* last,
                                                        RangeBoxes rb, unsigned box_blocks) {
    if (blockIdx.x < box_blocks) {
        range_boxes_level2(rb, n, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
        return;
    }
    for (int64_t i = (blockIdx.x - box_blocks) * (int64_t)blockDim.x + threadIdx.x; i < n - 1;
         i += (int64_t)(gridDim.x - box_blocks) * blockDim.x) {
        const int d = delta(keys, n, i, i + 1) > delta(keys, n, i, i - 1) ? 1 : -1;
        const int dmin = delta(keys, n, i, i - d);
        int64_t lmax = 2;
        while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
        int64_t l = 0;
        for (int64_t t = lmax >> 1; t >= 1; t >>= 1)
            if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
        const int64_t j = i + l * d;
        const int dnode = delta(keys, n, i, j);
        int64_t s = 0;
        for (int64_t div = 2;; div <<= 1) {
            const int64_t t = (l + div - 1) / div;
            if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
            if (t <= 1) break;
        }
        const int64_t g = i + s * d + (d < 0 ? -1 : 0);
        const int64_t lo = i < j ? i : j, hi = i < j ? j : i;
        const int32_t left = lo == g ? ~(int32_t)g : (int32_t)g;
        const int32_t right = hi == g + 1 ? ~(int32_t)(g + 1) : (int32_t)(g + 1);
        lch[i] = left;
        rch[i] = right;
        first[i] = (int32_t)lo;
        last[i] = (int32_t)hi;
        if (left >= 0) parent[left] = (int32_t)i;
        if (right >= 0) parent[right] = (int32_t)i;
        if (i == 0) parent[0] = -1;
    }
}

__device__ __forceinline__ int leaf_ref(int32_t first, int32_t count) { return ~((first << 4) | (count - 1)); }

struct LbvhView {
    const int32_t *lch, *rch, *first, *last, *parent;
    RangeBoxes rb;
    int64_t n;
    int leaf_max;
};

// A child of an inner node: its box, and whether it is folded into a leaf.
__device__ __forceinline__ TriBox child_box(const LbvhView& v, int32_t c) {
    return c >= 0 ? range_box(v.rb, v.first[c], v.last[c]) : v.rb.tab[0][~c];
}
__device__ __forceinline__ bool folded(const LbvhView& v, int32_t c) {
    return c < 0 || v.last[c] - v.first[c] + 1 <= v.leaf_max;
}
__device__ __forceinline__ int folded_ref(const LbvhView& v, int32_t c) {
    return c < 0 ? leaf_ref(~c, 1) : leaf_ref(v.first[c], v.last[c] - v.first[c] + 1);
}

// The kept inner nodes (not folded into a leaf) as two-child nodes, and those
// of them at even depth (parent hops to the root) as four-wide nodes.
__global__ void __launch_bounds__(256) lbvh_emit_kernel(LbvhView v, BvhNode* nodes2, Bvh4Node* nodes4) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < v.n - 1; i += (int64_t)gridDim.x * blockDim.x) {
        if (i != 0 && folded(v, (int32_t)i)) continue;
        const int32_t c[2] = {v.lch[i], v.rch[i]};
        const bool f[2] = {folded(v, c[0]), folded(v, c[1])};
        const TriBox b[2] = {child_box(v, c[0]), child_box(v, c[1])};
        BvhNode nd;
        nd.x = make_float4(b[0].lo.x, b[0].hi.x, b[1].lo.x, b[1].hi.x);
        nd.y = make_float4(b[0].lo.y, b[0].hi.y, b[1].lo.y, b[1].hi.y);
        nd.z = make_float4(b[0].lo.z, b[0].hi.z, b[1].lo.z, b[1].hi.z);
        nd.c = make_int4(f[0] ? folded_ref(v, c[0]) : c[0], f[1] ? folded_ref(v, c[1]) : c[1], 0, 0);
        nodes2[i] = nd;
        int d = 0;
        for (int32_t p = v.parent[i]; p >= 0 && d < v.n; p = v.parent[p]) ++d;
        if (d & 1) continue;
        // four-wide node: children, or grandchildren through an unfolded child
        TriBox q[4];
        int ref[4];
        int nc = 0;
        for (int a = 0; a < 2; ++a) {
            if (f[a]) {
                q[nc] = b[a];
                ref[nc++] = folded_ref(v, c[a]);
                continue;
            }
            const int32_t g[2] = {v.lch[c[a]], v.rch[c[a]]};
            for (int e = 0; e < 2; ++e) {
                q[nc] = child_box(v, g[e]);
                ref[nc++] = folded(v, g[e]) ? folded_ref(v, g[e]) : g[e];
            }
        }
        const float inf = __int_as_float(0x7f800000);
        for (int s = nc; s < 4; ++s) {  // empty slots: a box no ray enters
            q[s] = TriBox{make_float4(inf, inf, inf, 0.f), make_float4(-inf, -inf, -inf, 0.f)};
            ref[s] = ref[0];
        }
        Bvh4Node w;
        w.lox = make_float4(q[0].lo.x, q[1].lo.x, q[2].lo.x, q[3].lo.x);
        w.hix = make_float4(q[0].hi.x, q[1].hi.x, q[2].hi.x, q[3].hi.x);
        w.loy = make_float4(q[0].lo.y, q[1].lo.y, q[2].lo.y, q[3].lo.y);
        w.hiy = make_float4(q[0].hi.y, q[1].hi.y, q[2].hi.y, q[3].hi.y);
        w.loz = make_float4(q[0].lo.z, q[1].lo.z, q[2].lo.z, q[3].lo.z);
        w.hiz = make_float4(q[0].hi.z, q[1].hi.z, q[2].hi.z, q[3].hi.z);
        w.c = make_int4(ref[0], ref[1], ref[2], ref[3]);
        w.meta = make_int4(nc, 0, 0, 0);
        nodes4[i] = w;
    }
}

// A single triangle: both trees are a root whose two children are that leaf.
__global__ void lbvh_single_kernel(const TriBox* box, BvhNode* nodes2, Bvh4Node* nodes4) {
    const TriBox b = *box;
    BvhNode nd;
    nd.x = make_float4(b.lo.x, b.hi.x, b.lo.x, b.hi.x);
    nd.y = make_float4(b.lo.y, b.hi.y, b.lo.y, b.hi.y);
    nd.z = make_float4(b.lo.z, b.hi.z, b.lo.z, b.hi.z);
    nd.c = make_int4(leaf_ref(0, 1), leaf_ref(0, 1), 0, 0);
    nodes2[0] = nd;
    const float inf = __int_as_float(0x7f800000);  // slots 2 and 3 empty
    Bvh4Node q;
    q.lox = make_float4(b.lo.x, b.lo.x, inf, inf);
    q.hix = make_float4(b.hi.x, b.hi.x, -inf, -inf);
    q.loy = make_float4(b.lo.y, b.lo.y, inf, inf);
    q.hiy = make_float4(b.hi.y, b.hi.y, -inf, -inf);
    q.loz = make_float4(b.lo.z, b.lo.z, inf, inf);
    q.hiz = make_float4(b.hi.z, b.hi.z, -inf, -inf);
    q.c = make_int4(leaf_ref(0, 1), leaf_ref(0, 1), leaf_ref(0, 1), leaf_ref(0, 1));
    q.meta = make_int4(2, 0, 0, 0);
    nodes4[0] = q;
}

struct Carve {
    char* p;
    template <class T>
    T* take(int64_t count) {
        T* r = reinterpret_cast<T*>(p);
        p += ((size_t)count * sizeof(T) + 255) / 256 * 256;
        return r;
    }
};

}  // namespace

namespace {
struct LbvhScratch {
    uint32_t *keys[2], *vals[2], *hist, *sums, *bounds;
    int32_t *parent, *lch, *rch, *first, *last;
    RangeBoxes rb;
    size_t bytes;
};
LbvhScratch carve_lbvh(void* scratch, int64_t n) {
    const int64_t inner = n > 1 ? n - 1 : 1, m_hist = 256 * n_tiles_of(n), runs = (n + 31) / 32;
    char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(scratch) + 255) / 256 * 256);
    Carve c{base};
    LbvhScratch w;
    for (int i = 0; i < 2; ++i) {
        w.keys[i] = c.take<uint32_t>(n);
        w.vals[i] = c.take<uint32_t>(n);
    }
    w.hist = c.take<uint32_t>(m_hist);
    w.sums = c.take<uint32_t>(n_tiles_of(m_hist));
    w.bounds = c.take<uint32_t>(8);
    w.parent = c.take<int32_t>(inner);
    w.lch = c.take<int32_t>(inner);
    w.rch = c.take<int32_t>(inner);
    w.first = c.take<int32_t>(inner);
    w.last = c.take<int32_t>(inner);
    for (int j = 0; j < 5; ++j) w.rb.tab[j] = c.take<TriBox>(n);
    w.rb.pre1 = c.take<TriBox>(n);
    w.rb.suf1 = c.take<TriBox>(n);
    w.rb.pre2 = c.take<TriBox>(runs);
    w.rb.suf2 = c.take<TriBox>(runs);
    w.bytes = (size_t)(c.p - base) + 256;
    return w;
}
}  // namespace

size_t lbvh_scratch_bytes(int64_t np) { return np < 1 ? 256 : carve_lbvh(nullptr, np).bytes; }

// 80,000 triangles: 33 launches, 250 us a rebuild -> 13 launches, 132 us;
// 3,200: 202 -> 91; 320,000: 428 -> 282; 4,000,000: 2.58 -> 2.22 ms;
// 10,000,000, where a node near the root goes over up to 9,766 groups of 1,024
// in turn (range_box): 7.6 -> 5.7 ms (one GB300).  Before, three scan launches a sort pass, a climb of the tree
// for its boxes that waited on an atomic a level (52 us), and passes of their
// own for depths, node numbering, records and boxes.
cudaError_t launch_lbvh_build(const splat_ftri_t* ftri, int64_t n_tris, int leaf_max, void* scratch,
                              const LbvhOut& out, int sm_count, cudaStream_t s) {
    const int64_t n = n_tris - 1;  // the sentinel (index 1) is never hit
    if (n < 1) return cudaSuccess;
    const LbvhScratch w = carve_lbvh(scratch, n);
    const int64_t tiles = n_tiles_of(n);
    auto grid = [&](int64_t items) {
        int64_t b = (items + 255) / 256;
        const int64_t cap = (int64_t)sm_count * 8;
        return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
    };
    cudaError_t e = cudaMemsetAsync(w.bounds, 0, 8 * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    lbvh_bounds_kernel<<<grid(n), 256, 0, s>>>(ftri, n, w.bounds);
    lbvh_morton_kernel<<<(unsigned)tiles, kSortThreads, 0, s>>>(ftri, n, w.bounds, w.keys[0], w.vals[0], w.hist, tiles);
    g_launches += 2;
    int cur = 0;
    for (int shift = 0; shift < 32; shift += 8) {
        if (shift > 0) {
            radix_hist_kernel<<<(unsigned)tiles, kSortThreads, 0, s>>>(w.keys[cur], n, shift, w.hist, tiles);
            ++g_launches;
        }
        if (tiles > kInlineTiles && (e = scan_u32(w.hist, 256 * tiles, w.sums, s)) != cudaSuccess) return e;
        radix_scatter_kernel<<<(unsigned)tiles, kSortThreads, 0, s>>>(w.keys[cur], w.vals[cur], n, shift, w.hist, tiles,
                                                                      w.keys[cur ^ 1], w.vals[cur ^ 1]);
        ++g_launches;
        cur ^= 1;
    }
    lbvh_leaves_kernel<<<grid(n), 256, 0, s>>>(ftri, w.vals[cur], n, w.bounds, w.rb, out.order, out.recs, out.boxes,
                                               out.bvh_pos, out.scale);
    ++g_launches;
    if (n == 1) {
        lbvh_single_kernel<<<1, 1, 0, s>>>(w.rb.tab[0], out.nodes2, out.nodes4);
        ++g_launches;
        return cudaGetLastError();
    }
    const unsigned box_blocks = (unsigned)(((n + 31) / 32 + 255) / 256);
    lbvh_tree_kernel<<<box_blocks + grid(n - 1), 256, 0, s>>>(w.keys[cur], n, w.parent, w.lch, w.rch, w.first, w.last,
                                                              w.rb, box_blocks);
    const LbvhView v{w.lch, w.rch, w.first, w.last, w.parent, w.rb, n, leaf_max};
    lbvh_emit_kernel<<<grid(n - 1), 256, 0, s>>>(v, out.nodes2, out.nodes4);
    g_launches += 2;
    return cudaGetLastError();
}

// ---------------------------------------------------------- ray order
// A counting sort of the active rays by key: the direction octant above the
// BVH-order position of the triangle the ray leaves (ignore_tri), the
// position's low bits dropped so that the key has key_bits bits.  Bucket
// sizes are counted with global atomics, scanned into offsets, and every ray
// takes a slot in its bucket with one atomic per group of equal keys in a
// warp (__match_any_sync), so a warp's rays of one bucket stay together.
// The order inside a bucket is the atomics' order: only which rays share a
// warp changes with it, never a result.
constexpr int kOrderMaxBits = 22;
constexpr int kDirClasses = 8, kDirBits = 3;  // direction octants

__device__ __forceinline__ uint32_t ray_key(const float* __restrict__ f, int64_t cap, const int32_t* __restrict__ ignore,
                                            const int32_t* __restrict__ bvh_pos, int64_t n_tris, int pos_shift,
                                            uint32_t n_pos, int64_t k) {
    const uint32_t cls = (f[3 * cap + k] < 0.0f ? 1u : 0u) | (f[4 * cap + k] < 0.0f ? 2u : 0u) |
                         (f[5 * cap + k] < 0.0f ? 4u : 0u);
    const int32_t ig = ignore[k];
    const uint32_t pos = (ig >= 1 && (int64_t)ig <= n_tris) ? (uint32_t)bvh_pos[ig] : 0u;
    return cls * n_pos + (pos >> pos_shift);
}

// Bucket sizes: one atomic per group of equal keys in a warp.
__global__ void ray_bucket_count_kernel(const float* __restrict__ f, int64_t cap, const int32_t* __restrict__ ignore,
                                        const int64_t* __restrict__ d_count, const int32_t* __restrict__ bvh_pos,
                                        int64_t n_tris, int pos_shift, uint32_t n_pos, uint32_t* keys,
                                        uint32_t* cnt) {
    const int64_t n = min(cap, *d_count);
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; base < n; base += stride) {
        const int64_t k = base + lane;
        const bool valid = k < n;
        const uint32_t key = valid ? ray_key(f, cap, ignore, bvh_pos, n_tris, pos_shift, n_pos, k) : 0xffffffffu;
        if (valid) keys[k] = key;
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        if (valid && lane == __ffs(peers) - 1) atomicAdd(&cnt[key], (uint32_t)__popc(peers));
    }
}

__global__ void ray_bucket_place_kernel(const uint32_t* __restrict__ keys, int64_t cap,
                                        const int64_t* __restrict__ d_count, uint32_t* off, int32_t* perm) {
    const int64_t n = min(cap, *d_count);
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // warp-uniform trip count: every lane takes part in the vote
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; base < n; base += stride) {
        const int64_t k = base + lane;
        const bool valid = k < n;
        const uint32_t key = valid ? keys[k] : 0xffffffffu;
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(peers) - 1;
        uint32_t slot = 0;
        if (valid && lane == leader) slot = atomicAdd(&off[key], (uint32_t)__popc(peers));
        slot = __shfl_sync(0xffffffffu, slot, leader);
        if (valid) perm[slot + (uint32_t)__popc(peers & below)] = (int32_t)k;
    }
}

size_t ray_order_bytes(int64_t cap) {
    if (cap < 1) return 256;
    const int64_t buckets = int64_t(1) << kOrderMaxBits;
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    return 256 + 2 * al(4 * (size_t)cap) + al(4 * (size_t)buckets) + al(4 * (size_t)n_tiles_of(buckets));
}

cudaError_t launch_ray_order(const float* soa_f, const int32_t* ignore, int64_t cap, const int64_t* d_count,
                             const int32_t* bvh_pos, int64_t n_tris, int key_bits, void* scratch,
                             const int32_t** perm_out, int sm_count, cudaStream_t s) {
    if (cap < 1) return cudaSuccess;
    if (key_bits < 4) key_bits = 4;
    if (key_bits > kOrderMaxBits) key_bits = kOrderMaxBits;
    Carve c{reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(scratch) + 255) / 256 * 256)};
    uint32_t* keys = c.take<uint32_t>(cap);
    int32_t* perm = c.take<int32_t>(cap);
    uint32_t* cnt = c.take<uint32_t>(int64_t(1) << kOrderMaxBits);
    uint32_t* sums = c.take<uint32_t>(n_tiles_of(int64_t(1) << kOrderMaxBits));
    // positions 0 .. n_tris - 2 (the records); keep the high bits that fit
    int full_bits = 1;
    while (full_bits < 31 && (int64_t(1) << full_bits) < n_tris + 1) ++full_bits;
    const int pos_bits = full_bits < key_bits - kDirBits ? full_bits : key_bits - kDirBits;
    const int pos_shift = full_bits - pos_bits;
    const uint32_t n_pos = (uint32_t)((n_tris >> pos_shift) + 1);  // positions after the shift, all < n_pos
    const int64_t buckets = kDirClasses * (int64_t)n_pos;           // <= 2^key_bits
    int64_t b = (cap + 255) / 256;
    if (b > (int64_t)sm_count * 8) b = (int64_t)sm_count * 8;
    if (b < 1) b = 1;
    cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * (size_t)buckets, s);
    if (e != cudaSuccess) return e;
    ray_bucket_count_kernel<<<(unsigned)b, 256, 0, s>>>(soa_f, cap, ignore, d_count, bvh_pos, n_tris, pos_shift,
                                                        n_pos, keys, cnt);
    ++g_launches;
    if ((e = scan_u32(cnt, buckets, sums, s)) != cudaSuccess) return e;
    // one block per 256 rays (blocks start in index order), so a bucket's
    // slots go to its rays nearly in position order: the input order carries
    // the first bounce's tiles
    const int64_t bp = (cap + 255) / 256;
    ray_bucket_place_kernel<<<(unsigned)(bp < 1 ? 1 : bp), 256, 0, s>>>(keys, cap, d_count, cnt, perm);
    ++g_launches;
    *perm_out = perm;
    return cudaGetLastError();
}

size_t order_sums_count(int64_t buckets) { return (size_t)n_tiles_of(buckets < 1 ? 1 : buckets); }

cudaError_t launch_order_scan(uint32_t* cnt, int64_t buckets, uint32_t* sums, cudaStream_t s) {
    if (buckets < 1) return cudaSuccess;
    return scan_u32(cnt, buckets, sums, s);
}

}  // namespace splat
