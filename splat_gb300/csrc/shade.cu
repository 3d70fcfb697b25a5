// shade.cu -- the camera pass: camera rays, and the light-map / skydome
// shading of the rays the bounce loop retires.
//
//   camera_ray     src/ray_generators.jl:18-50 (rays of one camera grid)
//   shade          shade_tex4_kernel, src/ray_imagers.jl:383-438: per ray and
//                  upscale^2 sub-sample, a diffuse ray sums retina-weighted
//                  light-map texels over the spectrum at its hit's uv, an
//                  escaped ray reads the skydome at its direction's polar
//                  angles; channels clamp to [0, 1]
//
// Textures are the reference's CuTexture objects: 3-D float arrays with
// hardware linear filtering, clamped addressing and unnormalised coordinates,
// sampled at (u, v, plane) - 0.5 (Julia's 1-based texel centres).
#include <cmath>
#include <type_traits>

#include "optics.cuh"

namespace splat {

// ---------------------------------------------------------------------------
// camera rays
// ---------------------------------------------------------------------------

// dir(x, y, dv) of camera_ray and its x / y derivatives.  The reference's
// pixel indices are integers, so the direction is evaluated in double (one
// ForwardDiff partial per pass) and rounded to float once:
//   scale = height cos45 / fov_half_sin, _x = (x - height/2) / scale,
//   _y = (y - width/2) / scale, _z = sqrt((1 - _x^2) - _y^2)
//   dir = ((_x right + _y up) + _z dir) + (dv 0.025f) / max(height, width)
// with d(_x^2) = (p 2) _x, p = 1 / scale, and d sqrt(a) = (1 / (2 sqrt a)) p.
//
// Double arithmetic is what bounds these kernels (about two lanes a clock and
// SM).  Everything of one row or one column is the same for the whole line of
// the grid: a block takes a tile of ROWS x kCamTile / ROWS rays, computes its
// rows' and columns' terms once into shared memory, and each ray is left with
// one square root, one division and 40 adds, products and roundings, where it
// had five divisions and twice as many: 230,400 rays 56 -> 35 us, 57,960
// records 23 -> 13.5 us.
// ROWS: 32, a warp's lanes being consecutive rays, for grids of more than 16
// rows; lower ones would leave lanes idle and take 8 rows, or one.  us for
// records of 1 x 100,000, 5 x 30,000, 9 x 20,000, 16 x 10,000 rays: without
// tiles 41, 49, 57, 61; by 32 rows 353, 120, 87, 55; by these 39, 47, 55, 40.
constexpr int kCamTile = 512;
constexpr int kCamThreads = 256;

struct CamRow {
    double a, p, r[3];  // 1 - _x^2, -((p 2) _x), _x right
};
struct CamCol {
    double b, p, u[3];  // _y^2, -((p 2) _y), _y up
};

// Camera rays of tile t (0-based ray g = x + h y, x and y 1-based in the
// formulas above); their jitter dv = three uniforms of Philox(seed) at
// (g, 0, 2, 0).  put(g, ray) for each; every thread of the block calls.
template <int ROWS, class Put>
__device__ __forceinline__ void camera_tile(const CameraParams& c, int64_t n, int64_t t, const Put& put) {
    constexpr int kCols = kCamTile / ROWS;
    __shared__ CamRow s_row[ROWS];
    __shared__ CamCol s_col[kCols];
    const int64_t tile_rows = (c.h + ROWS - 1) / ROWS;
    const int64_t x0 = t % tile_rows * ROWS, y0 = t / tile_rows * kCols;
    const int i = threadIdx.x;
    auto column = [&](int j) {
        const double vy = ((double)(y0 + j + 1) - (double)c.w / 2.0) / c.scale;
        CamCol& q = s_col[j];
        q.b = vy * vy;
        q.p = -((c.p * 2.0) * vy);
        for (int k = 0; k < 3; ++k) q.u[k] = vy * (double)c.cam.up[k];
    };
    if (i < ROWS) {
        const double vx = ((double)(x0 + i + 1) - (double)c.h / 2.0) / c.scale;
        CamRow& q = s_row[i];
        q.a = 1.0 - vx * vx;
        q.p = -((c.p * 2.0) * vx);
        for (int k = 0; k < 3; ++k) q.r[k] = vx * (double)c.cam.right[k];
    } else if (kCols <= kCamThreads - 32 && i >= 32 && i < 32 + kCols) {
        column(i - 32);
    }
    if (kCols > kCamThreads - 32)
        for (int j = i; j < kCols; j += kCamThreads) column(j);
    __syncthreads();
    const float m = (float)(c.h > c.w ? c.h : c.w);
    const int64_t x = x0 + i % ROWS;
    const CamRow& row = s_row[i % ROWS];
    if (x >= c.h) return;
    for (int j = i / ROWS; j < kCols; j += kCamThreads / ROWS) {
        const int64_t g = x + c.h * (y0 + j);
        if (g >= n) return;
        const CamCol& col = s_col[j];
        const double vz = sqrt(row.a - col.b);
        const double dsq = 1.0 / (2.0 * vz);
        const double pzx = row.p * dsq, pzy = col.p * dsq;
        const uint4 rnd = philox(make_uint4((uint32_t)g, 0u, 2u, 0u), (uint32_t)c.seed, (uint32_t)(c.seed >> 32));
        const float dv[3] = {(uniform24(rnd.x) * 0.025f) / m, (uniform24(rnd.y) * 0.025f) / m,
                             (uniform24(rnd.z) * 0.025f) / m};
        float o[3], ox[3], oy[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            o[k] = (float)(((row.r[k] + col.u[k]) + (vz * c.d[k])) + (double)dv[k]);
            ox[k] = (float)(c.pr[k] + (pzx * c.d[k]));
            oy[k] = (float)(c.pu[k] + (pzy * c.d[k]));
        }
        RayState r;
        r.pos = {c.cam.pos[0], c.cam.pos[1], c.cam.pos[2]};
        const F3 z = {0.0f, 0.0f, 0.0f};
        r.dpl = z;
        r.dpx = z;
        r.dpy = z;
        r.ddl = z;
        r.dir = {o[0], o[1], o[2]};
        r.ddx = {ox[0], ox[1], ox[2]};
        r.ddy = {oy[0], oy[1], oy[2]};
        r.lam = c.lambda;
        r.x = 0.0f;
        r.y = 0.0f;
        r.ignore = 1;
        r.medium = 0;
        put(g, r);
    }
}

template <int ROWS>
__global__ void __launch_bounds__(kCamThreads) camera_soa_kernel(CameraParams c, int64_t n, RaySoA out,
                                                                 int64_t* count) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = n;
    camera_tile<ROWS>(c, n, blockIdx.x, [&](int64_t g, const RayState& r) { store_ray(out, g, r, (uint32_t)g); });
}

template <int ROWS>
__global__ void __launch_bounds__(kCamThreads) camera_aos_kernel(CameraParams c, int64_t n, splat_adray_t* out) {
    camera_tile<ROWS>(c, n, blockIdx.x, [&](int64_t g, const RayState& r) {
        ray_to_aos(out[g], r, kStatusActive);
        out[g].dest = g + 1;
    });
}

// go(rows, tiles): the tile's rows as a constant, the tiles of the whole grid.
template <class Go>
static void by_camera_rows(const CameraParams& c, const Go& go) {
    auto with = [&](auto rows) {
        const int64_t r = decltype(rows)::value, cols = kCamTile / r;
        go(rows, (unsigned)(((c.h + r - 1) / r) * ((c.w + cols - 1) / cols)));
    };
    if (c.h > 16)
        with(std::integral_constant<int, 32>{});
    else if (c.h > 4)
        with(std::integral_constant<int, 8>{});
    else
        with(std::integral_constant<int, 1>{});
}

static int grid_for_rays(int64_t n, int threads, int sm_count, int per_sm) {
    int64_t b = (n + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count * per_sm;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

cudaError_t launch_camera_soa(const CameraParams& c, int64_t n, RaySoA out, int64_t* count, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    by_camera_rows(c, [&](auto rows, unsigned tiles) {
        camera_soa_kernel<decltype(rows)::value><<<tiles, kCamThreads, 0, s>>>(c, n, out, count);
    });
    ++g_launches;
    return cudaGetLastError();
}

cudaError_t launch_camera_aos(const CameraParams& c, int64_t n, splat_adray_t* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    by_camera_rows(c, [&](auto rows, unsigned tiles) {
        camera_aos_kernel<decltype(rows)::value><<<tiles, kCamThreads, 0, s>>>(c, n, out);
    });
    ++g_launches;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// shading
// ---------------------------------------------------------------------------

// Julia clamp(x, 0, 1): NaN passes through.
__device__ __forceinline__ float clamp01(float x) { return x > 1.0f ? 1.0f : (x < 0.0f ? 0.0f : x); }

__device__ __forceinline__ void put_pixel(const ShadeParams& p, int64_t ray, int i, int j, float R, float G, float B) {
    const int64_t gx = ray % p.cam_h, gy = ray / p.cam_h;
    const int64_t row = (int64_t)p.nd * gx + i, col = (int64_t)p.nd * gy + j;
    float* o = p.rgb + 3 * (row + p.height * col);
    o[0] = clamp01(R);
    o[1] = clamp01(G);
    o[2] = clamp01(B);
}

// Sub-sample (i, j) of a diffuse ray (final-evolved, ignore = its hit
// triangle): retina x texel summed over the spectrum.  tex_uv
// (src/geo.jl:222-229) of the expanded position; a NaN uv skips that
// wavelength.
__device__ __forceinline__ void shade_diffuse(const ShadeParams& p, const RayState& r, const Tri& T, const TriUV& q,
                                              int64_t ray, int i, int j) {
    const float Wf = (float)p.map_w, Hf = (float)p.map_h;
    const float xs = r.x + p.deltas[i];
    const float ys = r.y + p.deltas[j];
    float R = 0.0f, G = 0.0f, B = 0.0f;
#pragma unroll 4
    for (int il = 0; il < p.n_lambda; ++il) {
        const F3 pos = p_expansion(r, p.spectrum[il], xs, ys);
        const float bu = dot(q.N, cross(q.e1, pos - T.b)) / q.denom;
        const float bv = dot(q.N, cross(q.e2, pos - T.c)) / q.denom;
        const float bw = (1.0f - bu) - bv;
        const float U = (T.ta.x * bu + T.tb.x * bv) + T.tc.x * bw;
        const float V = (T.ta.y * bu + T.tb.y * bv) + T.tc.y * bw;
        // no branch around the fetch, so that four wavelengths' are in flight
        const bool ok = !(isnan(U) || isnan(V));
        const float X = tex3D<float>(p.map_tex, ok ? U * Wf - 0.5f : 0.0f, ok ? V * Hf - 0.5f : 0.0f,
                                     (float)(il + 1) - 0.5f);
        R = ok ? R + p.retina[0][il] * X : R;
        G = ok ? G + p.retina[1][il] * X : G;
        B = ok ? B + p.retina[2][il] * X : B;
    }
    put_pixel(p, ray, i, j, R, G, B);
}

// Sub-sample (i, j) of an escaped ray: the skydome at theta = acos(dir_z),
// phi = atan(dir_y, dir_x) of its expanded direction, u = theta / pi * sky_w,
// v = ((phi / pi) + 1) / 2 * sky_h.
__device__ __forceinline__ void shade_sky(const ShadeParams& p, const RayState& r, int64_t ray, int i, int j) {
    const float kPi = 3.14159265358979323846f;
    const float xs = r.x + p.deltas[i];
    const float ys = r.y + p.deltas[j];
    float R = 0.0f, G = 0.0f, B = 0.0f;
    if (p.has_sky) {
        const F3 d = d_expansion(r, r.lam, xs, ys);
        const float th = acosf(d.z);
        const float ph = atan2f(d.y, d.x);
        const float v = ((ph / kPi) + 1.0f) * 0.5f;
        const float u = th / kPi;
        const float us = u * (float)p.sky_w, vs = v * (float)p.sky_h;
        R = tex3D<float>(p.sky_tex, us - 0.5f, vs - 0.5f, 0.5f);
        G = tex3D<float>(p.sky_tex, us - 0.5f, vs - 0.5f, 1.5f);
        B = tex3D<float>(p.sky_tex, us - 0.5f, vs - 0.5f, 2.5f);
    }
    put_pixel(p, ray, i, j, R, G, B);
}

// Fused form: the diffuse queue (final-evolved) and the sky queue of the
// camera bounce loop, one lane per queued ray and sub-sample (blockIdx.y).
// Texture fetches and their latency bound the diffuse one: 230,400 rays at
// 2 x 2 sub-samples and 16 planes take 95 us a lane per ray with one fetch in
// flight, 66 with four, 53 with a lane per sub-sample.
__global__ void __launch_bounds__(256) shade_diffuse_kernel(RaySoA q, const int64_t* __restrict__ count,
                                                            const splat_ftri_t* __restrict__ tris, ShadeParams p) {
    const int64_t n = *count;
    const int i = blockIdx.y / p.nd, j = blockIdx.y % p.nd;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const RayState r = load_ray(q, k);
        const Tri T = load_tri(tris, r.ignore);
        shade_diffuse(p, r, T, tri_uv(T), (int64_t)q.id[k], i, j);
    }
}

__global__ void __launch_bounds__(256) shade_sky_kernel(RaySoA q, const int64_t* __restrict__ count, ShadeParams p) {
    const int64_t n = *count;
    const int i = blockIdx.y / p.nd, j = blockIdx.y % p.nd;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        shade_sky(p, load_ray(q, k), (int64_t)q.id[k], i, j);
}

// Plugin form (continuum_shade!): the caller's AoS rays in pixel order after
// run_evolution!; diffuse rays are final-evolved in place first.  A block
// takes 32 records through shared memory: its first warp evolves them, then
// each warp shades one sub-sample after another.  Latency bounds it (57,960
// rays are three warps a scheduler one ray a lane): 40 us one ray a lane on the
// records in place, 30 us through shared memory, 21 us so (8 planes, 2 x 2
// sub-samples).
constexpr int kShadeAosWarps = 4;

__global__ void __launch_bounds__(32 * kShadeAosWarps) shade_aos_kernel(splat_adray_t* rays, int64_t n,
                                                                        const int32_t* __restrict__ hit_idx,
                                                                        const splat_ftri_t* __restrict__ tris,
                                                                        int64_t n_tris, int32_t* err, ShadeParams p) {
    __shared__ AosTile tile;
    const int lane = lane_id(), wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (int64_t base = blockIdx.x * (int64_t)32; base < n; base += gridDim.x * (int64_t)32) {
        const int64_t k = base + lane;
        splat_adray_t& a = aos_tile_ray(tile);
        if (wid == 0) {
            aos_tile_load(tile, rays, base, n);
            const int32_t i = k < n && a.status == kStatusDiffuse ? hit_idx[k] : 0;
            const bool dif = i >= 1 && i <= n_tris;
            if (dif) {
                HitDerivs h;
                const RayState r = ray_from_aos(a);
                const Tri T = load_tri(tris, i);
                const int32_t ih = get_hit_ad(r, i, T, h);
                RayState o;
                final_evolution(r, h, ih, o);
                ray_to_aos(a, o, kStatusDiffuse);
            }
            if (__any_sync(0xffffffffu, dif)) aos_tile_store(tile, rays, base, n);
        }
        __syncthreads();
        if (k < n) {
            const int status = a.status;
            const int32_t i = status == kStatusDiffuse ? hit_idx[k] : 0;
            const bool dif = i >= 1 && i <= n_tris;
            if (status == kStatusDiffuse && !dif && wid == 0) atomicOr(err, 16);
            const RayState r = ray_from_aos(a);
            Tri T;
            TriUV q;
            if (dif) {
                T = load_tri(tris, i);  // tri_view[ray_index]: the hit_idx triangle
                q = tri_uv(T);
            }
            for (int s = wid; s < p.nd * p.nd; s += warps) {
                const int x = s / p.nd, y = s % p.nd;
                if (dif)
                    shade_diffuse(p, r, T, q, k, x, y);
                else if (status == kStatusInfinity)
                    shade_sky(p, r, k, x, y);
                else
                    put_pixel(p, k, x, y, 0.0f, 0.0f, 0.0f);
            }
        }
        __syncthreads();
    }
}

cudaError_t launch_shade_diffuse(const RaySoA& q, const int64_t* count, const splat_ftri_t* tris,
                                 const ShadeParams& p, int64_t cap, int sm_count, cudaStream_t s) {
    if (cap <= 0) return cudaSuccess;
    shade_diffuse_kernel<<<dim3(grid_for_rays(cap, 256, sm_count, 8), p.nd * p.nd), 256, 0, s>>>(q, count, tris, p);
    ++g_launches;
    return cudaGetLastError();
}

cudaError_t launch_shade_sky(const RaySoA& q, const int64_t* count, const ShadeParams& p, int64_t cap, int sm_count,
                             cudaStream_t s) {
    if (cap <= 0) return cudaSuccess;
    shade_sky_kernel<<<dim3(grid_for_rays(cap, 256, sm_count, 8), p.nd * p.nd), 256, 0, s>>>(q, count, p);
    ++g_launches;
    return cudaGetLastError();
}

cudaError_t launch_shade_aos(splat_adray_t* rays, int64_t n, const int32_t* hit_idx, const splat_ftri_t* tris,
                             int64_t n_tris, int32_t* err, const ShadeParams& p, int sm_count, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int warps = p.nd > 1 ? kShadeAosWarps : 1;
    shade_aos_kernel<<<grid_for_rays(n, 32, sm_count, 32), 32 * warps, 0, s>>>(rays, n, hit_idx, tris, n_tris, err, p);
    ++g_launches;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// light map -> texture array
// ---------------------------------------------------------------------------

// int32 fixed point -> float texels (value / 2^frac_bits) through a surface,
// VEC texels of a row a thread.  Bound by memory (4 bytes in, 4 out a texel);
// one texel a thread with its place by 64-bit divisions was bound by those
// (63 us for 1024 x 1024 x 16, 20 us now).
constexpr int kMapLanes = 16, kMapRows = 16;  // a block's patch: kMapLanes VEC texels x kMapRows rows

template <int VEC>
__global__ void __launch_bounds__(kMapLanes * kMapRows) map_to_array_kernel(const int32_t* __restrict__ map, int w,
                                                                            int h, float inv_scale,
                                                                            cudaSurfaceObject_t surf) {
    const int x = (blockIdx.x * kMapLanes + threadIdx.x) * VEC, z = blockIdx.z;
    if (x >= w) return;
    for (int y = blockIdx.y * kMapRows + threadIdx.y; y < h; y += gridDim.y * kMapRows) {
        const int32_t* p = map + ((int64_t)z * h + y) * w + x;
        if (VEC == 4) {
            const int4 v = __ldcs(reinterpret_cast<const int4*>(p));
            surf3Dwrite(make_float4(__int2float_rn(v.x) * inv_scale, __int2float_rn(v.y) * inv_scale,
                                    __int2float_rn(v.z) * inv_scale, __int2float_rn(v.w) * inv_scale),
                        surf, x * 4, y, z);
        } else {
            surf3Dwrite(__int2float_rn(*p) * inv_scale, surf, x * 4, y, z);
        }
    }
}

cudaError_t launch_map_to_array(const int32_t* map, int64_t w, int64_t h, int64_t planes, float inv_scale,
                                cudaSurfaceObject_t surf, cudaStream_t s) {
    if (w <= 0 || h <= 0 || planes <= 0) return cudaSuccess;
    const dim3 block(kMapLanes, kMapRows);
    // four texels a thread where every row starts on 16 bytes
    const bool vec = w % 4 == 0 && reinterpret_cast<uintptr_t>(map) % 16 == 0;
    const int64_t per = kMapLanes * (vec ? 4 : 1);
    const dim3 grid((unsigned)((w + per - 1) / per), (unsigned)((h + kMapRows - 1) / kMapRows), (unsigned)planes);
    if (vec)
        map_to_array_kernel<4><<<grid, block, 0, s>>>(map, (int)w, (int)h, inv_scale, surf);
    else
        map_to_array_kernel<1><<<grid, block, 0, s>>>(map, (int)w, (int)h, inv_scale, surf);
    ++g_launches;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// iterations of one frame: out = out (k - 1) / k + rgb / k
// (src/tracer.jl:380-384; the first iteration copies)
// ---------------------------------------------------------------------------
__global__ void image_accumulate_kernel(float* __restrict__ out, const float* __restrict__ rgb, int64_t n, int32_t k) {
    const float kf = (float)k, km = (float)(k - 1);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = k == 1 ? rgb[i] : (out[i] * km) / kf + rgb[i] / kf;
}

cudaError_t launch_image_accumulate(float* out, const float* rgb, int64_t n, int32_t k, int sm_count,
                                    cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    image_accumulate_kernel<<<grid_for_rays(n, 256, sm_count, 8), 256, 0, s>>>(out, rgb, n, k);
    ++g_launches;
    return cudaGetLastError();
}

}  // namespace splat
