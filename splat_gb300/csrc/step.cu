// step.cu -- a small trace step in one launch.
//
// A step of few rays is a chain of launches (generate, per bounce hit,
// evolve, splat, statistics) that each finish in less time than the next
// takes to start.  Here eight lanes take a ray from the light to its splat
// (src/tracer.jl:317-342): all eight evaluate the ray itself, they share the
// search for its hit (a BVH walk of eight entries a step, or the brute-force
// records dealt out), and they split its planes in the splat.  Nothing but
// the map and the statistics leaves the SM, and there is nothing to compact.
//
// What bounds it: the dependent chain of one ray, depth x (tree depth in
// node loads + evolve's arithmetic).  Eight-fold evaluation of the ray costs
// more than launches save once the rays fill the GPU; kSmallStepRays lies
// where the two forms meet.
#include "hitcore.cuh"
#include "optics.cuh"

namespace splat {

constexpr int kStepThreads = 64;
constexpr int kStepGroup = 8;

struct SmallStepArgs {
    GenParams gen;
    int64_t n;
    const Bvh4Node* nodes4;  // null: brute force
    const TriHit* recs;
    const TriBox* boxes;
    int64_t n_recs;
    const splat_ftri_t* tris;
    int64_t n_tris, first_diffuse;
    int32_t* err;
    splat_material_t material;
    float force_rand;
    int32_t quirks, depth;
    SplatParams sp;
    splat_trace_stats_t* stats;
};

template <int MK>
__global__ void __launch_bounds__(kStepThreads) small_step_kernel(const __grid_constant__ SmallStepArgs A) {
    constexpr int kWarps = kStepThreads / 32, kGroups = 32 / kStepGroup;
    __shared__ int2 s_stack[kWarps][kGroups * kGroupStack<kStepGroup>];
    __shared__ int s_rays[8], s_diffuse, s_samples;
    const int lane = threadIdx.x & 31, gl = lane & (kStepGroup - 1), wid = threadIdx.x >> 5;
    if (threadIdx.x < 8) s_rays[threadIdx.x] = 0;
    if (threadIdx.x == 8) s_diffuse = s_samples = 0;
    __syncthreads();
    int2* stack = s_stack[wid] + (lane / kStepGroup) * kGroupStack<kStepGroup>;
    const int64_t k = (int64_t)blockIdx.x * (kStepThreads / kStepGroup) + threadIdx.x / kStepGroup;
    const int64_t kid = A.gen.ray_begin + (k < A.n ? k : 0);
    RayState r = gen_ray(A.gen, kid);
    bool live = k < A.n;
    int diffuse = 0, samples = 0;
    for (int b = 1; b <= A.depth; ++b) {
        const unsigned rays = __ballot_sync(0xffffffffu, live && gl == 0);
        if (rays == 0) break;
        if (lane == 0) atomicAdd(&s_rays[b - 1], __popc(rays));
        const HitRay hr{r.pos.x, r.pos.y, r.pos.z, r.dir.x, r.dir.y, r.dir.z, r.ignore};
        float t;
        int32_t i;
        if (A.nodes4)
            bvh4_closest_group<kStepGroup>(hr, live, Bvh4View{A.nodes4, A.recs}, stack, A.err, t, i);
        else
            brute_closest_group<kStepGroup>(hr, live, A.recs, A.boxes, A.n_recs, t, i);
        if (live) {
            EvolveView v{A.tris, A.n_tris, A.err, A.first_diffuse, A.material, A.gen.seed, (uint32_t)b,
                         A.force_rand, A.quirks != 0, b == A.depth};
            v.material.kind = MK;
            RayState o;
            int32_t ih;
            const int fate = evolve_one<true>(r, i, (uint32_t)kid, v, o, ih);
            live = fate == kFateKeep;
            if (fate == kFateDiffuse) {
                const Tri T = load_tri(A.tris, o.ignore);
                const TriUV quv = tri_uv(T);
                const int planes = A.sp.n_lambda > 0 ? A.sp.n_lambda : 1;
                for (int il = gl; il < planes; il += kStepGroup)
                    samples += splat_ray_plane_n<0>(A.sp, o, T, quv, il, DirectSink<SplatParams>{A.sp});
                diffuse += gl == 0 ? 1 : 0;
            }
            r = o;
        }
    }
    diffuse = __reduce_add_sync(0xffffffffu, diffuse);
    samples = __reduce_add_sync(0xffffffffu, samples);
    if (lane == 0) {
        if (diffuse) atomicAdd(&s_diffuse, diffuse);
        if (samples) atomicAdd(&s_samples, samples);
    }
    __syncthreads();
    if (!A.stats) return;
    if (threadIdx.x < 8 && s_rays[threadIdx.x])
        atomicAdd(reinterpret_cast<unsigned long long*>(&A.stats->rays_per_bounce[threadIdx.x]),
                  (unsigned long long)s_rays[threadIdx.x]);
    if (threadIdx.x == 8 && s_diffuse)
        atomicAdd(reinterpret_cast<unsigned long long*>(&A.stats->diffuse), (unsigned long long)s_diffuse);
    if (threadIdx.x == 9 && s_samples)
        atomicAdd(reinterpret_cast<unsigned long long*>(&A.stats->samples), (unsigned long long)s_samples);
    if (threadIdx.x == 10) {
        // the scene's word as it stands: bits from before the step, and any
        // that a ray of this block set
        const int32_t e = atomicOr(A.err, 0);
        if (e) atomicOr(reinterpret_cast<unsigned long long*>(&A.stats->error), (unsigned long long)(uint32_t)e);
    }
}

cudaError_t launch_small_step(const GenParams& gen, int64_t n, const Bvh4Node* nodes4, const TriHit* recs,
                              const TriBox* boxes, int64_t n_recs, const EvolveArgs& ea, int32_t depth,
                              const SplatParams& sp, splat_trace_stats_t* stats, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    SmallStepArgs a;
    a.gen = gen;
    a.n = n;
    a.nodes4 = nodes4;
    a.recs = recs;
    a.boxes = boxes;
    a.n_recs = n_recs;
    a.tris = ea.tris;
    a.n_tris = ea.n_tris;
    a.first_diffuse = ea.first_diffuse;
    a.err = ea.err;
    a.material = ea.material;
    a.force_rand = ea.force_rand;
    a.quirks = ea.quirks;
    a.depth = depth;
    a.sp = sp;
    a.stats = stats;
    const int64_t per = kStepThreads / kStepGroup;
    const unsigned grid = (unsigned)((n + per - 1) / per);
    switch (a.material.kind) {
        case SPLAT_MATERIAL_CAUCHY: small_step_kernel<SPLAT_MATERIAL_CAUCHY><<<grid, kStepThreads, 0, s>>>(a); break;
        case SPLAT_MATERIAL_SELLMEIER:
            small_step_kernel<SPLAT_MATERIAL_SELLMEIER><<<grid, kStepThreads, 0, s>>>(a);
            break;
        default: small_step_kernel<SPLAT_MATERIAL_LINEAR_REF><<<grid, kStepThreads, 0, s>>>(a); break;
    }
    ++g_launches;
    return cudaGetLastError();
}

}  // namespace splat
