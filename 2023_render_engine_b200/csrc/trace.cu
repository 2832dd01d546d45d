// Closest-hit and occlusion traversal of the compressed 8-wide BVH (sm_100a).
//
// k_trace_closest walks the rays (walk_queue, traverse.cuh) and leaves each ray's nearest triangle
// record; k_trace_finish then runs over the hits with all lanes busy: it proves or establishes
// the reference's answer, tests the analytic shapes and writes the result. Doing that work at
// the end of each ray's walk instead ran it with the few lanes whose rays had just ended.
//
// Reference parity (rt_trace_closest without RT_TRACE_FAST): the reference traversal
// (BVH::intersectRay, cuda_libraries/BVH.cu:355-448) returns, among the triangles it
// reaches, the last one in its static order that lowers its running offset and passes
// the error-bound test (Triangle.cu:569-593). That equals "smallest offset, ties to the
// highest static rank" — what the walk computes — unless (a) the winner is not
// reached because an ancestor box of the reference tree misses the ray, or (b) some
// triangle with a smaller offset fails the error-bound test after lowering the running
// offset. k_trace_finish proves (a) cannot happen with one slab test on the winner's own
// box (float rounding is monotonic, so every ancestor box passes when the winner's box
// does, for rays with tmax = inf and no zero direction component), and walks the winner's
// ancestors where that test does not decide; the walk detects (b) and marks the ray. Where
// either holds, k_trace_finish replays the reference traversal itself.
#include <algorithm>

#include "traverse.cuh"

namespace rtb {

namespace {

constexpr int kBlock = 128;

// What the exact walk leaves to do for a ray (ra, rb) with hit hv: the proof or the replay of the
// reference's answer (see the file comment), its id or record, and the analytic shapes.
template <bool FEW = false>
__device__ __forceinline__ float4 finish_exact(const SceneView &v, float4 ra, float4 rb, uint32_t flags, float4 hv,
                                               uint32_t *counters)
{
    const bool visible = (flags & kTraceVisible) != 0, shadow = (flags & RT_TRACE_SHADOW) != 0;
    float t = hv.x, b1 = hv.z, b2 = hv.w;
    int32_t rec = __float_as_int(hv.y), prim = rec;
    bool replay = rec == kHitReplay;
    const float tri_max = visible ? INFINITY : ra.w;
    if (rec >= 0 && !replay) {
        const float4 *p = reinterpret_cast<const float4 *>(v.tris + rec);
        const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
        prim = (int32_t)__float_as_uint(b.w);
        const float ix = fdiv(1.0f, rb.x), iy = fdiv(1.0f, rb.y), iz = fdiv(1.0f, rb.z);
        const float lx = fminf(fminf(a.x, b.x), c.x), ly = fminf(fminf(a.y, b.y), c.y),
                    lz = fminf(fminf(a.z, b.z), c.z);
        const float hx = fmaxf(fmaxf(a.x, b.x), c.x), hy = fmaxf(fmaxf(a.y, b.y), c.y),
                    hz = fmaxf(fmaxf(a.z, b.z), c.z);
        if (!(tri_max == INFINITY) || rb.x == 0.f || rb.y == 0.f || rb.z == 0.f ||
            !ref_box_test(lx, ly, lz, hx, hy, hz, ra.x, ra.y, ra.z, ix, iy, iz, tri_max)) {
            // walk the winner's ancestors in the reference tree (the root is never
            // box-tested)
            atomicAdd(counters, 1u);
            uint32_t j = v.ref_pos[prim];
            const uint32_t m = v.ntri, root = 2 * m - 2;
            while (m > 1) {
                const uint32_t q = m + j / 2;
                if (q >= root) break;
                const float2 *bx = v.ref_boxes + 3 * (size_t)q;
                const float2 b0 = __ldg(bx), b1v = __ldg(bx + 1), b2v = __ldg(bx + 2);
                if (!ref_box_test(b0.x, b0.y, b1v.x, b1v.y, b2v.x, b2v.y, ra.x, ra.y, ra.z, ix, iy, iz,
                                  tri_max)) {
                    replay = true;
                    break;
                }
                j = q;
            }
        }
    }
    if (replay) {
        const float4 r = replay_hit(v, ra, rb, tri_max, shadow, counters);
        t = r.x, prim = __float_as_int(r.y);
        if (prim >= 0) b1 = r.z, b2 = r.w;  // a ray the replay finds to miss keeps those of its walk
    }
    if (prim < 0) t = INFINITY;
    if ((flags & kTraceRecords) && prim >= 0) prim = (int32_t)v.leafpos[prim];
    if (v.nspheres)
        intersect_spheres<FEW>(v, v.subs ? __float_as_uint(rb.w) : 0u, ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, tri_max, shadow, t,
                          prim, b1, b2);
    return make_float4(t, __int_as_float(prim), b1, b2);
}

// The call's counters for the host: the last block to end writes them to `status` (pinned host memory;
// null: the host copies them itself) and clears them for the next call. Every thread of the block calls it.
__device__ __forceinline__ void publish_status(uint32_t *counters, uint32_t *status)
{
    if (!status) return;
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(counters + 4, 1u) != gridDim.x - 1) return;
    __threadfence();
    volatile uint32_t *c = counters, *out = status;
    for (int k = 0; k < 3; k++) out[k] = c[k];
    for (int k = 0; k < 5; k++) c[k] = 0;
    __threadfence_system();
}

// Scene::isVisible's decision on the ray's hit (see kTraceVisible).
__device__ __forceinline__ bool visible_hit(float4 h, float4 ra)
{
    return __float_as_int(h.y) != RT_PRIM_NONE && h.x <= ra.w;
}

// Whether an analytic shape occludes the ray before its tmax.
template <bool FEW = false>
__device__ __forceinline__ bool shape_occludes(const SceneView &v, float4 ra, float4 rb, bool shadow)
{
    if (!v.nspheres) return false;
    float t = ra.w, b1 = 0, b2 = 0;
    int32_t prim = -1;
    intersect_spheres<FEW>(v, 0u, ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, ra.w, shadow, t, prim, b1, b2);
    return prim >= 0 && t < ra.w;
}

// Ray i's decision, for a whole warp of consecutive rays from a multiple of 32: a byte, or the warp's word.
__device__ __forceinline__ void write_occlusion(void *out, bool bits, uint64_t i, uint64_t n, bool occ)
{
    if (bits) {
        const uint32_t word = __ballot_sync(kAllLanes, occ);
        if ((threadIdx.x & 31u) == 0 && i < n) static_cast<uint32_t *>(out)[i >> 5] = word;
    } else if (i < n) {
        static_cast<uint8_t *>(out)[i] = occ ? 1 : 0;
    }
}

// Persistent closest-hit kernel: warps fetch rays from counters[3] until all n are done.
// counters[0] counts the rays k_trace_finish has to look at beyond the walk's answer.
// A merged scene (rt_scene_merge) has no reference-order tree: a ray whose walk ran out of
// stack keeps the hit found so far there (status word set).
//
// kTraceVisible: the call wants Scene::isVisible's decision, hit and offset <= the ray's tmax, for the
// unbounded ray, and the walk is unbounded too. Skipping nodes that the ray enters beyond tmax would
// lose occluders: an entry distance is rounded by some 1e-7 of the origin's distance, which from a few
// hundred scene sizes away is more than the boxes' margin, and at grazing incidence the offset itself
// may lie before the entry (a barycentric mean of the vertices' offsets, not a point of the ray).
__device__ __forceinline__ uint2 walk_closest(const SceneView &v, TravWarp &scratch, const rt_ray *rays, uint64_t n,
                                              rt_hit *hits, uint32_t flags, uint32_t *counters)
{
    const bool shadow = (flags & RT_TRACE_SHADOW) != 0;
    return walk_queue<false, false, true>(
        v, scratch, (uint32_t)n, counters + 3,
        [&](uint32_t i, Walk &W) {
            float4 ra, rb;
            load_ray(rays, i, ra, rb);
            const uint32_t root = scene_root(v, v.subs ? __float_as_uint(rb.w) : 0u);
            walk_init(W, ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, (flags & kTraceVisible) ? INFINITY : ra.w, root, shadow);
        },
        [&](uint32_t i, Walk &W, float2 bary) {
            int32_t rec = (int32_t)W.brec;
            bool replay = false;
            if (!W.ok) {
                replay = v.subs == nullptr;
                if (v.subs) atomicCAS(counters + 1, 0u, (uint32_t)DEV_STACK_OVERFLOW);
            } else if (!(flags & RT_TRACE_FAST)) {
                replay = rec >= 0 && W.minblock < W.bt;
            }
            if (replay) {
                rec = kHitReplay;
                atomicAdd(counters, 1u);
            } else if (rec >= 0 && (flags & kTraceIds)) {
                rec = (int32_t)__float_as_uint(__ldg(&v.tris[rec].v1.w));
            }
            reinterpret_cast<float4 *>(hits)[i] = make_float4(W.bt, __int_as_float(rec), bary.x, bary.y);
        });
}

__global__ void __launch_bounds__(kBlock, RTB_TRAV_MIN_BLOCKS) k_trace_closest(SceneView v, const rt_ray *__restrict__ rays,
                                                                               uint64_t n,
                                                                               const uint32_t *__restrict__ n_dev,
                                                                               rt_hit *__restrict__ hits, uint32_t flags,
                                                                               uint32_t *__restrict__ counters)
{
    __shared__ TravWarp scratch[kBlock / 32];
    if (n_dev) n = min((uint64_t)*n_dev, n);
    walk_closest(v, scratch[threadIdx.x >> 5], rays, n, hits, flags, counters);
}

// A queue of at most 32 rays per resident warp in one launch: each warp takes one range of it, and
// finishes the rays of that range itself once they have all ended. 997 rays of a Cornell box took
// a memset, two kernels and a copy of the counters, 40 us a call; 29 us so.
__global__ void __launch_bounds__(kBlock, RTB_TRAV_MIN_BLOCKS) k_trace_small(SceneView v, const rt_ray *__restrict__ rays,
                                                                             uint64_t n, rt_hit *hits, uint32_t flags,
                                                                             uint32_t *counters, uint32_t *status)
{
    __shared__ TravWarp scratch[kBlock / 32];
    const uint2 mine = walk_closest(v, scratch[threadIdx.x >> 5], rays, n, hits, flags, counters);
    __syncwarp();
    if ((threadIdx.x & 31u) < mine.y) {
        const uint32_t i = mine.x + (threadIdx.x & 31u);
        float4 *h = reinterpret_cast<float4 *>(hits) + i;
        if (flags & RT_TRACE_FAST) {
            *h = finish_fast(v, rays, i, flags, *h, counters);
        } else {
            float4 ra, rb;
            load_ray(rays, i, ra, rb);
            *h = finish_exact(v, ra, rb, flags, *h, counters);
        }
    }
    publish_status(counters, status);
}

// Scenes of one node (up to four for occlusion) and few shapes: each warp takes 32 rays at a time, tests
// the node, every lane its triangles, and finishes them. All walks end after a step or so, so that idle
// lanes to refill or to help, pairs spread over the warp and a finishing pass over rays and hits cost more
// than they bring. 12-triangle box with two spheres, us by k_trace_closest and the finishing pass (or
// k_trace_small, k_trace_any) / so: 2^24 closest hits 1432 / 1153, in fast mode 1641 / 1116, 50,000 51 / 39,
// 200,000 any hits 46 / 37; 3,000,000 visibility decisions on 32 triangles 600 / 496.
// Bound by instructions, a sphere's test (90 per ray and sphere) above all.
enum TinyKind { kTinyExact, kTinyFast, kTinyVisible, kTinyAny };
constexpr int kTinyBlocks = 8;  // per SM: 7 / 8 / 9 gave 624 / 606 / 635 us for 2^23 rays (spills)
template <TinyKind KIND>
__global__ void __launch_bounds__(kBlock, kTinyBlocks) k_trace_tiny(SceneView v, const rt_ray *__restrict__ rays, uint64_t n,
                                                                    rt_hit *hits, uint32_t flags, void *__restrict__ out,
                                                                    bool bits, uint32_t *counters, uint32_t *status)
{
    __shared__ TravWarp scratch[kBlock / 32];
    TravWarp &sm = scratch[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const bool shadow = (flags & RT_TRACE_SHADOW) != 0;
    flags = (flags & RT_TRACE_SHADOW) | (KIND == kTinyVisible ? kTraceVisible : 0u);  // the rest is known here
    prefetch_shapes(v);
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(counters + 3, 32u);
        const uint64_t i = (uint64_t)__shfl_sync(kAllLanes, base, 0) + lane;
        if (i - lane >= n) break;
        float4 ra, rb;
        load_ray(rays, min(i, n - 1), ra, rb);
        Walk W;
        walk_init(W, ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, KIND == kTinyVisible ? INFINITY : ra.w,
                  i < n ? scene_root(v, 0u) : kNoRoot, shadow);
        bool active = W.cur != kNoRoot;
        do {
            if (walk_step<KIND == kTinyAny, false, false, true>(v, sm, W, active, INFINITY)) active = false;
        } while ((KIND == kTinyVisible || KIND == kTinyAny) && __any_sync(kAllLanes, active));
        bool occ = false;
        if (i < n) {
            load_ray(rays, i, ra, rb);  // again: held over the tests it would be spilled
            if (KIND == kTinyAny) {
                occ = (W.brec != kNoRec && W.bt < W.lim) || shape_occludes<true>(v, ra, rb, shadow);
            } else {
                int32_t rec = (int32_t)W.brec;
                const float2 bary = rec >= 0 ? sm.bary[lane] : make_float2(0.f, 0.f);
                if (KIND != kTinyFast && rec >= 0 && W.minblock < W.bt) {
                    rec = kHitReplay;
                    atomicAdd(counters, 1u);
                }
                float4 h = make_float4(W.bt, __int_as_float(rec), bary.x, bary.y);
                if (KIND == kTinyFast) {
                    if (rec >= 0) rec = (int32_t)__float_as_uint(__ldg(&v.tris[rec].v1.w));
                    intersect_spheres<true>(v, 0u, ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, ra.w, shadow, h.x, rec, h.z, h.w);
                    h.y = __int_as_float(rec);
                } else {
                    h = finish_exact<true>(v, ra, rb, flags, h, counters);
                }
                if (KIND == kTinyVisible)
                    occ = visible_hit(h, ra);
                else
                    reinterpret_cast<float4 *>(hits)[i] = h;
            }
        }
        if (KIND == kTinyVisible || KIND == kTinyAny) write_occlusion(out, bits, i, n, occ);
        __syncwarp();
    }
    publish_status(counters, status);
}

// Traversal work per ray (rt_trace_counts): the persistent walk of k_trace_closest without its
// exactness checks (closest hit) or the any-hit walk of the renderer's shadow rays, writing for
// ray i the BVH8 nodes it visited and the triangle records it tested.
template <bool ANY>
__global__ void __launch_bounds__(kBlock, RTB_TRAV_MIN_BLOCKS) k_trace_counts(SceneView v, const rt_ray *__restrict__ rays,
                                                                             uint64_t n, uint32_t flags,
                                                                             uint2 *__restrict__ counts,
                                                                             uint32_t *__restrict__ counters)
{
    __shared__ TravWarp scratch[kBlock / 32];
    const bool shadow = (flags & RT_TRACE_SHADOW) != 0;
    walk_queue<ANY, true, true>(
        v, scratch[threadIdx.x >> 5], (uint32_t)n, counters + 3,
        [&](uint32_t i, Walk &W) {
            float4 ra, rb;
            load_ray(rays, i, ra, rb);
            walk_init(W, ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, ra.w, scene_root(v, 0), shadow);
        },
        [&](uint32_t i, Walk &W, float2) {
            if (!W.ok)
                atomicCAS(counters + 1, 0u,
                          (uint32_t)(W.steps > v.nnodes + 1 ? DEV_STEP_CAP : DEV_STACK_OVERFLOW));
            counts[i] = make_uint2(W.cur == kNoRoot ? 0u : W.steps, W.tested);
        });
}

// The walk's hits -> the call's results, one thread per ray, without RT_TRACE_FAST: the proof or the
// replay of the reference's answer (see the file comment); the analytic shapes; triangle ids
// (kTraceRecords: the renderer's form, triangle records) or, for kTraceVisible, the occlusion
// decision in `out` (one byte per ray, or with bits one word per 32 rays).
__global__ void __launch_bounds__(kBlock, 8) k_trace_finish(SceneView v, const rt_ray *__restrict__ rays, uint64_t n,
                                                            const uint32_t *__restrict__ n_dev,
                                                            rt_hit *__restrict__ hits, uint32_t flags,
                                                            void *__restrict__ out, bool bits,
                                                            uint32_t *counters, uint32_t *status)
{
    if (n_dev) n = min((uint64_t)*n_dev, n);
    prefetch_shapes(v);
    const bool visible = (flags & kTraceVisible) != 0;
    // whole warps stay in the loop (the bit mask is gathered with a ballot)
    for (uint64_t i0 = (uint64_t)blockIdx.x * kBlock; i0 < n; i0 += (uint64_t)gridDim.x * kBlock) {
        const uint64_t i = i0 + threadIdx.x;
        bool occ = false;
        if (i < n) {
            float4 ra, rb;
            load_ray(rays, i, ra, rb);
            const float4 h = finish_exact(v, ra, rb, flags, reinterpret_cast<const float4 *>(hits)[i], counters);
            if (visible)
                occ = visible_hit(h, ra);
            else
                reinterpret_cast<float4 *>(hits)[i] = h;
        }
        if (visible) write_occlusion(out, bits, i, n, occ);
    }
    publish_status(counters, status);
}

// The same in fast mode (finish_fast). With nothing to do for most rays it only looks at those whose
// walk could not finish (counters[0] of them).
__global__ void __launch_bounds__(kBlock, 12) k_trace_finish_fast(SceneView v, const rt_ray *__restrict__ rays, uint64_t n,
                                                                  const uint32_t *__restrict__ n_dev,
                                                                  rt_hit *__restrict__ hits, uint32_t flags,
                                                                  uint32_t *counters, uint32_t *status)
{
    if (n_dev) n = min((uint64_t)*n_dev, n);
    if (!v.nspheres && *(volatile uint32_t *)counters == 0u) n = 0;
    if ((uint64_t)blockIdx.x * kBlock < n) prefetch_shapes(v);
    for (uint64_t i = (uint64_t)blockIdx.x * kBlock + threadIdx.x; i < n; i += (uint64_t)gridDim.x * kBlock) {
        float4 *h = reinterpret_cast<float4 *>(hits) + i;
        *h = finish_fast(v, rays, i, flags, *h, counters);
    }
    publish_status(counters, status);
}

// Any hit before tmax (RT_TRACE_FAST occlusion): the walk writes one byte per ray, k_any_finish
// adds the analytic shapes and packs the bits.
__global__ void __launch_bounds__(kBlock, RTB_TRAV_MIN_BLOCKS) k_trace_any(SceneView v, const rt_ray *__restrict__ rays,
                                                                          uint64_t n, uint8_t *__restrict__ occluded,
                                                                          uint32_t flags, uint32_t *counters,
                                                                          uint32_t *status)
{
    __shared__ TravWarp scratch[kBlock / 32];
    const bool shadow = (flags & RT_TRACE_SHADOW) != 0;
    walk_queue<true, false, true>(
        v, scratch[threadIdx.x >> 5], (uint32_t)n, counters + 3,
        [&](uint32_t i, Walk &W) {
            float4 ra, rb;
            load_ray(rays, i, ra, rb);
            walk_init(W, ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, ra.w, scene_root(v, 0), shadow);
        },
        [&](uint32_t i, Walk &W, float2) {
            if (!W.ok) atomicCAS(counters + 1, 0u, (uint32_t)DEV_STACK_OVERFLOW);
            occluded[i] = (W.brec != kNoRec && W.bt < W.lim) ? 1 : 0;
        });
    publish_status(counters, status);
}

template <bool BITS>
__global__ void __launch_bounds__(kBlock) k_any_finish(SceneView v, const rt_ray *__restrict__ rays, uint64_t n,
                                                       const uint8_t *occluded, void *out, uint32_t flags)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool occ = false;
    if (i < n) {
        occ = occluded[i] != 0;
        if (!occ && v.nspheres) {
            float4 ra, rb;
            load_ray(rays, i, ra, rb);
            occ = shape_occludes(v, ra, rb, (flags & RT_TRACE_SHADOW) != 0);
        }
    }
    write_occlusion(out, BITS, i, n, occ);  // the grid covers whole warps
}

}  // namespace

// Resident blocks of the persistent closest-hit kernel on the current device.
static unsigned persistent_blocks()
{
    unsigned cached = device_slot(SLOT_TRACE_RESIDENT);
    if (!cached) {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_closest, kBlock, 0);
        cached = device_sm_count() * (unsigned)std::max(per_sm, 1);
        set_device_slot(SLOT_TRACE_RESIDENT, cached);
    }
    return cached;
}

// Blocks of a walk over n rays: all that are resident, or one per 16 rays (4 per warp) where that is
// fewer.
static uint64_t walk_blocks(uint64_t n) { return std::min<uint64_t>((n + 15) / 16, persistent_blocks()); }

// The walk. n_dev: the count, when it is on the device (n bounds it).
static int launch_walk(const SceneView &v, const rt_ray *rays, uint64_t n, const uint32_t *n_dev, rt_hit *hits,
                       uint32_t flags, uint32_t *counters, cudaStream_t s)
{
    k_trace_closest<<<(unsigned)walk_blocks(n), kBlock, 0, s>>>(v, rays, n, n_dev, hits, flags, counters);
    RTB_CUDA(cudaGetLastError());
    return RT_OK;
}

// Fast, triangles only, ids wanted: the walk writes the ids itself; what is left are the rays whose walk
// could not finish, and their replays give ids.
static uint32_t walk_flags(const SceneView &v, uint32_t flags)
{
    return (flags & RT_TRACE_FAST) && !v.nspheres && !(flags & kTraceRecords) ? flags | kTraceIds : flags;
}

// Clears a call's counters unless the last call left them clear.
static int begin_call(const TraceCall &c, cudaStream_t s)
{
    if (!c.clean) RTB_CUDA(cudaMemsetAsync(c.counters, 0, 5 * sizeof(uint32_t), s));
    return RT_OK;
}

// The walk and what it leaves to do.
static int launch_trace(const SceneView &v, const rt_ray *rays, uint64_t n, const uint32_t *n_dev, rt_hit *hits,
                        uint32_t flags, void *out, bool bits, const TraceCall &c, cudaStream_t s)
{
    if (n == 0) return RT_OK;
    flags = walk_flags(v, flags);
    RTB_CHECK(begin_call(c, s));
    const unsigned finish = (unsigned)std::min<uint64_t>((n + kBlock - 1) / kBlock, 16ull * device_sm_count());
    RTB_CHECK(launch_walk(v, rays, n, n_dev, hits, flags, c.counters, s));
    if (flags & RT_TRACE_FAST)
        k_trace_finish_fast<<<finish, kBlock, 0, s>>>(v, rays, n, n_dev, hits, flags, c.counters, c.status);
    else
        k_trace_finish<<<finish, kBlock, 0, s>>>(v, rays, n, n_dev, hits, flags, out, bits, c.counters, c.status);
    RTB_CUDA(cudaGetLastError());
    return RT_OK;
}

// Scenes for k_trace_tiny: `nodes` at most (closest hits on four nodes, 3,000,000 rays: 375 us, 494 so), and
// so few shapes that skipping those a ray passes saves nothing (16 spheres, 2^23 rays: 1.33 ms against
// 1.60 without).
static bool tiny_scene(const SceneView &v, uint32_t nodes) { return !v.subs && v.nnodes <= nodes && v.nspheres <= 4; }

static int launch_tiny(TinyKind kind, const SceneView &v, const rt_ray *rays, uint64_t n, rt_hit *hits, uint32_t flags,
                       void *out, bool bits, const TraceCall &c, cudaStream_t s)
{
    RTB_CHECK(begin_call(c, s));
    const unsigned blocks = (unsigned)std::min<uint64_t>((n + kBlock - 1) / kBlock, (uint64_t)kTinyBlocks * device_sm_count());
    auto kernel = kind == kTinyExact  ? k_trace_tiny<kTinyExact>
                  : kind == kTinyFast ? k_trace_tiny<kTinyFast>
                  : kind == kTinyAny  ? k_trace_tiny<kTinyAny>
                                      : k_trace_tiny<kTinyVisible>;
    kernel<<<blocks, kBlock, 0, s>>>(v, rays, n, hits, flags, out, bits, c.counters, c.status);
    RTB_CUDA(cudaGetLastError());
    return RT_OK;
}

int launch_trace_closest(const SceneView &v, const rt_ray *rays, uint64_t n, rt_hit *hits, uint32_t flags,
                         const TraceCall &c, cudaStream_t s)
{
    flags &= RT_TRACE_SHADOW | RT_TRACE_FAST;
    if (n && tiny_scene(v, 1))
        return launch_tiny((flags & RT_TRACE_FAST) ? kTinyFast : kTinyExact, v, rays, n, hits, flags, nullptr, false, c, s);
    const uint64_t blocks = walk_blocks(n);
    if (n == 0 || n > 32ull * blocks * (kBlock / 32)) return launch_trace(v, rays, n, nullptr, hits, flags, nullptr, false, c, s);
    RTB_CHECK(begin_call(c, s));
    k_trace_small<<<(unsigned)blocks, kBlock, 0, s>>>(v, rays, n, hits, walk_flags(v, flags), c.counters, c.status);
    RTB_CUDA(cudaGetLastError());
    return RT_OK;
}

int launch_trace_closest_dev(const SceneView &v, const rt_ray *rays, const uint32_t *n_dev, uint32_t cap, rt_hit *hits,
                             uint32_t flags, uint32_t *counters, cudaStream_t s)
{
    return launch_trace(v, rays, cap, n_dev, hits, (flags & (RT_TRACE_SHADOW | RT_TRACE_FAST)) | kTraceRecords, nullptr,
                        false, TraceCall{counters, nullptr, false}, s);
}

int launch_walk_dev(const SceneView &v, const rt_ray *rays, const uint32_t *n_dev, uint32_t cap, rt_hit *hits,
                    uint32_t *counters, cudaStream_t s)
{
    return launch_walk(v, rays, cap, n_dev, hits, RT_TRACE_FAST | kTraceRecords, counters, s);
}

int launch_trace_visible(const SceneView &v, const rt_ray *rays, uint64_t n, rt_hit *hits, uint32_t flags, void *out,
                         bool bits, const TraceCall &c, cudaStream_t s)
{
    flags = (flags & RT_TRACE_SHADOW) | kTraceVisible;
    if (n && tiny_scene(v, 4)) return launch_tiny(kTinyVisible, v, rays, n, hits, flags, out, bits, c, s);
    return launch_trace(v, rays, n, nullptr, hits, flags, out, bits, c, s);
}

int launch_trace_counts(const SceneView &v, const rt_ray *rays, uint64_t n, uint32_t flags, bool anyhit,
                        uint32_t *counts, uint32_t *counters, cudaStream_t s)
{
    if (n == 0) return RT_OK;
    RTB_CUDA(cudaMemsetAsync(counters, 0, 4 * sizeof(uint32_t), s));
    const uint64_t blocks = std::min<uint64_t>((n + kBlock - 1) / kBlock, persistent_blocks());
    auto kernel = anyhit ? k_trace_counts<true> : k_trace_counts<false>;
    kernel<<<(unsigned)blocks, kBlock, 0, s>>>(v, rays, n, flags, reinterpret_cast<uint2 *>(counts), counters);
    RTB_CUDA(cudaGetLastError());
    return RT_OK;
}

int launch_trace_any(const SceneView &v, const rt_ray *rays, uint64_t n, uint8_t *walk_out, void *out, bool bits,
                     uint32_t flags, const TraceCall &c, cudaStream_t s)
{
    if (n == 0) return RT_OK;
    if (tiny_scene(v, 4)) return launch_tiny(kTinyAny, v, rays, n, nullptr, flags & RT_TRACE_SHADOW, out, bits, c, s);
    RTB_CHECK(begin_call(c, s));
    const uint64_t blocks = walk_blocks(n);
    k_trace_any<<<(unsigned)blocks, kBlock, 0, s>>>(v, rays, n, walk_out, flags, c.counters, c.status);
    RTB_CUDA(cudaGetLastError());
    if (bits || v.nspheres) {
        const uint64_t all = (n + kBlock - 1) / kBlock;
        auto kernel = bits ? k_any_finish<true> : k_any_finish<false>;
        kernel<<<(unsigned)all, kBlock, 0, s>>>(v, rays, n, walk_out, out, flags);
        RTB_CUDA(cudaGetLastError());
    }
    return RT_OK;
}

}  // namespace rtb
