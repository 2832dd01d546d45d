// BVH8 traversal and reference replay shared by the trace and render kernels.
// See trace.cu for the parity argument.
#pragma once

#include <cfloat>

#include "exact_math.cuh"
#include "rt_internal.h"

namespace rtb {

// Entries of a walk's stack (8 bytes each, in local memory). A walk that would need more drops
// the entries its best hit has already passed, and if that makes no room it ends, and its ray is
// replayed on the reference tree (exact); 32 entries overflowed on dense triangle soups without
// changing the render's speed.
#ifndef RTB_KSTACK
#define RTB_KSTACK 56
#endif
constexpr int kStack = RTB_KSTACK;

// Resident blocks of 128 threads per SM the traversal kernels are compiled for (register cap
// 65536 / (128 * N)): 9 gives 56 registers and 36 warps per SM.
#ifndef RTB_TRAV_MIN_BLOCKS
#define RTB_TRAV_MIN_BLOCKS 9
#endif
// Idle lanes a warp collects before it fetches new rays for them.
#ifndef RTB_REFILL
#define RTB_REFILL 8
#endif

__device__ __forceinline__ uint32_t byte_of(uint32_t w, int k) { return (w >> (8 * k)) & 0xFFu; }

// Scene records (nodes, triangles) and streamed rays. Evict-last L2 policies on the scene loads
// with evict-first ray loads were measured against these plain read-only loads: 3207 against 3183
// Mrays/s on the 2^24 BVH-stress rays, 1821 against 1832 on the render; not kept.
__device__ __forceinline__ uint4 ld_scene(const uint4 *ptr) { return __ldg(ptr); }
__device__ __forceinline__ float4 ld_scene(const float4 *ptr) { return __ldg(ptr); }
__device__ __forceinline__ float4 ld_stream(const float4 *ptr) { return __ldg(ptr); }

__device__ __forceinline__ void load_ray(const rt_ray *rays, uint64_t i, float4 &a, float4 &b)
{
    const float4 *r4 = reinterpret_cast<const float4 *>(rays);
    a = ld_stream(r4 + 2 * i);
    b = ld_stream(r4 + 2 * i + 1);
}

// Sorting network for 8 keys (ascending).
__device__ __forceinline__ void cas(uint32_t &a, uint32_t &b)
{
    uint32_t lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}
__device__ __forceinline__ void sort8(uint32_t k[8])
{
    cas(k[0], k[1]); cas(k[2], k[3]); cas(k[4], k[5]); cas(k[6], k[7]);
    cas(k[0], k[2]); cas(k[1], k[3]); cas(k[4], k[6]); cas(k[5], k[7]);
    cas(k[1], k[2]); cas(k[5], k[6]); cas(k[0], k[4]); cas(k[3], k[7]);
    cas(k[1], k[5]); cas(k[2], k[6]);
    cas(k[1], k[4]); cas(k[3], k[6]);
    cas(k[2], k[4]); cas(k[3], k[5]);
    cas(k[3], k[4]);
}

constexpr unsigned kAllLanes = 0xFFFFFFFFu;
constexpr uint32_t kNoRec = 0xFFFFFFFFu;  // no triangle record (record indices are below 2^30)

// One ray's walk, held by one lane of a warp.
struct Walk {
    float ox, oy, oz;
    float ix, iy, iz;  // 1 / direction
    float Sx, Sy, Sz;  // shear of the watertight test (make_watertight)
    uint32_t kz;       // its axis; bits 2..6: the lane that fetched the ray (walk_queue's groups)
    float lim;         // nodes that the ray enters beyond this are skipped
    uint32_t cur;      // node to visit next
    int sp;
    uint32_t steps;
    bool ok;      // false: ran out of stack or steps
    bool shadow;  // checkShadow semantics: transparent primitives are skipped
    float bt;     // the best hit so far: offset, triangle record (its barycentrics: TravWarp::bary)
    uint32_t brec;
    float minblock;   // smallest offset that failed the error-bound test
    uint32_t tested;  // triangle records tested (rt_trace_counts only; steps counts nodes)
    // node index, entry distance bits: one 8-byte local access per push / pop. Keeping the bottom
    // 4 or 8 entries in shared memory instead (the rest in local memory) measured slower
    uint2 st[kStack];
};

// What the lanes of a warp exchange in shared memory while they test triangles.
struct alignas(16) TravWarp {
    float4 res[32];     // offset, record and flags, b1, b2 of the pair lane j tested
    float2 bary[32];    // b1, b2 of each lane's best hit
    uint16_t pair[32];  // lane that owns pair j, its triangle's offset in the node's block << 5
    // per ray in flight, at the lane that fetched it: how many lanes walk it, and what the lanes
    // that ended have found between them
    uint32_t lanes[32];
    float4 found[32];   // offset, triangle record, b1, b2
    float blocked[32];  // minblock; -1: a lane ran out of stack or steps
};
constexpr uint32_t kPairBlocked = 0x80000000u;      // TravWarp::res.y: fails the error-bound test
constexpr uint32_t kPairTransparent = 0x40000000u;  // transparent to shadow rays
constexpr uint32_t kPairRecord = 0x3FFFFFFFu;

// BVH8 root of scene `sub` (0 for a plain scene) and its spheres [s0, s0 + ns).
__device__ __forceinline__ uint32_t scene_root(const SceneView &v, uint32_t sub)
{
    if (v.subs) return v.subs[min(sub, v.nsubs - 1)].root;
    return v.ntri ? 0u : kNoRoot;
}
__device__ __forceinline__ void scene_spheres(const SceneView &v, uint32_t sub, uint32_t &s0, uint32_t &ns)
{
    if (v.subs) {
        const SubScene &ss = v.subs[min(sub, v.nsubs - 1)];
        s0 = ss.sph0;
        ns = ss.nsph;
    } else {
        s0 = 0;
        ns = v.nspheres;
    }
}

// root: the BVH8 node the walk starts at (kNoRoot: the scene has no triangles; the walk is
// skipped). lim: the ray's limit.
__device__ __forceinline__ void walk_init(Walk &W, float ox, float oy, float oz, float dx, float dy, float dz,
                                          float lim, uint32_t root, bool shadow)
{
    W.ox = ox;
    W.oy = oy;
    W.oz = oz;
    W.ix = 1.0f / dx;
    W.iy = 1.0f / dy;
    W.iz = 1.0f / dz;
    const WatertightRay w = make_watertight(ox, oy, oz, dx, dy, dz, lim);
    W.Sx = w.Sx;
    W.Sy = w.Sy;
    W.Sz = w.Sz;
    W.kz = (uint32_t)w.kz | ((threadIdx.x & 31u) << 2);
    W.lim = lim;
    W.cur = root;
    W.sp = 0;
    W.steps = 0;
    W.ok = true;
    W.shadow = shadow;
    W.bt = INFINITY;
    W.brec = kNoRec;
    W.minblock = INFINITY;
    W.tested = 0;
}

// The triangles of a node's hit leaves for one lane, one after the other: what walk_step does with
// SERIAL, and what its pairs give.
template <bool ANY>
__device__ __forceinline__ void lane_triangles(const SceneView &v, TravWarp &sm, Walk &W, uint32_t tri_base, uint32_t trimask)
{
    WatertightRay w;
    w.ox = W.ox, w.oy = W.oy, w.oz = W.oz;
    w.Sx = W.Sx, w.Sy = W.Sy, w.Sz = W.Sz;
    w.tmax = W.lim;
    w.kz = (int)(W.kz & 3u);
    w.kx = w.kz == 2 ? 0 : w.kz + 1;
    w.ky = w.kx == 2 ? 0 : w.kx + 1;
#pragma unroll 1
    while (trimask) {
        const uint32_t rec = tri_base + (uint32_t)__ffs(trimask) - 1u;
        trimask &= trimask - 1u;
        const float4 *p = reinterpret_cast<const float4 *>(v.tris + rec);
        const float4 a = ld_scene(p), b = ld_scene(p + 1), c = ld_scene(p + 2);
        TriHit h;
        if (!watertight_test(w, a, b, c, h)) continue;
        if (W.shadow && (__float_as_uint(c.w) & 1u)) continue;
        if (h.t > W.bt) continue;
        if (h.t == W.bt && W.brec != kNoRec && __float_as_uint(a.w) < __float_as_uint(__ldg(&v.tris[W.brec].v0.w))) continue;
        if (h.t <= watertight_delta_t(h)) {
            W.minblock = fminf(W.minblock, h.t);
            continue;
        }
        W.bt = h.t;
        W.brec = rec;
        sm.bary[threadIdx.x & 31u] = make_float2(fmul(h.e1, h.invDet), fmul(h.e2, h.invDet));
        if (ANY) return;
    }
}

// One step of a warp's walks: each active lane visits its next node, then the warp tests the
// triangles of the leaves its lanes hit, one (ray, triangle) pair per lane: the pairs are numbered
// by a prefix sum over the lanes, each lane reads its pair's ray from the owner by shuffles, and the
// owner takes the results in its own triangle order, so a walk gives what it gives when every
// lane tests its own triangles one after the other. A step hits about as many triangles as a
// warp has lanes, so they mostly take one round, where the serial loop took as many as the lane
// with the most of them, with a few lanes active in each and a triangle fetch of latency per round.
// shared_t: the ray's best offset among other lanes (INFINITY: none). Returns whether the walk ended.
// ORDERED: hit children are visited near to far and skipped once the best hit lies before them.
// Without it (a walk that ends at any hit, whose limit never shrinks) they are visited as they come
// in the node and the stack holds node indices only, twice as many.
// SERIAL: every lane tests its own triangles.
template <bool ANY, bool COUNT, bool ORDERED, bool SERIAL = false>
__device__ __forceinline__ bool walk_step(const SceneView &v, TravWarp &sm, Walk &W, bool active, float shared_t)
{
    const unsigned lane = threadIdx.x & 31u;
    // visit a node: its eight quantized child boxes; the triangles of the hit leaves as a
    // mask over the node's block of records, the hit interior children pushed far to near
    uint32_t trimask = 0, leafend = 0, tri_base = 0, next = kNoRoot;
    float next_t = 0.f;
    bool done = false;
    if (active) {
        if (++W.steps > v.nnodes + 1) {
            W.ok = false;
            done = true;
        } else {
            const uint4 *np = reinterpret_cast<const uint4 *>(v.nodes + W.cur);
            const uint4 n0 = ld_scene(np), n1 = ld_scene(np + 1), n2 = ld_scene(np + 2), n3 = ld_scene(np + 3),
                        n4 = ld_scene(np + 4);
            const float sx = __uint_as_float((n0.w & 0xFFu) << 23);
            const float sy = __uint_as_float(((n0.w >> 8) & 0xFFu) << 23);
            const float sz = __uint_as_float(((n0.w >> 16) & 0xFFu) << 23);
            const uint32_t imask = n0.w >> 24;
            const uint32_t child_base = n1.x;
            tri_base = n1.y;
            const uint32_t meta_lo = n1.z, meta_hi = n1.w;
            // the planes the ray meets first and last on each axis, by the sign of its direction:
            // a selection per node instead of a minimum and a maximum per child and axis
            const bool fx = W.ix < 0.f, fy = W.iy < 0.f, fz = W.iz < 0.f;
            const uint32_t nx[2] = {fx ? n3.z : n2.x, fx ? n3.w : n2.y}, hx[2] = {fx ? n2.x : n3.z, fx ? n2.y : n3.w};
            const uint32_t ny[2] = {fy ? n4.x : n2.z, fy ? n4.y : n2.w}, hy[2] = {fy ? n2.z : n4.x, fy ? n2.w : n4.y};
            const uint32_t nz[2] = {fz ? n4.z : n3.x, fz ? n4.w : n3.y}, hz[2] = {fz ? n3.x : n4.z, fz ? n3.y : n4.w};
            // per-axis affine map t = q * (s * inv) + (p * inv - o * inv)
            const float ax = sx * W.ix, bx = fmaf(__uint_as_float(n0.x), W.ix, -W.ox * W.ix);
            const float ay = sy * W.iy, by = fmaf(__uint_as_float(n0.y), W.iy, -W.oy * W.iy);
            const float az = sz * W.iz, bz = fmaf(__uint_as_float(n0.z), W.iz, -W.oz * W.iz);
            const float tlimit = fminf(fminf(W.bt, W.lim), shared_t);
            uint32_t keys[8];
            uint32_t nint = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int b = k & 3;
                const uint32_t meta = byte_of(k < 4 ? meta_lo : meta_hi, b);
                float t1x = fmaf((float)byte_of(nx[k >> 2], b), ax, bx), t2x = fmaf((float)byte_of(hx[k >> 2], b), ax, bx);
                float t1y = fmaf((float)byte_of(ny[k >> 2], b), ay, by), t2y = fmaf((float)byte_of(hy[k >> 2], b), ay, by);
                float t1z = fmaf((float)byte_of(nz[k >> 2], b), az, bz), t2z = fmaf((float)byte_of(hz[k >> 2], b), az, bz);
                // a bound that is NaN (of a zero direction component) does not limit the ray; the other
                // bound of its axis still does in the counts
                if (COUNT) {
                    const float lx = fminf(t1x, t2x), ly = fminf(t1y, t2y), lz = fminf(t1z, t2z);
                    t2x = fmaxf(t1x, t2x), t2y = fmaxf(t1y, t2y), t2z = fmaxf(t1z, t2z);
                    t1x = lx, t1y = ly, t1z = lz;
                }
                const float tn = fmaxf(fmaxf(t1x, t1y), fmaxf(t1z, 0.0f));
                const float tf = fminf(fminf(t2x, t2y), fminf(t2z, tlimit));
                const bool hit = (meta != 0xFFu) && (tn <= tf);
                const bool interior = (imask >> k) & 1u;
                if (ORDERED) {
                    keys[k] = (hit && interior) ? ((__float_as_uint(tn) & ~7u) | meta) : 0xFFFFFFFFu;
                    nint += (hit && interior) ? 1u : 0u;
                } else if (hit && interior) {
                    if (next != kNoRoot) {
                        if (W.sp < 2 * kStack)
                            reinterpret_cast<uint32_t *>(W.st)[W.sp++] = next;
                        else
                            W.ok = false, done = true;
                    }
                    next = child_base + meta;
                }
                if (hit && !interior) {
                    trimask |= ((2u << (meta >> 5)) - 1u) << (meta & 31u);
                    if (COUNT) leafend |= (1u << (meta >> 5)) << (meta & 31u);
                }
            }
            if (ORDERED && nint) {
                sort8(keys);
                if (W.sp + (int)nint - 1 > kStack) {  // drop the entries beyond the best hit
                    int kept = 0;
#pragma unroll 1
                    for (int e = 0; e < W.sp; e++) {
                        const uint2 x = W.st[e];
                        if (__uint_as_float(x.y) <= tlimit) W.st[kept++] = x;
                    }
                    W.sp = kept;
                    if (W.sp + (int)nint - 1 > kStack) {
                        W.ok = false;
                        done = true;
                    }
                }
                if (!done) {
#pragma unroll
                    for (int j = 7; j >= 1; j--)
                        if (j < (int)nint) {
                            W.st[W.sp] = make_uint2(child_base + (keys[j] & 7u), keys[j] & ~7u);
                            W.sp++;
                        }
                }
                next = child_base + (keys[0] & 7u);
                next_t = __uint_as_float(keys[0] & ~7u);
            }
        }
    }
    // the triangles of the whole warp, 32 pairs a round
    const uint32_t mytris = (uint32_t)__popc(trimask);
    if (SERIAL) {
        lane_triangles<ANY>(v, sm, W, tri_base, trimask);
        __syncwarp();
    } else if (__any_sync(kAllLanes, trimask != 0)) {
        uint32_t incl = mytris;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kAllLanes, incl, o);
            if (lane >= (unsigned)o) incl += y;
        }
        const uint32_t total = __shfl_sync(kAllLanes, incl, 31);
        uint32_t at = incl - mytris, left = trimask;
        if (COUNT && !ANY) W.tested += mytris;
        uint32_t before = 0;  // triangles of this lane offered in earlier rounds (COUNT)
        for (uint32_t r0 = 0; r0 < total; r0 += 32) {
            const uint32_t first = at;
#pragma unroll 1
            while (left && at < r0 + 32) {
                const uint32_t off = (uint32_t)__ffs(left) - 1u;
                left &= left - 1u;
                sm.pair[at - r0] = (uint16_t)(lane | (off << 5));
                at++;
            }
            __syncwarp();
            const bool on = r0 + lane < total;
            const uint32_t e = on ? sm.pair[lane] : lane;
            const int src = (int)(e & 31u);
            WatertightRay w;
            w.ox = __shfl_sync(kAllLanes, W.ox, src);
            w.oy = __shfl_sync(kAllLanes, W.oy, src);
            w.oz = __shfl_sync(kAllLanes, W.oz, src);
            w.Sx = __shfl_sync(kAllLanes, W.Sx, src);
            w.Sy = __shfl_sync(kAllLanes, W.Sy, src);
            w.Sz = __shfl_sync(kAllLanes, W.Sz, src);
            const uint32_t axis_base = __shfl_sync(kAllLanes, (tri_base << 2) | (W.kz & 3u), src);
            w.tmax = __shfl_sync(kAllLanes, W.lim, src);
            w.kz = (int)(axis_base & 3u);
            w.kx = w.kz == 2 ? 0 : w.kz + 1;
            w.ky = w.kx == 2 ? 0 : w.kx + 1;
            bool hit = false;
            if (on) {
                const uint32_t rec = (axis_base >> 2) + (e >> 5);
                const float4 *p = reinterpret_cast<const float4 *>(v.tris + rec);
                const float4 a = ld_scene(p), b = ld_scene(p + 1), c = ld_scene(p + 2);
                TriHit h;
                hit = watertight_test(w, a, b, c, h);
                if (hit) {
                    const float dt = watertight_delta_t(h);
                    const uint32_t fl = rec | (h.t <= dt ? kPairBlocked : 0u) |
                                        ((__float_as_uint(c.w) & 1u) ? kPairTransparent : 0u);
                    sm.res[lane] =
                        make_float4(h.t, __uint_as_float(fl), fmul(h.e1, h.invDet), fmul(h.e2, h.invDet));
                }
            }
            uint32_t mine = __ballot_sync(kAllLanes, hit);
            __syncwarp();
            // the owner takes the results of its own pairs, in order
            mine = at > first ? (mine >> (first - r0)) & ((1u << (at - first)) - 1u) : 0u;
            if (ANY && W.brec != kNoRec) mine = 0;
#pragma unroll 1
            while (mine) {
                const uint32_t j = first - r0 + (uint32_t)__ffs(mine) - 1u;
                mine &= mine - 1u;
                const float2 tf = *reinterpret_cast<const float2 *>(&sm.res[j]);
                const uint32_t fl = __float_as_uint(tf.y), rec = fl & kPairRecord;
                if (W.shadow && (fl & kPairTransparent)) continue;
                if (tf.x > W.bt) continue;
                if (tf.x == W.bt && W.brec != kNoRec &&
                    __float_as_uint(__ldg(&v.tris[rec].v0.w)) < __float_as_uint(__ldg(&v.tris[W.brec].v0.w)))
                    continue;
                if (fl & kPairBlocked) {
                    W.minblock = fminf(W.minblock, tf.x);
                    continue;
                }
                W.bt = tf.x;
                W.brec = rec;
                sm.bary[lane] = *(reinterpret_cast<const float2 *>(&sm.res[j]) + 1);
                if (ANY) {
                    if (COUNT) {  // the triangles up to the end of this one's leaf
                        const uint32_t off = sm.pair[j] >> 5;
                        const uint32_t end = (uint32_t)__ffs(leafend >> off) - 1u + off;
                        before = (uint32_t)__popc(trimask & ((2u << end) - 1u));
                    }
                    break;
                }
            }
            if (COUNT && ANY) __syncwarp();  // the owners have read their pairs (above) before the next round's
        }
        if (COUNT && ANY) W.tested += W.brec != kNoRec ? before : mytris;
        __syncwarp();
    }
    if (active) {
        // the nearest hit child, or the top stack entry the best hit has not passed
        const float tl = fminf(fminf(W.bt, W.lim), shared_t);
        if (ANY && (W.brec != kNoRec || shared_t < INFINITY)) done = true;
        if (!done) {
            if (next != kNoRoot && next_t <= tl) {
                W.cur = next;
            } else if (!ORDERED) {
                if (W.sp > 0)
                    W.cur = reinterpret_cast<uint32_t *>(W.st)[--W.sp];
                else
                    done = true;
            } else {
                done = true;
#pragma unroll 1
                while (W.sp > 0) {
                    W.sp--;
                    const uint2 e = W.st[W.sp];
                    if (__uint_as_float(e.y) <= tl) {
                        W.cur = e.x;
                        done = false;
                        break;
                    }
                }
            }
        }
    }
    return active && done;
}

// Walks the rays [0, n) of a queue: every lane of a persistent warp runs its own ray, and lanes
// whose rays are done fetch the next ones together (measured for 1 / 4 / 8 / 16 idle lanes:
// 2^24 rays of the BVH-stress scene 4.60 / 4.60 / 4.58 / 4.98 ms, its 1080p x 64 spp frame 212 / 209
// / 209 / 217 ms).
//
// Once the queue is empty, idle lanes help: each takes the top stack entry of a lane that has one
// and walks that subtree for the same ray, so the few longest rays, which pass hundreds of nodes,
// no longer hold the kernel up one node at a time (2^22 rays: the last SM ran 0.4 of 1.3 ms by
// itself). The lanes of a ray share its best offset for skipping nodes, and the last of them to
// end reports what they found together: the nearest hit, ties to the higher rank, which does not
// depend on who found it. A short queue is dealt out over all warps (quota rays each), so that
// there are idle lanes to help from the start.
//
// init(i, W) prepares ray i (walk_init); finish(i, W, bary) consumes its result. ANY: the walk
// ends at the first accepted hit in triangle order (in the node that has one). Returns the warp's
// rays where each warp takes one range of the queue ([x, x + y), y = 0 otherwise). COUNT: also
// counts the triangles a serial walk would test (whole leaves, up to the leaf of the accepted hit
// under ANY), and every ray keeps its own lane.
template <bool ANY, bool COUNT, bool ORDERED, typename Init, typename Finish>
__device__ __forceinline__ uint2 walk_queue(const SceneView &v, TravWarp &sm, uint32_t n, uint32_t *work,
                                           Init init, Finish finish)
{
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x / 32u);
    const uint32_t quota = COUNT ? 32u : min(max((n + warps - 1u) / warps, 1u), 32u);
    // with quota * warps >= n the first fetch of each warp takes all there is for it
    const bool single = !COUNT && (uint64_t)quota * warps >= n;
    uint32_t ray = 0xFFFFFFFFu;
    bool exhausted = false;
    uint2 taken = make_uint2(0u, 0u);
    Walk W;
    for (;;) {
        const unsigned idle = __ballot_sync(kAllLanes, ray == 0xFFFFFFFFu);
        const uint32_t busy = 32u - (uint32_t)__popc(idle);
        if (!exhausted && busy + min(quota, (uint32_t)RTB_REFILL) <= quota) {
            const uint32_t want = quota - busy;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(work, want);
            base = __shfl_sync(kAllLanes, base, 0);
            exhausted = single || base + want >= n;
            if (single && base < n) taken = make_uint2(base, min(want, n - base));
            const uint32_t rank = (uint32_t)__popc(idle & ((1u << lane) - 1u));
            if (ray == 0xFFFFFFFFu && rank < want && base + rank < n) {
                ray = base + rank;
                init(ray, W);
                if (W.cur == kNoRoot) {
                    finish(ray, W, make_float2(0.f, 0.f));
                    ray = 0xFFFFFFFFu;
                }
            }
            __syncwarp();
            if (!COUNT && exhausted) break;
        }
        const bool active = ray != 0xFFFFFFFFu;
        if (!__any_sync(kAllLanes, active)) {
            if (exhausted) return taken;
            continue;
        }
        if (walk_step<ANY, COUNT, ORDERED>(v, sm, W, active, INFINITY)) {
            finish(ray, W, W.brec != kNoRec ? sm.bary[lane] : make_float2(0.f, 0.f));
            ray = 0xFFFFFFFFu;
        }
    }
    if (COUNT) return taken;
    // the queue is empty: the warp's last rays, with all its lanes
    sm.lanes[lane] = 1;
    sm.found[lane] = make_float4(INFINITY, __uint_as_float(kNoRec), 0.f, 0.f);
    sm.blocked[lane] = INFINITY;
    __syncwarp();
    for (;;) {
        const unsigned idle = __ballot_sync(kAllLanes, ray == 0xFFFFFFFFu);
        if (idle == kAllLanes) return taken;
        // idle lane k takes the top entry of the k-th lane that has one
        const bool give = ray != 0xFFFFFFFFu && W.sp > 0;
        const unsigned givers = __ballot_sync(kAllLanes, give);
        if (idle && givers) {
            const uint32_t below = (1u << lane) - 1u;
            const uint32_t moves = min((uint32_t)__popc(idle), (uint32_t)__popc(givers));
            const uint32_t k = (uint32_t)__popc((give ? givers : idle) & below);
            uint2 e = make_uint2(0u, 0u);
            if (give && k < moves) {
                if (ORDERED)
                    e = W.st[--W.sp];
                else
                    e.x = reinterpret_cast<uint32_t *>(W.st)[--W.sp];
                sm.pair[k] = (uint16_t)lane;
            }
            __syncwarp();
            const bool take = ray == 0xFFFFFFFFu && k < moves;
            const int src = take ? (int)sm.pair[k] : (int)lane;
            const uint32_t ex = __shfl_sync(kAllLanes, e.x, src), ey = __shfl_sync(kAllLanes, e.y, src);
            const uint32_t r = __shfl_sync(kAllLanes, ray, src), kz = __shfl_sync(kAllLanes, W.kz, src);
            const float ox = __shfl_sync(kAllLanes, W.ox, src), oy = __shfl_sync(kAllLanes, W.oy, src),
                        oz = __shfl_sync(kAllLanes, W.oz, src);
            const float ix = __shfl_sync(kAllLanes, W.ix, src), iy = __shfl_sync(kAllLanes, W.iy, src),
                        iz = __shfl_sync(kAllLanes, W.iz, src);
            const float Sx = __shfl_sync(kAllLanes, W.Sx, src), Sy = __shfl_sync(kAllLanes, W.Sy, src),
                        Sz = __shfl_sync(kAllLanes, W.Sz, src);
            const float lim = __shfl_sync(kAllLanes, W.lim, src), bt = __shfl_sync(kAllLanes, W.bt, src);
            const bool shadow = __shfl_sync(kAllLanes, (int)W.shadow, src) != 0;
            // an entry the giver's best hit has passed is dropped
            if (take && __uint_as_float(ey) <= fminf(bt, lim)) {
                ray = r;
                W.ox = ox, W.oy = oy, W.oz = oz;
                W.ix = ix, W.iy = iy, W.iz = iz;
                W.Sx = Sx, W.Sy = Sy, W.Sz = Sz;
                W.kz = kz;
                W.lim = lim;
                W.cur = ex;
                W.sp = 0;
                W.steps = 0;
                W.ok = true;
                W.shadow = shadow;
                W.bt = INFINITY;
                W.brec = kNoRec;
                W.minblock = INFINITY;
                atomicAdd(&sm.lanes[kz >> 2], 1u);
            }
            __syncwarp();
        }
        const bool active = ray != 0xFFFFFFFFu;
        const float shared_t = active ? sm.found[W.kz >> 2].x : INFINITY;
        const bool done = walk_step<ANY, COUNT, ORDERED>(v, sm, W, active, shared_t);
        // one ended lane after the other adds what it found to its ray's; the last reports it
        unsigned ended = __ballot_sync(kAllLanes, done);
        while (ended) {
            const unsigned who = __ffs(ended) - 1;
            ended &= ended - 1u;
            if (lane == who) {
                const uint32_t home = W.kz >> 2;
                const float4 f = sm.found[home];
                const uint32_t frec = __float_as_uint(f.y);
                const bool take = W.brec != kNoRec && !(W.bt > f.x) &&
                                  !(W.bt == f.x && frec != kNoRec &&
                                    __float_as_uint(__ldg(&v.tris[W.brec].v0.w)) <
                                        __float_as_uint(__ldg(&v.tris[frec].v0.w)));
                const float4 g = take ? make_float4(W.bt, __uint_as_float(W.brec), sm.bary[lane].x, sm.bary[lane].y)
                                      : f;
                const float mb = W.ok ? fminf(sm.blocked[home], W.minblock) : -1.f;
                if (--sm.lanes[home] == 0) {
                    W.ok = mb >= 0.f;
                    W.bt = g.x;
                    W.brec = __float_as_uint(g.y);
                    W.minblock = mb;
                    finish(ray, W, make_float2(g.z, g.w));
                } else {
                    sm.found[home] = g;
                    sm.blocked[home] = mb;
                }
                ray = 0xFFFFFFFFu;
            }
            __syncwarp();
        }
    }
}

// The exact test of one analytic shape. A plane hit reports its object-space (x, y); 0 for spheres.
__device__ __forceinline__ bool shape_hit(const SphereRecord &sr, float ox, float oy, float oz, float dx, float dy,
                                          float dz, float tmax, float &t, float &u, float &v)
{
    u = v = 0.f;
    return (sr.flags & kShapePlane) ? plane_test(sr.w2o, ox, oy, oz, dx, dy, dz, tmax, t, u, v)
                                    : sphere_test(sr.w2o, sr.radius, ox, oy, oz, dx, dy, dz, tmax, t);
}
// Out of line, where a ray comes for the few shapes it may hit.
__device__ __noinline__ static bool shape_test(const SphereRecord *sr, float ox, float oy, float oz, float dx, float dy,
                                               float dz, float tmax, float3 *hit)
{
    float t, u, v;
    const bool ok = shape_hit(*sr, ox, oy, oz, dx, dy, dz, tmax, t, u, v);
    if (ok) *hit = make_float3(t, u, v);
    return ok;
}

// The shapes' records into the L1 cache, which every kernel finds empty: the loop over the shapes reads
// record after record, each a trip to the L2 otherwise.
__device__ __forceinline__ void prefetch_shapes(const SceneView &v)
{
    const uint32_t lines = (min(v.nspheres, 256u) * (uint32_t)sizeof(SphereRecord) + 127u) / 128u;
    for (uint32_t i = threadIdx.x; i < lines; i += blockDim.x)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char *>(v.spheres) + 128u * i));
}

// Scene::intersects' loop over the analytic shapes (Scene.cu:141-146) of scene `sub`. FEW: of few shapes
// some ray of a warp comes near each, so that the test for those it passes by a margin saves nothing.
template <bool FEW = false>
__device__ __forceinline__ void intersect_spheres(const SceneView &v, uint32_t sub, float ox, float oy, float oz,
                                                  float dx, float dy, float dz, float tmax, bool shadow, float &t,
                                                  int32_t &prim, float &b1, float &b2)
{
    uint32_t s0, ns;
    scene_spheres(v, sub, s0, ns);
    for (uint32_t s = s0; s < s0 + ns; s++) {
        float3 hit;  // offset, and of a plane the object-space (x, y)
        if (FEW) {
            const SphereRecord &sr = v.spheres[s];
            if (shadow && (sr.flags & 1u)) continue;
            if (!shape_hit(sr, ox, oy, oz, dx, dy, dz, tmax, hit.x, hit.y, hit.z)) continue;
        } else {
            const SphereRecord *sr = v.spheres + s;
            const float4 *m = reinterpret_cast<const float4 *>(sr->w2o);
            const float4 tail = __ldg(reinterpret_cast<const float4 *>(&sr->radius));  // radius, material, shape id, flags
            const uint32_t flags = __float_as_uint(tail.w);
            if (shadow && (flags & 1u)) continue;
            if ((flags & kShapeAffine) && sphere_missed(m, tail.x, ox, oy, oz, dx, dy, dz)) continue;
            if (!shape_test(sr, ox, oy, oz, dx, dy, dz, tmax, &hit)) continue;
        }
        if (hit.x < t) {
            t = hit.x;
            prim = RT_PRIM_SHAPE | (int32_t)s;
            b1 = hit.y;
            b2 = hit.z;
        }
    }
}

// Replays BVH::intersectRay on the reference tree for one ray (BVH.cu:355-448).
__device__ __noinline__ static int32_t replay_reference(const SceneView &v, const WatertightRay &w, float ix, float iy, float iz,
                                    bool shadow, float &tOut, float &b1, float &b2, bool &overflow)
{
    const uint32_t n = v.ntri;
    float h = INFINITY;
    int32_t hit = -1;
    auto tri_seq = [&](uint32_t tri) {
        const float4 *p = reinterpret_cast<const float4 *>(v.tris + v.leafpos[tri]);
        float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
        if (shadow && (__float_as_uint(c.w) & 1u)) return;
        TriHit th;
        if (!watertight_test(w, a, b, c, th)) return;
        if (th.t > h) return;
        h = th.t;
        if (h <= watertight_delta_t(th)) return;
        hit = (int32_t)tri;
        b1 = fmul(th.e1, th.invDet);
        b2 = fmul(th.e2, th.invDet);
    };
    if (n == 1) {
        tri_seq(v.ref_sorted[0]);
        tOut = h;
        return hit;
    }
    uint32_t stack[64];
    int sp = 0;
    stack[sp++] = 2 * n - 2;
    while (sp > 0) {
        uint32_t node = stack[--sp];
        uint32_t ch0 = 2 * (node - n);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            uint32_t c = ch0 + (uint32_t)k;
            if (c < n) {
                tri_seq(v.ref_sorted[c]);
            } else {
                const float2 *bx = v.ref_boxes + 3 * (size_t)c;
                float2 b0 = __ldg(bx), b1v = __ldg(bx + 1), b2v = __ldg(bx + 2);
                if (ref_box_test(b0.x, b0.y, b1v.x, b1v.y, b2v.x, b2v.y, w.ox, w.oy, w.oz, ix, iy, iz, w.tmax)) {
                    if (sp < 64)
                        stack[sp++] = c;
                    else
                        overflow = true;
                }
            }
        }
    }
    tOut = h;
    return hit;
}

// rt_hit::prim between the walk and the end of a trace: a triangle record, -1, or
constexpr int32_t kHitReplay = 0x7FFFFFFE;  // the reference traversal decides

// The reference traversal's hit of a ray: offset, triangle id or -1, b1, b2. Out of line, values in and
// out, so that the few rays that need it cost the others no memory.
__device__ __noinline__ static float4 replay_hit(const SceneView &v, float4 ra, float4 rb, float tmax, bool shadow,
                                                 uint32_t *counters)
{
    const WatertightRay w = make_watertight(ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, tmax);
    bool overflow = false;
    float t, b1 = 0.f, b2 = 0.f;
    const int32_t prim =
        replay_reference(v, w, fdiv(1.0f, rb.x), fdiv(1.0f, rb.y), fdiv(1.0f, rb.z), shadow, t, b1, b2, overflow);
    if (overflow) atomicCAS(counters + 1, 0u, (uint32_t)DEV_STACK_OVERFLOW);
    atomicAdd(counters + 2, 1u);
    return make_float4(t, __int_as_float(prim), b1, b2);
}

// What a fast-mode walk (RT_TRACE_FAST) leaves to do for ray i: the replay of a walk that ran out of
// stack, the triangle's id unless the caller wants records or the walk wrote ids, and the
// analytic shapes. Returns the ray's hit.
__device__ __forceinline__ float4 finish_fast(const SceneView &v, const rt_ray *rays, uint64_t i, uint32_t flags,
                                              float4 hv, uint32_t *counters)
{
    float t = hv.x, b1 = hv.z, b2 = hv.w;
    int32_t prim = __float_as_int(hv.y);
    const bool replay = prim == kHitReplay, shadow = (flags & RT_TRACE_SHADOW) != 0;
    if (!v.nspheres && !replay) return hv;
    float4 ra, rb;
    load_ray(rays, i, ra, rb);
    if (replay) {
        const WatertightRay w = make_watertight(ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, ra.w);
        bool overflow = false;
        prim = replay_reference(v, w, fdiv(1.0f, rb.x), fdiv(1.0f, rb.y), fdiv(1.0f, rb.z), shadow, t, b1, b2, overflow);
        if (overflow) atomicCAS(counters + 1, 0u, (uint32_t)DEV_STACK_OVERFLOW);
        atomicAdd(counters + 2, 1u);
        if ((flags & kTraceRecords) && prim >= 0) prim = (int32_t)v.leafpos[prim];
    } else if (prim >= 0 && !(flags & (kTraceRecords | kTraceIds))) {
        prim = (int32_t)__float_as_uint(__ldg(&v.tris[prim].v1.w));
    }
    if (prim < 0) t = INFINITY;
    // the ray's last word is its scene in a merged scene
    if (v.nspheres)
        intersect_spheres(v, v.subs ? __float_as_uint(rb.w) : 0u, ra.x, ra.y, ra.z, rb.x, rb.y, rb.z, ra.w, shadow, t, prim,
                          b1, b2);
    return make_float4(t, __int_as_float(prim), b1, b2);
}

}  // namespace rtb
