// k-nearest photon query over the implicit kd-tree and the photon density estimate,
// shared by the photon-map entry points (photon.cu) and the renderer (render.cu).
#pragma once

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "surface.cuh"

namespace rtb {

constexpr uint32_t kKnnMaxK = 128;

// Euclidean norm as the reference evaluates it: s = 0; s += r*r per axis; sqrt
// (kdtree.h:175-176, difference kdtree.h:67-76).
__device__ __forceinline__ float ref_dist(float qx, float qy, float qz, float4 p)
{
    float dx = __fsub_rn(qx, p.x), dy = __fsub_rn(qy, p.y), dz = __fsub_rn(qz, p.z);
    float s = __fadd_rn(__fadd_rn(__fadd_rn(0.f, __fmul_rn(dx, dx)), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    return __fsqrt_rn(s);
}

// The same without the root (0 + r*r is r*r).
__device__ __forceinline__ float ref_dist2(float qx, float qy, float qz, float4 p)
{
    float dx = __fsub_rn(qx, p.x), dy = __fsub_rn(qy, p.y), dz = __fsub_rn(qz, p.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// nn::KDTree::nearest_neighbors_impl (kdtree.h:111-152) without recursion: photons with
// distance < bound on the query's shape (or any, sid = -1) enter a max-heap of k; the bound
// becomes the k-th distance once k are held; the far side of a split is visited only when
// the plane is nearer than the bound. Fills hd/hi (max-heap) and returns the count.
__device__ __forceinline__ uint32_t knn_query(const float4 *__restrict__ node_pos, const int2 *__restrict__ node_aux,
                                              uint32_t n, float qx, float qy, float qz, int32_t sid, uint32_t k,
                                              float radius, float *hd, int32_t *hi)
{
    uint32_t cnt = 0;
    float rcur = radius;
    uint32_t sl[64], sr[64];
    float sd[64];
    int sp = 1;
    sl[0] = 0;
    sr[0] = n;
    sd[0] = 0.f;
    while (sp > 0) {
        sp--;
        const uint32_t l = sl[sp], r = sr[sp];
        if (!(sd[sp] < rcur) || r <= l) continue;
        const uint32_t m = (l + r) >> 1;
        const float4 p = __ldg(node_pos + m);
        const int2 aux = __ldg(node_aux + m);
        const float dist = ref_dist(qx, qy, qz, p);
        if (dist < rcur && (sid == -1 || aux.x == sid)) {
            if (cnt < k) {  // sift up
                uint32_t c = cnt++;
                while (c > 0) {
                    uint32_t par = (c - 1) >> 1;
                    if (!(hd[par] < dist)) break;
                    hd[c] = hd[par];
                    hi[c] = hi[par];
                    c = par;
                }
                hd[c] = dist;
                hi[c] = aux.y;
                if (cnt == k) rcur = hd[0];
            } else {  // replace the farthest, sift down
                uint32_t c = 0;
                for (;;) {
                    uint32_t a = 2 * c + 1, b = a + 1, big = c;
                    float bd = dist;
                    if (a < k && hd[a] > bd) {
                        big = a;
                        bd = hd[a];
                    }
                    if (b < k && hd[b] > bd) {
                        big = b;
                        bd = hd[b];
                    }
                    if (big == c) break;
                    hd[c] = hd[big];
                    hi[c] = hi[big];
                    c = big;
                }
                hd[c] = dist;
                hi[c] = aux.y;
                rcur = hd[0];
            }
        }
        if (r - l > 1) {
            const uint32_t axis = __float_as_uint(p.w);
            const float qa = axis == 0 ? qx : (axis == 1 ? qy : qz);
            const float pa = axis == 0 ? p.x : (axis == 1 ? p.y : p.z);
            const float diff = __fsub_rn(qa, pa);
            const float pd = __fsqrt_rn(__fmul_rn(diff, diff));  // norm(p - pplane) (kdtree.h:138-148)
            uint32_t nl, nr, fl, fr;
            if (qa < pa) {
                nl = l, nr = m, fl = m + 1, fr = r;
            } else {
                nl = m + 1, nr = r, fl = l, fr = m;
            }
            if (sp + 2 <= 64) {
                sl[sp] = fl, sr[sp] = fr, sd[sp] = pd, sp++;  // far side, tested again when popped
                sl[sp] = nl, sr[sp] = nr, sd[sp] = 0.f, sp++;
            }
        }
    }
    return cnt;
}

// Max-heap -> ascending distance, in place.
__device__ __forceinline__ void heap_to_sorted(float *hd, int32_t *hi, uint32_t cnt)
{
    for (uint32_t end = cnt; end > 1; end--) {
        float td = hd[0];
        int32_t ti = hi[0];
        float ld = hd[end - 1];
        int32_t li = hi[end - 1];
        uint32_t c = 0;
        const uint32_t m = end - 1;
        for (;;) {
            uint32_t a = 2 * c + 1, b = a + 1, big = c;
            float bd = ld;
            if (a < m && hd[a] > bd) {
                big = a;
                bd = hd[a];
            }
            if (b < m && hd[b] > bd) {
                big = b;
                bd = hd[b];
            }
            if (big == c) break;
            hd[c] = hd[big];
            hi[c] = hi[big];
            c = big;
        }
        hd[c] = ld;
        hi[c] = li;
        hd[end - 1] = td;
        hi[end - 1] = ti;
    }
}

// Radius of the subsurface gather: th_photonSubsurfaceContributions' searchRadius (Scene.cu:802).
constexpr float kSubsurfaceRadius = 0.3f;

// impPaper_dipoleDiffusionAproximation (geometricMath.cu:455-490), one channel: the dipole
// diffuse reflectance Rd at distance r with the reduced scattering coefficient (1 - g) sigma_s.
// The terms that do not depend on r are set up once per query (DipoleChannel); dipole_eval
// evaluates the rest per photon, the hot loop of the subsurface gather, with reciprocal square
// roots and the hardware exponential (relative error about 1e-6, against 1e-7 for the IEEE
// operations): with d = sqrt(r^2 + z^2), 1/d and 1/d^3 come from one rsqrt.
struct DipoleChannel {
    float tr, zr, zv, omf, alpha;  // sigma_tr, real and virtual source depths, 1 - Fdr, albedo
};

__device__ __forceinline__ DipoleChannel dipole_setup(float ss, float sa, float g, float eta)
{
    DipoleChannel c;
    const float rs = (1 - g) * ss;
    const float rt = rs + sa;
    c.alpha = rs / rt;
    c.tr = sqrtf(3 * sa * rt);
    const float fdr = (-1.440f / (eta * eta)) + (0.710f / eta) + 0.668f + 0.0636f * eta;
    const float A = (1 + fdr) / (1 - fdr);
    c.zr = sqrtf(3 * (1 - c.alpha)) / c.tr;
    c.zv = c.zr * A;
    c.omf = 1 - fdr;
    return c;
}

__device__ __forceinline__ float dipole_eval(const DipoleChannel &c, float r2)
{
    const float xr = r2 + c.zr * c.zr, xv = r2 + c.zv * c.zv;
    const float ir = rsqrtf(xr), iv = rsqrtf(xv);  // 1/dr, 1/dv
    const float trdr = c.tr * (xr * ir), trdv = c.tr * (xv * iv);
    const float rd = (trdr + 1) * __expf(-trdr) * c.zr * (ir * ir * ir) + (trdv + 1) * __expf(-trdv) * c.zv * (iv * iv * iv);
    const float c1 = c.zr * (c.tr + ir);
    return c1 * rd * c.omf * c.alpha;
}

// Largest squared distance whose root is below radius (-1: none): the search compares squared
// distances, and roots are taken of its answers only.
inline float radius_squared(float radius)
{
    if (!(radius > 0.f)) return -1.f;
    float s = std::min(radius * radius, FLT_MAX);
    while (s > 0.f && !(std::sqrt(s) < radius)) s = std::nextafter(s, 0.f);
    while (s < FLT_MAX && std::sqrt(std::nextafter(s, FLT_MAX)) < radius) s = std::nextafter(s, FLT_MAX);
    return s;
}

// ------------------------------------------------------- warp-cooperative queries
// A warp answers its queries together, with their traversal stacks in shared memory. Every lane of
// the warp must call these functions together. Serial per-node chains of local-memory stack and
// heap traffic are what bound the one-thread-per-query form: here a subtree below a given size (a
// contiguous range of the implicit tree) is read with coalesced loads, k-nearest candidates go to a
// buffer that is narrowed to about k now and then, and the photons' attributes lie in tree order.

// Device view of a built photon map, all arrays in tree-slot order.
struct PhotonTree {
    const float4 *pos;  // xyz, split axis (uint bits)
    const int2 *aux;    // shape id, photon index
    const float4 *pw;   // power rgb, cosine of the photon's normal with its reversed direction
    const float4 *dir;  // arrival direction xyz, 0
    uint32_t n;
};

inline PhotonTree photon_tree(const rt_photon_map *m)
{
    PhotonTree t;
    t.pos = m->node_pos.as<float4>();
    t.aux = m->node_aux.as<int2>();
    t.pw = m->node_pw.as<float4>();
    t.dir = m->node_dir.as<float4>();
    t.n = (uint32_t)m->n;
    return t;
}

constexpr uint32_t kRadiusScan = 256;  // scanned subtree size of a fixed-radius query
// Stack bound: a popped range is replaced by its two halves, and for n < 2^32 ranges of more
// than kRadiusScan (or kGroupScan) photons lie on at most 27 levels, so the stack holds at most 28
// entries.
constexpr int kWarpStack = 32;
constexpr unsigned kFullMask = 0xFFFFFFFFu;

struct PhotonWarpScratch {  // per warp, in shared memory
    uint32_t sl[kWarpStack], sr[kWarpStack];
    float sd[kWarpStack];
    float d2[64];  // squared distances and
    uint32_t slot[64];  // tree slots of photons found and not yet added
};

__device__ __forceinline__ float warp_sum(float v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
    return v;
}

__device__ __forceinline__ float warp_max(float v)
{
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFullMask, v, o));
    return v;
}

// The pruned traversal of knn_query (kdtree.h:111-152) for a warp: the same depth-first,
// near-side-first order with the same pruning (a far side is skipped when its split plane is
// not nearer than the bound), decided warp-uniformly with the stack in shared memory. A range
// of at most Scan photons is read 32 photons per load instead of node by node. bound() is the squared
// search distance (warp-uniform); visit(valid, squared distance, shape, slot) is offered up to 32
// photons, one per lane (an internal node's photon on lane 0).
template <uint32_t Scan, class Scratch, class Bound, class Visit>
__device__ __forceinline__ void warp_traverse(const PhotonTree &t, float qx, float qy, float qz, Scratch &sm,
                                              Bound &&bound, Visit &&visit)
{
    const uint32_t lane = threadIdx.x & 31u;
    int sp = 1;
    if (lane == 0) {
        sm.sl[0] = 0;
        sm.sr[0] = t.n;
        sm.sd[0] = 0.f;
    }
    __syncwarp();
    while (sp > 0) {
        sp--;
        const uint32_t l = sm.sl[sp], r = sm.sr[sp];
        const float pd = sm.sd[sp];
        __syncwarp();  // every lane has read the entry before lane 0 reuses it
        if (!(pd <= bound()) || r <= l) continue;
        if (r - l <= Scan) {
            for (uint32_t base = l; base < r; base += 64) {  // two loads in flight per lane
                const uint32_t j0 = base + lane, j1 = base + 32 + lane;
                float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f), p1 = p0;
                int s0 = -1, s1 = -1;
                if (j0 < r) {
                    p0 = __ldg(t.pos + j0);
                    s0 = __ldg(&t.aux[j0].x);
                }
                if (j1 < r) {
                    p1 = __ldg(t.pos + j1);
                    s1 = __ldg(&t.aux[j1].x);
                }
                visit(j0 < r, j0 < r ? ref_dist2(qx, qy, qz, p0) : INFINITY, s0, j0);
                if (base + 32 < r) visit(j1 < r, j1 < r ? ref_dist2(qx, qy, qz, p1) : INFINITY, s1, j1);
            }
            continue;
        }
        const uint32_t m = (l + r) >> 1;
        const float4 p = __ldg(t.pos + m);  // one address for the warp
        visit(lane == 0, ref_dist2(qx, qy, qz, p), __ldg(&t.aux[m].x), m);
        const uint32_t axis = __float_as_uint(p.w);
        const float qa = axis == 0 ? qx : (axis == 1 ? qy : qz);
        const float pa = axis == 0 ? p.x : (axis == 1 ? p.y : p.z);
        const float diff = __fsub_rn(qa, pa);
        const float pd2 = __fmul_rn(diff, diff);  // squared norm(p - pplane) (kdtree.h:138-148)
        if (sp + 2 <= kWarpStack) {  // holds for n < 2^31 (kWarpStack)
            if (lane == 0) {
                if (qa < pa) {
                    sm.sl[sp] = m + 1, sm.sr[sp] = r, sm.sd[sp] = pd2;  // far side
                    sm.sl[sp + 1] = l, sm.sr[sp + 1] = m, sm.sd[sp + 1] = 0.f;
                } else {
                    sm.sl[sp] = l, sm.sr[sp] = m, sm.sd[sp] = pd2;
                    sm.sl[sp + 1] = m + 1, sm.sr[sp + 1] = r, sm.sd[sp + 1] = 0.f;
                }
            }
            sp += 2;
        }
        __syncwarp();
    }
}

// ------------------------------------------------------- k-nearest queries, a warp each
// For few queries (density_lanes), where a query's own time counts: a whole warp scans and selects for it.
// 500 / 4,000 estimates of 50 among 830,000 photons: 108 / 160 us, with 8 lanes each 176 / 263.
constexpr uint32_t kKnnScan = 64;  // scanned subtree size
// Candidate buffer: after a selection it holds k <= kKnnMaxK, and it is selected again before an append
// could take it past kKnnBuf.
constexpr uint32_t kKnnBuf = 256;
static_assert(kKnnBuf >= 2 * kKnnMaxK, "room for k plus one batch of candidates");

struct KnnWarpScratch {  // per warp, in shared memory
    float kd[kKnnBuf];     // candidates' squared distances (unordered)
    uint32_t ki[kKnnBuf];  // and tree slots
    uint32_t sl[kWarpStack], sr[kWarpStack];
    float sd[kWarpStack];
};

// The k nearest photons within the radius (radius2: radius_squared of it) on shape sid (-1: any), up to
// the order in which photons at exactly equal distances compete for the last place. Candidates are
// appended to a buffer; when it first holds k, and whenever it is nearly full, the k nearest are kept and
// the bound becomes the k-th distance, as the reference's heap bound does once it holds k. Leaves the
// neighbours' tree slots unordered in sm.ki; returns their count (all lanes).
__device__ __forceinline__ uint32_t warp_knn(const PhotonTree &t, float qx, float qy, float qz, int32_t sid, uint32_t k,
                                             float radius2, KnnWarpScratch &sm)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t below = (1u << lane) - 1u;
    uint32_t cnt = 0, select_at = k;
    // photons nearer than this (squared): all within the radius at first
    float rcur = radius2 < 0.f ? -1.f : __int_as_float(__float_as_int(radius2) + 1);
    // keep the k nearest of cnt > k buffered: the k-th smallest distance v (bitwise search on
    // the float bits, which order like the values for distances >= 0), then the ones below it
    // and as many equal to it as fill k
    auto select = [&]() {
        uint32_t key[kKnnBuf / 32], slot[kKnnBuf / 32];
#pragma unroll
        for (uint32_t i = 0; i < kKnnBuf / 32; i++) {
            const uint32_t j = lane + 32 * i;
            key[i] = j < cnt ? __float_as_uint(sm.kd[j]) : 0xFFFFFFFFu;
            slot[i] = j < cnt ? sm.ki[j] : 0u;
        }
        // largest v with fewer than k keys below it (the k-th smallest key), or the first
        // threshold met with exactly k below it (then those k are the k nearest, no tie)
        uint32_t v = 0, less = 0;
        bool exact = false;
        for (int bit = 30; bit >= 0; bit--) {
            const uint32_t tv = v | (1u << bit);
            uint32_t c = 0;
#pragma unroll
            for (uint32_t i = 0; i < kKnnBuf / 32; i++) c += key[i] < tv;
            c = __reduce_add_sync(kFullMask, c);
            if (c == k) {
                v = tv;
                less = k;
                exact = true;
                break;
            }
            if (c < k) {
                v = tv;
                less = c;
            }
        }
        const uint32_t need = k - less;
        __syncwarp();  // every lane holds its entries before the buffer is rewritten
        uint32_t blt = 0, beq = 0;
#pragma unroll
        for (uint32_t i = 0; i < kKnnBuf / 32; i++) {
            const bool lt = key[i] < v, eq = key[i] == v;
            const unsigned mlt = __ballot_sync(kFullMask, lt), meq = __ballot_sync(kFullMask, eq);
            if (lt) {
                const uint32_t pos = blt + __popc(mlt & below);
                sm.kd[pos] = __uint_as_float(key[i]);
                sm.ki[pos] = slot[i];
            }
            if (eq && !exact) {
                const uint32_t rk = beq + __popc(meq & below);
                if (rk < need) {
                    sm.kd[less + rk] = __uint_as_float(key[i]);
                    sm.ki[less + rk] = slot[i];
                }
            }
            blt += __popc(mlt);
            beq += __popc(meq);
        }
        __syncwarp();
        cnt = k;
        // the bound: the largest kept distance (v itself unless the search stopped early)
        float mx = 0.f;
        for (uint32_t j = lane; j < k; j += 32) mx = fmaxf(mx, sm.kd[j]);
        rcur = exact ? warp_max(mx) : __uint_as_float(v);
        select_at = kKnnBuf - 32;
    };
    warp_traverse<kKnnScan>(t, qx, qy, qz, sm, [&]() { return rcur; },
                            [&](bool valid, float dist2, int shape, uint32_t slot) {
                                const bool c = valid && dist2 < rcur && (sid == -1 || shape == sid);
                                const unsigned mask = __ballot_sync(kFullMask, c);
                                if (!mask) return;
                                if (c) {
                                    const uint32_t pos = cnt + __popc(mask & below);
                                    sm.kd[pos] = dist2;
                                    sm.ki[pos] = slot;
                                }
                                cnt += __popc(mask);
                                __syncwarp();
                                if (cnt >= select_at) select();
                            });
    if (cnt > k) select();
    __syncwarp();
    return cnt;
}

// ------------------------------------------------------- k-nearest queries, 8 lanes each
// A warp answers four k-nearest queries at a time, kGroup lanes each. A whole warp per query was
// bound by instructions, most of them the same on all lanes (a node step, a selection's counting
// loop); four queries share them. All 32 lanes run these functions together, converged; a group
// without a query is idle (on = false). Gathers of a hybrid frame (960x540, 2 samples per pixel,
// 413,000 photons, k = 50) 8.05 -> 5.45 ms, density of 50,021 points at k = 100 0.56 -> 0.44 ms.
// Still bound by instructions (0.72 issued per cycle and scheduler): 20 leaves and 44 nodes per
// query, three selections of about 130 candidates. Leaves of 16 or 64 photons visit 31 or 12 leaves and
// 62 or 32 nodes, for the same work.
constexpr uint32_t kGroup = 8;
// Lanes of a group's ballot.
template <uint32_t G>
__device__ __forceinline__ uint32_t group_mask()
{
    return 0xFFFFFFFFu >> (32u - G);
}
constexpr uint32_t kGroupScan = 32;  // subtrees of at most this many photons are read whole
// Candidates a group may append between two looks at its buffer: a leaf and the nodes above it.
constexpr uint32_t kGroupBatch = 64;
static_assert(kGroupScan + 28 <= kGroupBatch, "a descent's candidates");
// Blocks of 128 threads per SM the density kernels are compiled for (72 registers); their shared
// memory holds 7 at k = 50, 5 at k = 128.
constexpr int kGatherBlocks = 7;
// Candidates a selection may keep beyond k: with some room it ends after two or three counts.
constexpr uint32_t kKnnSlack = 8;

// Buffer entries of a query: the k and the slack, a batch, and what may gather between selections. Half
// of k: at k = 50 room for 40 against 64 gave 1.30 / 1.33 ms on 200,003 queries (a tighter bound
// sooner), at k = 100 458 / 441 us on 50,021 densities (a selection more).
__host__ __device__ constexpr uint32_t knn_cap(uint32_t k)
{
    return (k + kKnnSlack + kGroupBatch + 16 + k / 2 + 7) / 8 * 8;
}
// 32-bit words of shared memory a query takes: distances, tree slots, traversal stack; 8 more than a
// multiple of 32, so that the four groups' accesses fall on different banks.
__host__ __device__ constexpr uint32_t knn_words(uint32_t k)
{
    return (2 * knn_cap(k) + 3 * kWarpStack + 23) / 32 * 32 + 8;
}
static_assert(knn_words(50) >= 2 * knn_cap(50) + 3 * kWarpStack && knn_words(50) % 32 == 8, "layout");

struct KnnGroup {
    float *kd;     // candidates' squared distances (unordered)
    uint32_t *ki;  // and tree slots
    uint32_t *sl, *sr;
    float *sd;
    uint32_t cap;
};

// The calling lane's group of G lanes in `words`, the shared memory of the warp (32 / G * knn_words(k)).
template <uint32_t G = kGroup>
__device__ __forceinline__ KnnGroup knn_group(uint32_t *words, uint32_t k)
{
    KnnGroup g;
    g.cap = knn_cap(k);
    uint32_t *w = words + ((threadIdx.x & 31u) / G) * knn_words(k);
    g.kd = reinterpret_cast<float *>(w);
    g.ki = w + g.cap;
    g.sl = g.ki + g.cap;
    g.sr = g.sl + kWarpStack;
    g.sd = reinterpret_cast<float *>(g.sr + kWarpStack);
    return g;
}

template <uint32_t G, typename T>
__device__ __forceinline__ T group_sum(T v)
{
#pragma unroll
    for (uint32_t o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
    return v;
}
template <uint32_t G>
__device__ __forceinline__ float group_max(float v)
{
#pragma unroll
    for (uint32_t o = G / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFullMask, v, o));
    return v;
}

// Distances that differ by fewer than this many steps of their squares' float representation may
// be equal.
constexpr int kRootSteps = 4;

// Keeps the nearest of the groups' candidates where there are more than k + slack: all of those at
// a squared distance v or less, with v such that there are k to k + slack of them, found by
// interpolation between counts (photons lie on surfaces: their number grows with the square) and
// halving on the float bits in turn (the values are not negative, so their bits order like them).
// Where equal distances leave no such v, exactly k are kept. bound becomes v, or a little more than
// the largest value where nothing has to go; groups of fewer than k candidates are left alone.
template <uint32_t G>
__device__ __forceinline__ void group_select(const KnnGroup &g, uint32_t k, uint32_t slack, uint32_t &cnt, float &bound)
{
    const uint32_t lane = threadIdx.x & (G - 1u), shift = threadIdx.x & 31u & ~(G - 1u);
    const uint32_t mine = cnt >= k ? cnt : 0u;
    float mx = 0.f;
    for (uint32_t j = lane; j < mine; j += G) mx = fmaxf(mx, g.kd[j]);
    int lo = -1, hi = __float_as_int(group_max<G>(mx)) + 2 * kRootSteps;
    uint32_t clo = 0, chi = mine;
    for (uint32_t it = 0;; it++) {
        const bool more = chi > k + slack && hi - lo > 1;
        if (!__any_sync(kFullMask, more)) break;
        int mid = lo + (hi - lo) / 2;
        if (!(it & 1u)) {
            const float a = lo < 0 ? 0.f : __int_as_float(lo), b = __int_as_float(hi);
            const float f = __fdividef((float)(k + slack / 2 - clo), (float)(chi - clo));
            mid = min(max(__float_as_int(a + (b - a) * f), lo + 1), hi - 1);
        }
        uint32_t c = 0;
        for (uint32_t j = lane; j < mine; j += G) c += __float_as_int(g.kd[j]) <= mid ? 1u : 0u;
        c = group_sum<G>(c);
        if (more) {
            if (c >= k) {
                hi = mid;
                chi = c;
            } else {
                lo = mid;
                clo = c;
            }
        }
    }
    const bool tied = chi > k + slack;  // lo and hi are neighbours
    if (mine) bound = fminf(bound, __int_as_float(hi));
    // in place: a kept entry moves down or stays
    const bool cut = mine > chi || tied;
    const uint32_t most = __reduce_max_sync(kFullMask, cut ? mine : 0u);
    const bool ties = __any_sync(kFullMask, tied);
    uint32_t kept = 0, equal = 0;
    for (uint32_t j0 = 0; j0 < most; j0 += G) {
        const uint32_t j = j0 + lane;
        const bool in = j < mine;
        const float d = in ? g.kd[j] : 0.f;
        const uint32_t s = in ? g.ki[j] : 0u;
        const int key = __float_as_int(d);
        bool keep = in && key <= hi;
        if (ties) {
            const uint32_t eq = (__ballot_sync(kFullMask, in && key == hi) >> shift) & group_mask<G>();
            if (tied && key == hi) keep = keep && clo + equal + __popc(eq & ((1u << lane) - 1u)) < k;
            equal += __popc(eq);
        }
        const uint32_t m = (__ballot_sync(kFullMask, keep) >> shift) & group_mask<G>();
        if (keep) {
            const uint32_t at = kept + __popc(m & ((1u << lane) - 1u));
            g.kd[at] = d;
            g.ki[at] = s;
        }
        kept += __popc(m);
        __syncwarp();
    }
    if (cut) cnt = kept;
}

// The photons nearest to (qx, qy, qz) within the radius (radius2: radius_squared of it) on shape sid
// (-1: any), as nn::KDTree::nearest_neighbors_impl finds them (kdtree.h:111-152): the near side of
// a split first, the far side only where the plane is nearer than the search distance, which becomes
// an upper bound of the k-th distance once k are held. Leaves the candidates unordered in g.kd / g.ki
// and returns their number: all there are if fewer than k, else the k nearest and up to slack more.
// bound: every photon within the radius that is not among them has a squared distance above it, or
// (exactly k kept among equals) one equal to it.
template <uint32_t G = kGroup>
__device__ __forceinline__ uint32_t group_knn(const float4 *__restrict__ pos, const int2 *__restrict__ aux, uint32_t n,
                                              float qx, float qy, float qz, int32_t sid, uint32_t k, float radius2,
                                              uint32_t slack, bool on, const KnnGroup &g, float &bound)
{
    const uint32_t lane = threadIdx.x & (G - 1u), shift = threadIdx.x & 31u & ~(G - 1u);
    const uint32_t below = (1u << lane) - 1u;
    uint32_t l = 0, r = n, cnt = 0, limit = k;
    int sp = 0;
    bool live = on && n > 0;
    bound = radius2;
    while (__any_sync(kFullMask, live)) {
        // down to a leaf
        for (;;) {
            const bool down = live && r - l > kGroupScan;
            if (!__any_sync(kFullMask, down)) break;
            if (down) {
                const uint32_t m = (uint32_t)(((uint64_t)l + r) >> 1);
                const float4 p = __ldg(pos + m);  // one address for the group
                const float d = ref_dist2(qx, qy, qz, p);
                if (d <= bound && (sid == -1 || __ldg(&aux[m].x) == sid)) {
                    if (lane == 0) {
                        g.kd[cnt] = d;
                        g.ki[cnt] = m;
                    }
                    cnt++;
                }
                const uint32_t axis = __float_as_uint(p.w);
                const float qa = axis == 0 ? qx : (axis == 1 ? qy : qz);
                const float pa = axis == 0 ? p.x : (axis == 1 ? p.y : p.z);
                const float diff = __fsub_rn(qa, pa);
                const float pd = __fmul_rn(diff, diff);  // squared norm(p - pplane) (kdtree.h:138-148)
                const bool left = qa < pa;
                if (pd <= bound) {
                    if (lane == 0) {
                        g.sl[sp] = left ? m + 1 : l;
                        g.sr[sp] = left ? r : m;
                        g.sd[sp] = pd;
                    }
                    sp++;
                }
                if (left)
                    r = m;
                else
                    l = m + 1;
            }
        }
        float4 p[kGroupScan / G];
#pragma unroll
        for (uint32_t i = 0; i < kGroupScan / G; i++)
            if (live && l + lane + G * i < r) p[i] = __ldg(pos + l + lane + G * i);
#pragma unroll
        for (uint32_t i = 0; i < kGroupScan / G; i++) {
            const uint32_t j = l + lane + G * i;
            const float d = ref_dist2(qx, qy, qz, p[i]);
            bool c = live && j < r && d <= bound;
            if (c && sid != -1) c = __ldg(&aux[j].x) == sid;
            const uint32_t m = (__ballot_sync(kFullMask, c) >> shift) & group_mask<G>();
            if (c) {
                const uint32_t at = cnt + __popc(m & below);
                g.kd[at] = d;
                g.ki[at] = j;
            }
            cnt += __popc(m);
        }
        __syncwarp();
        // all groups select together: one by itself would take as long
        if (__any_sync(kFullMask, live && cnt >= limit)) {
            group_select<G>(g, k, kKnnSlack, cnt, bound);
            if (cnt >= k) limit = g.cap - kGroupBatch;
        }
        if (live) {
            live = false;
            while (sp > 0) {
                sp--;
                if (g.sd[sp] <= bound) {
                    l = g.sl[sp];
                    r = g.sr[sp];
                    if (r > l) {
                        live = true;
                        break;
                    }
                }
            }
        }
        __syncwarp();
    }
    if (__any_sync(kFullMask, cnt > k + slack)) group_select<G>(g, k, slack, cnt, bound);
    return cnt;
}

// Scene::combinePhotonContributions (Scene.cu:607-635) at point p with shading normal nn and
// world outgoing direction wo_w, for a group: sum over the k nearest photons of
// power * f(wo, -dir)|cos| (SurfaceInteraction::lightScattered, SurfaceInteraction.cu:278-292)
// / (pi * maxDist^2). The reference weights each photon by |cos| although the photon density
// already carries the projected-area factor; with compat = false the estimate uses f alone
// (the radiance estimate of photon mapping). The cnt terms (tree slots) are summed lane-parallel. Returns
// the estimate on every lane of the group.
template <uint32_t G>
__device__ __forceinline__ V3 photon_density(const PhotonTree &t, const Bsdf &bs, V3 p, V3 nn, V3 wo_w, bool compat,
                                             const uint32_t *slots, uint32_t cnt)
{
    V3 tt, b;
    onb(nn, tt, b);
    const V3 wo = v3(dot(wo_w, tt), dot(wo_w, b), dot(wo_w, nn));
    V3 sum = v3(0, 0, 0);
    float maxd = 0.f;
    for (uint32_t j = threadIdx.x & (G - 1u); j < cnt; j += G) {
        const uint32_t s = slots[j];
        const float4 pp = __ldg(t.pos + s), pw = __ldg(t.pw + s), pd = __ldg(t.dir + s);
        maxd = fmaxf(maxd, length(v3(pp.x, pp.y, pp.z) - p));
        const V3 w = -v3(pd.x, pd.y, pd.z);
        const V3 wl = v3(dot(w, tt), dot(w, b), dot(w, nn));
        float pdf;
        V3 f = bsdf_eval(bs, wo, wl, pdf);
        if (!compat) {
            const float c = abs_cos(wl);
            f = c > 0 ? f * (1.0f / c) : v3(0, 0, 0);
        }
        sum = sum + v3(pw.x, pw.y, pw.z) * f;
    }
    __syncwarp();
    sum = v3(group_sum<G>(sum.x), group_sum<G>(sum.y), group_sum<G>(sum.z));
    maxd = group_max<G>(maxd);
    if (cnt == 0) return v3(0, 0, 0);
    return sum * (1.0f / (kPi * maxd * maxd));
}

// The estimate of a group of G lanes (on = false: none), and of a whole warp.
template <uint32_t G = kGroup>
__device__ __forceinline__ V3 group_photon_density(const PhotonTree &t, const Bsdf &bs, V3 p, V3 nn, V3 wo_w, int32_t sid,
                                                   uint32_t k, float radius2, bool compat, bool on, const KnnGroup &g)
{
    float bound;
    const uint32_t cnt = group_knn<G>(t.pos, t.aux, t.n, p.x, p.y, p.z, sid, k, radius2, 0, on, g, bound);
    return photon_density<G>(t, bs, p, nn, wo_w, compat, g.ki, cnt);
}
__device__ __forceinline__ V3 warp_photon_density(const PhotonTree &t, const Bsdf &bs, V3 p, V3 nn, V3 wo_w, int32_t sid,
                                                  uint32_t k, float radius2, bool compat, KnnWarpScratch &sm)
{
    const uint32_t cnt = warp_knn(t, p.x, p.y, p.z, sid, k, radius2, sm);
    return photon_density<32>(t, bs, p, nn, wo_w, compat, sm.ki, cnt);
}

// Scene::combinePhotonsSubsurface (Scene.cu:667-701) at point p (shading normal nn, direction
// to the camera wo_w) of an SSMaterial m with diffuse colour kd (m's kd, times its texel at
// the point when it has a texture: SSMaterial::getBSSDFparameters, SSMaterial.cu:245-263), for a warp. Over the photons within `radius` on the
// same shape (nn::KDTree::nearest_neighbors with an unbounded k, as
// Scene::search_nearest(p, radius, (ulong)-1, shapeId) calls it, Scene.cu:808-813): sum of
// power * kd * diffusionTermBSSRDF (geometricMath.cu:503-522:
// Rd * (1 - F(cos_o)) * (1 - F(cos_i)) / pi) / (2 pi maxDist^2). With no photon the reference
// divides 0 by 0 (a NaN sample, which the film drops); `compat` keeps that, otherwise 0. The
// terms are summed lane-parallel. Returns the estimate on every lane.
__device__ __forceinline__ V3 warp_photon_subsurface(const PhotonTree &t, const rt_material &m, V3 kd, V3 p, V3 nn,
                                                     V3 wo_w, int32_t sid, float radius2, bool compat,
                                                     PhotonWarpScratch &sm)
{
    const float eta = m.ior, g = m.roughness[1];
    const float cos_o = dot(nn, wo_w) / (length(nn) * length(wo_w));
    const float ft_o = 1.f - fresnel_dielectric_ref(cos_o, 1.f, eta);
    const DipoleChannel d0 = dipole_setup(m.eta[0], m.extra[0], g, eta), d1 = dipole_setup(m.eta[1], m.extra[1], g, eta),
                        d2 = dipole_setup(m.eta[2], m.extra[2], g, eta);
    V3 sum = v3(0, 0, 0);
    float maxd2 = 0.f;
    uint32_t cnt = 0, held = 0;
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    auto add = [&](uint32_t e) {  // entry e of the photons found
        const float4 pw = __ldg(t.pw + sm.slot[e]);
        const float r2 = sm.d2[e];
        maxd2 = fmaxf(maxd2, r2);
        const float sc = kInvPi * (1.f - fresnel_dielectric_ref(pw.w, 1.f, eta)) * ft_o;
        const V3 rd = v3(dipole_eval(d0, r2), dipole_eval(d1, r2), dipole_eval(d2, r2));
        sum = sum + rd * sc * v3(pw.x, pw.y, pw.z) * kd;
    };
    // photons within the radius are collected and added 32 at a time: where they were found, most of the
    // lanes waited for the few whose photons lay within it
    warp_traverse<kRadiusScan>(t, p.x, p.y, p.z, sm, [&]() { return radius2; },
                               [&](bool valid, float dist2, int shape, uint32_t s) {
        const bool ok = valid && dist2 <= radius2 && (sid == -1 || shape == sid);
        const unsigned found = __ballot_sync(kFullMask, ok);
        if (!found) return;
        if (ok) {
            const uint32_t at = held + __popc(found & below);
            sm.d2[at] = dist2;
            sm.slot[at] = s;
        }
        cnt += __popc(found);
        held += __popc(found);
        __syncwarp();
        if (held >= 32) {
            held -= 32;
            add(held + lane);
            __syncwarp();
        }
    });
    if (lane < held) add(lane);
    __syncwarp();
    if (cnt == 0) return compat ? v3(NAN, NAN, NAN) : v3(0, 0, 0);
    sum = v3(warp_sum(sum.x), warp_sum(sum.y), warp_sum(sum.z));
    const float maxd = __fsqrt_rn(warp_max(maxd2));
    return sum * (1.f / (2.f * kPi * maxd * maxd));
}

}  // namespace rtb
