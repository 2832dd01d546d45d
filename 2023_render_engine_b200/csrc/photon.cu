// Photon tracing, the photon-map kd-tree and k-nearest-neighbour gathering (sm_100a).
//
// Tracing (integration/photonDispersion.cu:26-192, Scene.cu:989-1026): photons start at
// the point lights and bounce as paths do in the renderer (same surfaces, BSDFs and Russian
// roulette, surface.cuh); at every hit on a scattering material a photon is stored. Paths
// run as waves (all photons of one bounce per wave, closest hits by the BVH8 kernel);
// stored photons are appended with a (path, depth) key and sorted by it at the end, so the
// photon order does not depend on scheduling.
//
// The kd-tree is the reference's implicit balanced tree (kdtree.h:78-108): the element at
// the middle of a range is the node, split on the axis of largest extent, built on the GPU
// (kdtree.cu), or on the host with the same partial ordering. Nearest-neighbour queries run on eight
// lanes each (k_knn_group), or on one thread with a bounded max-heap of the k best candidates in local
// memory (k_knn: few neighbours of many queries, and queries with equal distances).
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <new>
#include <thread>
#include <vector>

#include "photon_query.cuh"
#include "traverse.cuh"

namespace rtb {
namespace {

constexpr int kPB = 128;

struct PhotonBuffers {
    rt_ray *rays[2];
    float4 *beta[2];   // path throughput
    float4 *carry[2];  // carried light rgb, path index bits
    uint4 *rng[2];     // rng state lo/hi, -, depth
    rt_hit *hits;
    rt_photon *store;          // unsorted stored photons
    unsigned long long *keys;  // (path << 8) | depth
    uint32_t store_cap;
    uint32_t cap;
    uint32_t *queued;     // paths at each depth
    uint32_t *stored;     // photons stored
    uint32_t *trace_cnt;  // the walk's counters
};

__device__ __forceinline__ Pcg photon_rng(uint64_t path, uint32_t seed)
{
    return pcg_init((uint32_t)path, 0xFFFFFFFFu, seed ^ 0x9E3779B9u);
}

// Light choice proportional to power, as Scene::selectOneRandomLight (Scene.cu:421-438).
__global__ void k_select(RenderView rv, uint64_t n, uint32_t seed, const float *cdf_power, float total,
                         uint32_t *sel, unsigned long long *per_light)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Pcg r = photon_rng(i, seed);
    float u = pcg_float(r);
    uint32_t l = rv.nplights - 1;
    for (uint32_t k = 0; k < rv.nplights; k++) {
        u -= cdf_power[k] / total;
        if (u <= 0) {
            l = k;
            break;
        }
    }
    sel[i] = l;
    // one add per distinct light of the warp: every thread adding to one of a few counters
    // serialised the kernel (1.9 ms for 10M photons and two lights)
    const unsigned peers = __match_any_sync(__activemask(), l);
    if ((int)(threadIdx.x & 31u) == __ffs(peers) - 1) atomicAdd(per_light + l, (unsigned long long)__popc(peers));
}

// PointLight::sampleLight(sampler, n) (PointLight.cu:68-95) and the selection-pdf division
// (Scene.cu:1008-1012): power = I * 4 pi / n_l / p_l, direction uniform on the sphere.
__global__ void k_emit(RenderView rv, uint64_t n, uint32_t seed, const float *power, float total,
                       const uint32_t *sel, const unsigned long long *per_light, PhotonBuffers pb)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Pcg r = photon_rng(i, seed);
    (void)pcg_float(r);  // the selection sample
    const uint32_t l = sel[i];
    float u1 = pcg_float(r), u2 = pcg_float(r);
    float phi = 2 * kPi * u1;
    float th = acosf(2 * u2 - 1);
    float st, ct, sp, cp;
    sincosf(th, &st, &ct);
    sincosf(phi, &sp, &cp);
    V3 d = v3(st * cp, st * sp, ct);
    float4 lp = rv.plights[2 * l], li = rv.plights[2 * l + 1];
    const float pl = power[l] / total;
    const float scale = (4 * kPi) / (float)per_light[l] / pl;
    const uint32_t q = (uint32_t)i;
    reinterpret_cast<float4 *>(pb.rays[0])[2 * q] = make_float4(lp.x, lp.y, lp.z, INFINITY);
    reinterpret_cast<float4 *>(pb.rays[0])[2 * q + 1] = make_float4(d.x, d.y, d.z, 0.f);
    pb.beta[0][q] = make_float4(1.f, 1.f, 1.f, 0.f);
    pb.carry[0][q] = make_float4(li.x * scale, li.y * scale, li.z * scale, __uint_as_float((uint32_t)i));
    pb.rng[0][q] = make_uint4((uint32_t)r.state, (uint32_t)(r.state >> 32), 0u, 0u);
}

// One bounce of the paths at `depth0`, whose hits the walk left (finish_fast). The paths that continue
// are the next depth's.
__global__ void __launch_bounds__(kPB) k_photon_shade(RenderView rv, PhotonBuffers pb, uint32_t depth0,
                                                      uint32_t max_depth, uint32_t rr_depth, uint32_t seed, uint32_t flags)
{
    const uint32_t n = min(pb.queued[depth0], pb.cap);
    const int cur = depth0 & 1, nxt = cur ^ 1;
    const bool compat = (flags & RT_RENDER_COMPAT) != 0;
    // the next walk's work counter; this depth's walk is over, and none of the replays below use it
    if (blockIdx.x == 0 && threadIdx.x == 0) pb.trace_cnt[3] = 0;
    if (blockIdx.x * blockDim.x < n) prefetch_shapes(rv.sv);
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const float4 hv = finish_fast(rv.sv, pb.rays[cur], q, RT_TRACE_FAST | kTraceRecords,
                                      reinterpret_cast<const float4 *>(pb.hits)[q], pb.trace_cnt);
        rt_hit h{hv.x, __float_as_int(hv.y), hv.z, hv.w};
        if (h.prim < 0) continue;  // escaped
        float4 r0 = reinterpret_cast<const float4 *>(pb.rays[cur])[2 * q];
        float4 r1 = reinterpret_cast<const float4 *>(pb.rays[cur])[2 * q + 1];
        float4 b4 = pb.beta[cur][q], c4 = pb.carry[cur][q];
        uint4 s4 = pb.rng[cur][q];
        V3 o = v3(r0.x, r0.y, r0.z), d = v3(r1.x, r1.y, r1.z);
        V3 beta = v3(b4.x, b4.y, b4.z), carry = v3(c4.x, c4.y, c4.z);
        const uint32_t path = __float_as_uint(c4.w);
        const uint32_t depth = s4.w;
        Pcg rng;
        rng.state = ((uint64_t)s4.y << 32) | s4.x;
        rng.inc = ((((uint64_t)0xFFFFFFFFu << 32) | (seed ^ 0x9E3779B9u)) << 1u) | 1u;
        Surface sf = surface_at(rv, h, o, d, compat);
        const rt_material &m = rv.mats[min(sf.mat, rv.nmats - 1)];
        Bsdf bs = load_bsdf(m);
        const bool scattering = is_scattering(bs);  // from the material's own kd
        if (m.texture) {
            const float2 uv = surface_uv(rv, h, sf);
            texture_bsdf(bs, tex_color(rv, m.texture - 1u, uv.x, uv.y));
        }
        if (scattering) {  // samplePhotonIntersections (photonDispersion.cu:40-54)
            uint32_t slot = append(pb.stored);
            if (slot < pb.store_cap) {
                V3 pw = carry * beta;
                rt_photon ph;
                ph.pos[0] = sf.p.x;
                ph.pos[1] = sf.p.y;
                ph.pos[2] = sf.p.z;
                ph.shape_id = sf.shape;
                ph.dir[0] = d.x;
                ph.dir[1] = d.y;
                ph.dir[2] = d.z;
                ph.path = path;
                ph.power[0] = pw.x;
                ph.power[1] = pw.y;
                ph.power[2] = pw.z;
                ph.depth = depth;
                ph.normal[0] = sf.n.x;
                ph.normal[1] = sf.n.y;
                ph.normal[2] = sf.n.z;
                ph.reserved = 0.f;
                pb.store[slot] = ph;
                pb.keys[slot] = ((unsigned long long)path << 8) | depth;
            }
        }
        V3 t, bv;
        onb(sf.n, t, bv);
        V3 wow = -d;
        V3 wo = v3(dot(wow, t), dot(wow, bv), dot(wow, sf.n));
        V3 Le = (bs.type == RT_MAT_LIGHT) ? bs.color * m.intensity : v3(0, 0, 0);
        V3 wi;
        float pdf;
        bool delta;
        V3 f = bsdf_sample(bs, wo, rng, compat, wi, pdf, delta);
        carry = carry + beta * Le;  // photonDispersion.cu:64-65
        beta = beta * f;
        bool finished = is_black(f);
        if (!finished && scattering && depth > rr_depth) {  // finishStep (pathTracing.cu:91-102)
            float qrr = fmaxf(0.05f, 1.f - luminance(beta));
            if (pcg_float(rng) < qrr)
                finished = true;
            else
                beta = beta * (1.f / (1.f - qrr));
        }
        if (finished || depth + 1 >= max_depth) continue;
        V3 wiw = t * wi.x + bv * wi.y + sf.n * wi.z;
        V3 no = spawn_origin(sf.p, sf.n, sf.perr, wiw);
        uint32_t qn = append(pb.queued + depth0 + 1);
        reinterpret_cast<float4 *>(pb.rays[nxt])[2 * qn] = make_float4(no.x, no.y, no.z, INFINITY);
        reinterpret_cast<float4 *>(pb.rays[nxt])[2 * qn + 1] = make_float4(wiw.x, wiw.y, wiw.z, 0.f);
        pb.beta[nxt][qn] = make_float4(beta.x, beta.y, beta.z, 0.f);
        pb.carry[nxt][qn] = make_float4(carry.x, carry.y, carry.z, __uint_as_float(path));
        pb.rng[nxt][qn] = make_uint4((uint32_t)rng.state, (uint32_t)(rng.state >> 32), 0u, depth + 1);
    }
}

__global__ void k_gather_photons(const rt_photon *src, const uint32_t *order, uint64_t n, rt_photon *dst)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[order[i]];
}

__global__ void k_iota(uint32_t *v, uint64_t n)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = (uint32_t)i;
}

// ------------------------------------------------------------------- kNN

// Mark in a query's count: it has equal distances and waits for the reference's heap (k is at most 128).
constexpr uint32_t kKnnTied = 0x80000000u;

// One thread per query, the reference's own heap. tied_only: only for the queries that k_knn_group marked.
__global__ void __launch_bounds__(128) k_knn(const float4 *__restrict__ node_pos, const int2 *__restrict__ node_aux,
                                             uint32_t n, const float *__restrict__ queries,
                                             const int32_t *__restrict__ qshape, uint64_t nq, uint32_t k,
                                             float radius, bool tied_only, int32_t *__restrict__ out_idx,
                                             float *__restrict__ out_dist, uint32_t *__restrict__ out_count)
{
    const uint64_t qi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (qi >= nq || (tied_only && !(out_count[qi] & kKnnTied))) return;
    float hd[kKnnMaxK];
    int32_t hi[kKnnMaxK];
    const uint32_t cnt = knn_query(node_pos, node_aux, n, queries[3 * qi], queries[3 * qi + 1], queries[3 * qi + 2],
                                   qshape ? qshape[qi] : -1, k, radius, hd, hi);
    heap_to_sorted(hd, hi, cnt);
    for (uint32_t j = 0; j < k; j++) {
        out_idx[qi * k + j] = j < cnt ? hi[j] : -1;
        if (out_dist) out_dist[qi * k + j] = j < cnt ? hd[j] : INFINITY;
    }
    out_count[qi] = cnt;
}

// The reference's own query for one thread, its heap in hd / hi (k entries).
__device__ __noinline__ static uint32_t knn_serial(const float4 *node_pos, const int2 *node_aux, uint32_t n, float qx,
                                                   float qy, float qz, int32_t sid, uint32_t k, float radius, float *hd,
                                                   int32_t *hi)
{
    const uint32_t cnt = knn_query(node_pos, node_aux, n, qx, qy, qz, sid, k, radius, hd, hi);
    heap_to_sorted(hd, hi, cnt);
    return cnt;
}

// Few neighbours of many queries are found faster by a thread each: the heap is then in registers and
// cache, and the threads fill the device. Measured in 500,000 points, us by thread / by group of lanes:
// 200,003 queries k = 1: 224 / 406, 4: 365 / 465, 8: 543 / 529; 50,000 queries k = 1: 133 / 148,
// 2: 160 / 155, 4: 212 / 166; 10,000 queries k = 1: 111 / 78. In 1,000 points the lines lie alike.
inline bool knn_by_thread(uint32_t k, uint64_t nq) { return k <= 8 && nq >= 25000ull * k; }

// k-nearest queries, kGroup lanes each: group_knn finds the candidates, each lane then ranks its own
// by counting. Where no two distances are equal that is the only answer; otherwise the order, and at
// the k-th distance the choice, are those of the reference's heap, which one lane then runs on the
// host's tree (exact_pos, exact_aux; a few queries in ten thousand on scattered points). Without that
// tree (exact_pos null) the query is marked in its count, and *any_tied set.
// 500,000 points, 200,003 queries, k = 50: 3.10 ms one query per thread, 1.30 ms so.
constexpr int kQueryBlock = 128;
__global__ void __launch_bounds__(kQueryBlock) k_knn_group(const float4 *__restrict__ node_pos,
                                                           const int2 *__restrict__ node_aux,
                                                           const float4 *__restrict__ exact_pos,
                                                           const int2 *__restrict__ exact_aux, uint32_t n,
                                                           const float *__restrict__ queries,
                                                           const int32_t *__restrict__ qshape, uint64_t nq, uint32_t k,
                                                           float radius, float radius2, int32_t *__restrict__ out_idx,
                                                           float *__restrict__ out_dist, uint32_t *__restrict__ out_count,
                                                           uint32_t *any_tied)
{
    extern __shared__ __align__(16) uint32_t knn_smem[];
    const KnnGroup g = knn_group(knn_smem + (threadIdx.x >> 5) * 4 * knn_words(k), k);
    const uint64_t qi = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / kGroup;
    const uint32_t lane = threadIdx.x & (kGroup - 1u), shift = threadIdx.x & 31u & ~(kGroup - 1u);
    const bool on = qi < nq;
    const float qx = on ? queries[3 * qi] : 0.f, qy = on ? queries[3 * qi + 1] : 0.f, qz = on ? queries[3 * qi + 2] : 0.f;
    const int32_t sid = on && qshape ? qshape[qi] : -1;
    float bound;
    const uint32_t cnt = group_knn(node_pos, node_aux, n, qx, qy, qz, sid, k, radius2, kKnnSlack, on, g, bound);
    uint32_t ranks = 0;
    bool tied = false;
    for (uint32_t e = lane; e < cnt; e += kGroup) {
        const float d2 = g.kd[e];
        tied |= cnt >= k && bound < radius2 && __float_as_int(bound) - __float_as_int(d2) < kRootSteps;
        g.kd[e] = __fsqrt_rn(d2);
    }
    if (lane < 4) g.kd[cnt + lane] = INFINITY;  // the last step of the loop below
    __syncwarp();
    for (uint32_t e = lane; e < cnt; e += kGroup) {
        const float d = g.kd[e];
        uint32_t rank = 0;
        for (uint32_t j = 0; j < cnt; j += 4) {
            const float4 x = *reinterpret_cast<const float4 *>(g.kd + j);
            rank += (x.x < d) + (x.y < d) + (x.z < d) + (x.w < d);
        }
        ranks += rank;
        if (rank < k) {
            out_idx[qi * k + rank] = __ldg(&node_aux[g.ki[e]].y);
            if (out_dist) out_dist[qi * k + rank] = d;
        }
    }
    __syncwarp();
    // equal distances share a rank
    tied |= group_sum<kGroup>(ranks) != cnt * (cnt - 1) / 2;
    tied = ((__ballot_sync(kFullMask, tied) >> shift) & 0xFFu) != 0;
    if (!on) return;
    const uint32_t found = min(cnt, k);
    if (lane == 0) {
        const bool wait = tied && !exact_pos;
        out_count[qi] = found | (wait ? kKnnTied : 0u);
        if (wait) {
            *any_tied = 1;
        } else if (tied) {
            int32_t *hi = reinterpret_cast<int32_t *>(g.ki);
            knn_serial(exact_pos, exact_aux, n, qx, qy, qz, sid, k, radius, g.kd, hi);
            for (uint32_t j = 0; j < found; j++) {
                out_idx[qi * k + j] = hi[j];
                if (out_dist) out_dist[qi * k + j] = g.kd[j];
            }
        }
    }
    for (uint32_t j = found + lane; j < k; j += kGroup) {
        out_idx[qi * k + j] = -1;
        if (out_dist) out_dist[qi * k + j] = INFINITY;
    }
}

// Resident blocks per SM of the subsurface kernel (64 registers): 4.5 / 4.5 / 5.1 M queries/s for no
// bound (80 registers) / 6 / 8, on a 2.1M-photon map.
#ifndef RTB_QUERY_MIN_BLOCKS
#define RTB_QUERY_MIN_BLOCKS 8
#endif

// The photons' shading attributes in tree-slot order, so that a query reads them with the
// positions it scans: power and cos(normal, -direction) (the photon's factor of
// diffusionTermBSSRDF, geometricMath.cu:503-522), and the arrival direction.
__global__ void k_tree_attrs(const int2 *__restrict__ node_aux, const rt_photon *__restrict__ photons, uint64_t n,
                             float4 *__restrict__ pw, float4 *__restrict__ dir)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const rt_photon ph = photons[node_aux[i].y];
    const V3 pn = v3(ph.normal[0], ph.normal[1], ph.normal[2]);
    const V3 wi = -v3(ph.dir[0], ph.dir[1], ph.dir[2]);
    const float cos_i = dot(pn, wi) / (length(pn) * length(wi));
    pw[i] = make_float4(ph.power[0], ph.power[1], ph.power[2], cos_i);
    dir[i] = make_float4(ph.dir[0], ph.dir[1], ph.dir[2], 0.f);
}


// Lanes per query of k_density, of n photons: a query's own time counts where there are few, the instructions
// all of them take where there are many, and their buffers' shared memory at large k. us by 32 / 16 / 8
// lanes, 830,000 photons: 1,000 queries of 50 151 / 181 / 218, 12,000 of 50 220 / 239 / 291, 20,000 of 50
// 278 / 268 / 299, 50,000 of 50 541 / 461 / 453, of 128 681 / 628 / 709; 20,000 photons: 4,000 of 50
// 63 / 62 / 75, 8,000 of 50 89 / 75 / 79, 12,000 of 50 115 / 98 / 85, of 128 150 / 142 / 171.
inline uint32_t density_lanes(uint64_t n, uint32_t k, uint64_t nq)
{
    const bool large = n >= 1u << 17;  // beyond the L1 caches
    if (nq <= (large ? 14000u : 6000u)) return 32;
    return k > 110 || (k > 85 && nq > 14000 && nq < 20000) || nq <= (large ? 40000u : 10000u) ? 16 : kGroup;
}

// Scene::combinePhotonContributions (Scene.cu:607-635) per query: the k nearest photons on
// the same shape within radius, sum of power * lightScattered(-photon direction), divided by
// pi * (largest neighbour distance)^2.
template <uint32_t G>
__global__ void __launch_bounds__(kQueryBlock, G == 32 ? 8 : kGatherBlocks) k_density(PhotonTree tree, rt_material mat,
                                                                       const float *__restrict__ pts,
                                                                       const float *__restrict__ nrm,
                                                                       const float *__restrict__ wo,
                                                                       const int32_t *__restrict__ shape, uint64_t nq,
                                                                       uint32_t k, float radius2, float *__restrict__ out)
{
    extern __shared__ __align__(16) uint32_t knn_smem[];
    const uint64_t qi = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const bool on = qi < nq;
    const uint64_t i = on ? qi : nq - 1;
    V3 p = v3(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
    V3 nn = normalize(v3(nrm[3 * i], nrm[3 * i + 1], nrm[3 * i + 2]));
    V3 w = v3(wo[3 * i], wo[3 * i + 1], wo[3 * i + 2]);
    const int32_t sid = shape ? shape[i] : -1;
    V3 c;
    if (G == 32)
        c = warp_photon_density(tree, load_bsdf(mat), p, nn, w, sid, k, radius2, true,
                                reinterpret_cast<KnnWarpScratch *>(knn_smem)[threadIdx.x >> 5]);
    else
        c = group_photon_density<G>(tree, load_bsdf(mat), p, nn, w, sid, k, radius2, true, on,
                                    knn_group<G>(knn_smem + (threadIdx.x >> 5) * (32 / G) * knn_words(k), k));
    if (on && (threadIdx.x & (G - 1u)) == 0) {
        out[3 * qi] = c.x;
        out[3 * qi + 1] = c.y;
        out[3 * qi + 2] = c.z;
    }
}

__global__ void __launch_bounds__(kQueryBlock, RTB_QUERY_MIN_BLOCKS) k_subsurface(PhotonTree tree, rt_material mat,
                                                            const float *__restrict__ pts,
                                                            const float *__restrict__ nrm,
                                                            const float *__restrict__ wo,
                                                            const int32_t *__restrict__ shape, uint64_t nq,
                                                            float radius2, int compat, float *__restrict__ out)
{
    __shared__ PhotonWarpScratch scratch[kQueryBlock / 32];
    const uint64_t qi = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (qi >= nq) return;  // warp-uniform
    const V3 p = v3(pts[3 * qi], pts[3 * qi + 1], pts[3 * qi + 2]);
    const V3 nn = v3(nrm[3 * qi], nrm[3 * qi + 1], nrm[3 * qi + 2]);
    const V3 w = v3(wo[3 * qi], wo[3 * qi + 1], wo[3 * qi + 2]);
    const V3 c = warp_photon_subsurface(tree, mat, v3(mat.color[0], mat.color[1], mat.color[2]), p, nn, w,
                                        shape ? shape[qi] : -1, radius2, compat != 0, scratch[threadIdx.x >> 5]);
    if ((threadIdx.x & 31u) == 0) {
        out[3 * qi] = c.x;
        out[3 * qi + 1] = c.y;
        out[3 * qi + 2] = c.z;
    }
}

// ---------------------------------------------------- host kd-tree build

struct KdElem {
    float p[3];
    int32_t shape;
    uint32_t idx;
};

// build_tree (kdtree.h:78-103): bounding box of the range, axis of largest extent (first
// axis on ties), std::nth_element at the middle, recurse on both halves.
void kd_build(std::vector<KdElem> &e, std::vector<uint8_t> &axis, size_t left, size_t right, int depth)
{
    if (right - left <= 1) return;
    float lo[3], hi[3];
    for (int c = 0; c < 3; c++) lo[c] = hi[c] = e[left].p[c];
    for (size_t i = left + 1; i < right; i++)
        for (int c = 0; c < 3; c++) {
            if (lo[c] > e[i].p[c]) lo[c] = e[i].p[c];
            if (hi[c] < e[i].p[c]) hi[c] = e[i].p[c];
        }
    const size_t median = (right + left) / 2;
    int ax = 0;
    float mx = hi[0] - lo[0];
    for (int c = 1; c < 3; c++)
        if (hi[c] - lo[c] > mx) {
            ax = c;
            mx = hi[c] - lo[c];
        }
    std::nth_element(e.begin() + left, e.begin() + median, e.begin() + right,
                     [ax](const KdElem &a, const KdElem &b) { return a.p[ax] < b.p[ax]; });
    axis[median] = (uint8_t)ax;
    if (right - left > 400000 && depth < 4) {
        std::thread t([&, left, median, depth]() { kd_build(e, axis, left, median, depth + 1); });
        kd_build(e, axis, median + 1, right, depth + 1);
        t.join();
    } else {
        kd_build(e, axis, left, median, depth + 1);
        kd_build(e, axis, median + 1, right, depth + 1);
    }
}

void map_context(rt_photon_map *m, rt_context *ctx)
{
    m->ctx = ctx;
    for (DevBuf *b : {&m->photons, &m->node_pos, &m->node_aux, &m->node_pw, &m->node_dir, &m->exact_pos, &m->exact_aux, &m->any_tied})
        b->ctx = ctx;
}

// The host build of a map's tree, uploaded to pos and aux.
int kd_build_host(rt_photon_map *m, DevBuf &pos, DevBuf &aux) try {
    cudaStream_t st = m->ctx->stream;
    const uint64_t n = m->n;
    std::vector<rt_photon> ph(n);
    if (n) {
        RTB_CUDA(cudaMemcpyAsync(ph.data(), m->photons.ptr, n * sizeof(rt_photon), cudaMemcpyDeviceToHost, st));
        RTB_CUDA(cudaStreamSynchronize(st));
    }
    std::vector<KdElem> e(n);
    for (uint64_t i = 0; i < n; i++) {
        e[i].p[0] = ph[i].pos[0];
        e[i].p[1] = ph[i].pos[1];
        e[i].p[2] = ph[i].pos[2];
        e[i].shape = ph[i].shape_id;
        e[i].idx = (uint32_t)i;
    }
    std::vector<uint8_t> axis(n, 0);
    kd_build(e, axis, 0, n, 0);
    std::vector<float4> np(n);
    std::vector<int2> na(n);
    for (uint64_t i = 0; i < n; i++) {
        uint32_t ax = axis[i];
        float axf;
        std::memcpy(&axf, &ax, 4);
        np[i] = make_float4(e[i].p[0], e[i].p[1], e[i].p[2], axf);
        na[i] = make_int2(e[i].shape, (int)e[i].idx);
    }
    RTB_CHECK(pos.upload(np.data(), n * sizeof(float4), st));
    RTB_CHECK(aux.upload(na.data(), n * sizeof(int2), st));
    RTB_CUDA(cudaStreamSynchronize(st));
    return RT_OK;
} catch (const std::bad_alloc &) {
    return fail(RT_ERR_OOM, "photon map: no host memory for the tree");
}

// That tree, where the map's own is not it: built when a query first needs it.
int exact_tree(rt_photon_map *m)
{
    std::lock_guard<std::mutex> lk(m->exact_mu);
    if (!m->exact) RTB_CHECK(kd_build_host(m, m->exact_pos, m->exact_aux));
    m->exact = true;
    return RT_OK;
}

}  // namespace
}  // namespace rtb

using namespace rtb;

extern "C" {

int rt_photon_map_destroy(rt_photon_map *m)
{
    if (!m) return RT_OK;
    cudaSetDevice(m->ctx->device);
    cudaStreamSynchronize(m->ctx->stream);
    m->photons.release();
    m->node_pos.release();
    m->node_aux.release();
    m->node_pw.release();
    m->node_dir.release();
    delete m;
    return RT_OK;
}

int rt_photon_map_count(rt_photon_map *m, uint64_t *n)
{
    if (!m || !n) return fail(RT_ERR_INVALID, "rt_photon_map_count: null argument");
    *n = m->n;
    return RT_OK;
}

int rt_photon_map_get(rt_photon_map *m, uint64_t first, uint64_t n, rt_photon *out)
{
    if (!m || (!out && n)) return fail(RT_ERR_INVALID, "rt_photon_map_get: null argument");
    if (first + n > m->n) return fail(RT_ERR_INVALID, "rt_photon_map_get: range out of bounds");
    if (n == 0) return RT_OK;
    RTB_CUDA(cudaSetDevice(m->ctx->device));
    RTB_CUDA(cudaMemcpyAsync(out, m->photons.as<rt_photon>() + first, n * sizeof(rt_photon), cudaMemcpyDeviceToHost,
                             m->ctx->stream));
    RTB_CUDA(cudaStreamSynchronize(m->ctx->stream));
    return RT_OK;
}

int rt_photon_map_from_points(rt_context *ctx, const float *pos, const int32_t *shape, uint64_t n,
                              rt_photon_map **out)
{
    if (!ctx || !out || (!pos && n)) return fail(RT_ERR_INVALID, "rt_photon_map_from_points: null argument");
    if (n >= 0xFFFFFFFFull) return fail(RT_ERR_INVALID, "rt_photon_map_from_points: too many points");
    RTB_CUDA(cudaSetDevice(ctx->device));
    std::vector<float> hp(3 * n);
    std::vector<int32_t> hs(n, -1);
    if (n) {
        RTB_CUDA(cudaMemcpyAsync(hp.data(), pos, 12 * n, cudaMemcpyDeviceToHost, ctx->stream));
        if (shape) RTB_CUDA(cudaMemcpyAsync(hs.data(), shape, 4 * n, cudaMemcpyDeviceToHost, ctx->stream));
        RTB_CUDA(cudaStreamSynchronize(ctx->stream));
    }
    std::vector<rt_photon> ph(n);
    for (uint64_t i = 0; i < n; i++) {
        std::memset(&ph[i], 0, sizeof(rt_photon));
        ph[i].pos[0] = hp[3 * i];
        ph[i].pos[1] = hp[3 * i + 1];
        ph[i].pos[2] = hp[3 * i + 2];
        ph[i].shape_id = hs[i];
        ph[i].path = (uint32_t)i;
    }
    rt_photon_map *m = new rt_photon_map();
    map_context(m, ctx);
    m->n = n;
    m->points = true;
    int st = m->photons.upload(ph.data(), n * sizeof(rt_photon), ctx->stream);
    if (st != RT_OK) {
        delete m;
        return st;
    }
    *out = m;
    return RT_OK;
}

int rt_photon_map_build(rt_photon_map *m)
{
    if (!m) return fail(RT_ERR_INVALID, "rt_photon_map_build: null map");
    RTB_CUDA(cudaSetDevice(m->ctx->device));
    cudaStream_t st = m->ctx->stream;
    const uint64_t n = m->n;
    std::lock_guard<std::mutex> lk(m->exact_mu);
    m->exact = m->host_order = false;
    RTB_CHECK(m->any_tied.reserve(4));
    RTB_CUDA(cudaMemsetAsync(m->any_tied.ptr, 0, 4, st));
    RTB_CHECK(m->node_pos.reserve(std::max<uint64_t>(n, 1) * sizeof(float4)));
    RTB_CHECK(m->node_aux.reserve(std::max<uint64_t>(n, 1) * sizeof(int2)));
    RTB_CHECK(m->node_pw.reserve(std::max<uint64_t>(n, 1) * sizeof(float4)));
    RTB_CHECK(m->node_dir.reserve(std::max<uint64_t>(n, 1) * sizeof(float4)));
    // The host build where the device build gives no valid tree or finds no room for its workspace
    // (about 100 bytes per photon), and for a point set with equal coordinates, whose queries need
    // the host's order.
    uint32_t report = kKdNotFinite, ties = 0;
    if (n <= kKdDeviceMax) {
        const int rc = kd_build_device(m->ctx, m->photons.as<rt_photon>(), n, m->node_pos.as<float4>(),
                                       m->node_aux.as<int2>(), &report, &ties);
        if (rc == RT_ERR_OOM) {
            (void)cudaGetLastError();
            report = kKdNotFinite;
        } else if (rc != RT_OK) {
            return rc;
        }
    }
    // A query with equal distances is answered a second time, by one lane: not where they are the rule
    // (lattices).
    m->scattered = !(report & kKdNotFinite) && ties <= n / 64;
    if ((report & kKdNotFinite) || (m->points && (report & kKdTies))) {
        RTB_CHECK(kd_build_host(m, m->node_pos, m->node_aux));
        report = 0;
    }
    m->host_order = report == 0;
    if (n) {
        k_tree_attrs<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(m->node_aux.as<int2>(), m->photons.as<rt_photon>(), n,
                                                                 m->node_pw.as<float4>(), m->node_dir.as<float4>());
        RTB_CUDA(cudaGetLastError());
    }
    RTB_CUDA(cudaStreamSynchronize(st));
    m->built = true;
    return RT_OK;
}

int rt_photon_knn(rt_photon_map *m, const float *q, const int32_t *qs, uint64_t nq, uint32_t k, float radius,
                  int32_t *out_idx, float *out_dist, uint32_t *out_count)
{
    if (!m || (nq && (!q || !out_idx || !out_count))) return fail(RT_ERR_INVALID, "rt_photon_knn: null argument");
    if (!m->built) return fail(RT_ERR_STATE, "rt_photon_knn: map not built (rt_photon_map_build)");
    if (k == 0 || k > kKnnMaxK) return fail(RT_ERR_INVALID, "rt_photon_knn: k must be in [1, 128]");
    if (nq == 0) return RT_OK;
    RTB_CUDA(cudaSetDevice(m->ctx->device));
    cudaStream_t st = m->ctx->stream;
    const uint32_t n = (uint32_t)m->n;
    bool exact = m->host_order;  // the host's tree is there
    if (!exact) {
        if (!m->scattered) RTB_CHECK(exact_tree(m));
        std::lock_guard<std::mutex> lk(m->exact_mu);
        exact = m->exact;
    }
    const DevBuf &pos = m->host_order ? m->node_pos : m->exact_pos, &aux = m->host_order ? m->node_aux : m->exact_aux;
    auto by_thread = [&](bool tied_only) -> int {
        k_knn<<<(unsigned)((nq + 127) / 128), 128, 0, st>>>(pos.as<float4>(), aux.as<int2>(), n, q, qs, nq, k, radius,
                                                            tied_only, out_idx, out_dist, out_count);
        RTB_CUDA(cudaGetLastError());
        RTB_CUDA(cudaStreamSynchronize(st));
        return RT_OK;
    };
    if (!m->scattered || (exact && knn_by_thread(k, nq))) return by_thread(false);
    const uint64_t blocks = (nq * kGroup + kQueryBlock - 1) / kQueryBlock;
    k_knn_group<<<(unsigned)blocks, kQueryBlock, kQueryBlock / kGroup * 4 * knn_words(k), st>>>(
        m->node_pos.as<float4>(), m->node_aux.as<int2>(), exact ? pos.as<float4>() : nullptr, exact ? aux.as<int2>() : nullptr,
        n, q, qs, nq, k, radius, radius_squared(radius), out_idx, out_dist, out_count, m->any_tied.as<uint32_t>());
    RTB_CUDA(cudaGetLastError());
    // set once and for all by the first query with equal distances: from then on the host's tree is there
    uint32_t any_tied = 0;
    if (!exact) RTB_CUDA(cudaMemcpyAsync(&any_tied, m->any_tied.ptr, 4, cudaMemcpyDeviceToHost, st));
    RTB_CUDA(cudaStreamSynchronize(st));
    if (!any_tied) return RT_OK;
    RTB_CHECK(exact_tree(m));
    return by_thread(true);
}

int rt_photon_subsurface(rt_photon_map *m, const rt_material *mat, const float *pts, const float *nrm, const float *wo,
                         const int32_t *shape, uint64_t nq, float radius, uint32_t flags, float *out_rgb)
{
    if (!m || !mat) return fail(RT_ERR_INVALID, "rt_photon_subsurface: null argument");
    if (!m->built) return fail(RT_ERR_STATE, "rt_photon_subsurface: photon map not built");
    if (mat->type != RT_MAT_SUBSURFACE) return fail(RT_ERR_INVALID, "rt_photon_subsurface: not a subsurface material");
    if (nq == 0) return RT_OK;
    if (!pts || !nrm || !wo || !out_rgb) return fail(RT_ERR_INVALID, "rt_photon_subsurface: null buffer");
    RTB_CUDA(cudaSetDevice(m->ctx->device));
    if (nq > (1ull << 31) / 32) return fail(RT_ERR_INVALID, "rt_photon_subsurface: nq must be at most 2^26");
    const uint64_t blocks = (nq * 32 + kQueryBlock - 1) / kQueryBlock;
    k_subsurface<<<(unsigned)blocks, kQueryBlock, 0, m->ctx->stream>>>(photon_tree(m), *mat, pts, nrm, wo, shape, nq,
                                                                       radius_squared(radius),
                                                                       (flags & RT_RENDER_COMPAT) ? 1 : 0,
                                                                       out_rgb);
    RTB_CUDA(cudaGetLastError());
    RTB_CUDA(cudaStreamSynchronize(m->ctx->stream));
    return RT_OK;
}

int rt_photon_density(rt_photon_map *m, const rt_material *mat, const float *pts, const float *nrm, const float *wo,
                      const int32_t *shape, uint64_t nq, uint32_t k, float radius, float *out_rgb)
{
    if (!m || !mat || (nq && (!pts || !nrm || !wo || !out_rgb)))
        return fail(RT_ERR_INVALID, "rt_photon_density: null argument");
    if (!m->built) return fail(RT_ERR_STATE, "rt_photon_density: map not built (rt_photon_map_build)");
    if (k == 0 || k > kKnnMaxK) return fail(RT_ERR_INVALID, "rt_photon_density: k must be in [1, 128]");
    if (nq == 0) return RT_OK;
    RTB_CUDA(cudaSetDevice(m->ctx->device));
    if (nq > (1ull << 31) / 32) return fail(RT_ERR_INVALID, "rt_photon_density: nq must be at most 2^26");
    auto launch = [&](auto kernel, uint32_t lanes) {
        const uint64_t blocks = (nq * lanes + kQueryBlock - 1) / kQueryBlock;
        const size_t smem = lanes == 32 ? kQueryBlock / 32 * sizeof(KnnWarpScratch)
                                        : kQueryBlock / lanes * 4 * (size_t)knn_words(k);
        kernel<<<(unsigned)blocks, kQueryBlock, smem, m->ctx->stream>>>(photon_tree(m), *mat, pts, nrm, wo, shape, nq, k,
                                                                       radius_squared(radius), out_rgb);
    };
    switch (density_lanes(m->n, k, nq)) {
    case 32: launch(k_density<32>, 32); break;
    case 16: launch(k_density<16>, 16); break;
    default: launch(k_density<kGroup>, kGroup);
    }
    RTB_CUDA(cudaGetLastError());
    RTB_CUDA(cudaStreamSynchronize(m->ctx->stream));
    return RT_OK;
}

int rt_photons_trace(rt_scene *s, uint64_t n, uint32_t max_depth, uint32_t rr_depth, uint32_t seed, uint32_t flags,
                     rt_photon_map **out, rt_photon_trace_stats *stats)
{
    if (!s || !out) return fail(RT_ERR_INVALID, "rt_photons_trace: null argument");
    if (s->merged) return fail(RT_ERR_UNSUPPORTED, "rt_photons_trace: not available on a merged scene");
    if (!s->committed) return fail(RT_ERR_STATE, "rt_photons_trace: scene not committed");
    if (n == 0 || n >= (1ull << 31)) return fail(RT_ERR_INVALID, "rt_photons_trace: n must be in [1, 2^31)");
    if (max_depth == 0 || max_depth > 255) return fail(RT_ERR_INVALID, "rt_photons_trace: max_depth in [1, 255]");
    if (s->plights.empty()) return fail(RT_ERR_STATE, "rt_photons_trace: the scene has no point lights");
    RTB_CUDA(cudaSetDevice(s->ctx->device));
    cudaStream_t st = s->ctx->stream;
    RenderView rv;
    RTB_CHECK(make_render_view(s, rv));
    const uint32_t nl = (uint32_t)s->plight_rgbi.size();
    std::vector<float> power(nl);
    float total = 0.f;
    for (uint32_t l = 0; l < nl; l++) {  // sum(Light::power()) = sum(color * I * 4 pi) (PointLight.cu:40-43)
        const auto &p = s->plight_rgbi[l];
        power[l] = (p.r * p.i * 4.0f * kPi) + (p.g * p.i * 4.0f * kPi) + (p.b * p.i * 4.0f * kPi);
        total += power[l];
    }
    if (!(total > 0)) return fail(RT_ERR_STATE, "rt_photons_trace: lights have no power");
    const uint32_t cap = (uint32_t)n;
    rt_context *ctx = s->ctx;  // buffers of its pool, freed on return
    DevBuf rays[2]{DevBuf(ctx), DevBuf(ctx)}, beta[2]{DevBuf(ctx), DevBuf(ctx)}, carry[2]{DevBuf(ctx), DevBuf(ctx)},
        rng[2]{DevBuf(ctx), DevBuf(ctx)}, hits(ctx), sel(ctx), perl(ctx), dpow(ctx), cnt(ctx);
    for (int b = 0; b < 2; b++) {
        RTB_CHECK(rays[b].reserve(32ull * cap));
        RTB_CHECK(beta[b].reserve(16ull * cap));
        RTB_CHECK(carry[b].reserve(16ull * cap));
        RTB_CHECK(rng[b].reserve(16ull * cap));
    }
    RTB_CHECK(hits.reserve(16ull * cap));
    RTB_CHECK(sel.reserve(4ull * cap));
    RTB_CHECK(perl.reserve(8ull * nl));
    RTB_CHECK(dpow.upload(power.data(), 4ull * nl, st));
    // paths at each depth (max_depth <= 255), photons stored
    constexpr uint32_t kStored = 256, kCounts = 257;
    RTB_CHECK(cnt.reserve(4 * kCounts));
    RTB_CHECK(s->scratch.counters.reserve(64));
    uint64_t store_cap = std::max<uint64_t>(4 * n, 1024);
    rt_photon_map *m = nullptr;
    cudaEvent_t e0, e1;
    RTB_CUDA(cudaEventCreate(&e0));
    RTB_CUDA(cudaEventCreate(&e1));
    uint64_t stored = 0, rays_traced = 0;
    for (int attempt = 0; attempt < 2; attempt++) {
        DevBuf store(ctx), keys(ctx);
        RTB_CHECK(store.reserve(sizeof(rt_photon) * store_cap));
        RTB_CHECK(keys.reserve(8 * store_cap));
        PhotonBuffers pb;
        for (int b = 0; b < 2; b++) {
            pb.rays[b] = rays[b].as<rt_ray>();
            pb.beta[b] = beta[b].as<float4>();
            pb.carry[b] = carry[b].as<float4>();
            pb.rng[b] = rng[b].as<uint4>();
        }
        pb.hits = hits.as<rt_hit>();
        pb.store = store.as<rt_photon>();
        pb.keys = keys.as<unsigned long long>();
        pb.store_cap = (uint32_t)std::min<uint64_t>(store_cap, 0xFFFFFFFFull);
        pb.cap = cap;
        pb.queued = cnt.as<uint32_t>();
        pb.stored = pb.queued + kStored;
        pb.trace_cnt = s->scratch.counters.as<uint32_t>();
        RTB_CUDA(cudaEventRecord(e0, st));
        RTB_CUDA(cudaMemsetAsync(cnt.ptr, 0, 4 * kCounts, st));
        RTB_CUDA(cudaMemsetAsync(pb.trace_cnt, 0, 16, st));
        RTB_CUDA(cudaMemsetAsync(perl.ptr, 0, 8ull * nl, st));
        const unsigned blocks = (unsigned)((n + kPB - 1) / kPB);
        k_select<<<blocks, kPB, 0, st>>>(rv, n, seed, dpow.as<float>(), total, sel.as<uint32_t>(),
                                         perl.as<unsigned long long>());
        k_emit<<<blocks, kPB, 0, st>>>(rv, n, seed, dpow.as<float>(), total, sel.as<uint32_t>(),
                                       perl.as<unsigned long long>(), pb);
        RTB_CUDA(cudaGetLastError());
        uint32_t n0 = (uint32_t)n;
        RTB_CUDA(cudaMemcpyAsync(cnt.ptr, &n0, 4, cudaMemcpyHostToDevice, st));
        // Two launches a depth: a depth without paths costs less than asking for their number, which
        // the host does every kDepths depths (a copy, a wait and a gap of 20 us).
        constexpr uint32_t kDepths = 16;
        const unsigned shade_blocks = std::min<unsigned>(cap / kPB + 1, 16u * device_sm_count());
        uint32_t hc[kCounts];
        for (uint32_t depth = 0; depth < max_depth; depth++) {
            RTB_CHECK(launch_walk_dev(rv.sv, pb.rays[depth & 1], pb.queued + depth, cap, pb.hits, pb.trace_cnt, st));
            k_photon_shade<<<shade_blocks, kPB, 0, st>>>(rv, pb, depth, max_depth, rr_depth, seed, flags);
            RTB_CUDA(cudaGetLastError());
            if ((depth + 1) % kDepths && depth + 1 < max_depth) continue;
            RTB_CUDA(cudaMemcpyAsync(hc, cnt.ptr, sizeof(hc), cudaMemcpyDeviceToHost, st));
            RTB_CUDA(cudaStreamSynchronize(st));
            if (hc[depth + 1] == 0) break;
        }
        rays_traced = 0;
        for (uint32_t depth = 0; depth < max_depth; depth++) rays_traced += hc[depth];
        stored = hc[kStored];
        if (stored > store_cap) {  // deterministic: retrace with room for every photon
            store_cap = stored;
            continue;
        }
        // order by (path, depth)
        DevBuf keys_out(ctx), idx_in(ctx), idx_out(ctx), tmp(ctx), sorted(ctx);
        RTB_CHECK(keys_out.reserve(8 * std::max<uint64_t>(stored, 1)));
        RTB_CHECK(idx_in.reserve(4 * std::max<uint64_t>(stored, 1)));
        RTB_CHECK(idx_out.reserve(4 * std::max<uint64_t>(stored, 1)));
        RTB_CHECK(sorted.reserve(sizeof(rt_photon) * std::max<uint64_t>(stored, 1)));
        if (stored) {
            k_iota<<<(unsigned)((stored + 255) / 256), 256, 0, st>>>(idx_in.as<uint32_t>(), stored);
            size_t tmp_bytes = 0;
            RTB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, keys.as<unsigned long long>(),
                                                     keys_out.as<unsigned long long>(), idx_in.as<uint32_t>(),
                                                     idx_out.as<uint32_t>(), (int)stored, 0, 64, st));
            RTB_CHECK(tmp.reserve(tmp_bytes));
            RTB_CUDA(cub::DeviceRadixSort::SortPairs(tmp.ptr, tmp_bytes, keys.as<unsigned long long>(),
                                                     keys_out.as<unsigned long long>(), idx_in.as<uint32_t>(),
                                                     idx_out.as<uint32_t>(), (int)stored, 0, 64, st));
            k_gather_photons<<<(unsigned)((stored + 255) / 256), 256, 0, st>>>(store.as<rt_photon>(),
                                                                             idx_out.as<uint32_t>(), stored,
                                                                             sorted.as<rt_photon>());
            RTB_CUDA(cudaGetLastError());
        }
        RTB_CUDA(cudaEventRecord(e1, st));
        RTB_CUDA(cudaEventSynchronize(e1));
        m = new rt_photon_map();
        map_context(m, ctx);
        m->n = stored;
        m->photons = std::move(sorted);
        break;
    }
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (!m) return fail(RT_ERR_CAPACITY, "rt_photons_trace: photon store overflow");
    if (stats) {
        stats->emitted = n;
        stats->stored = stored;
        stats->rays = rays_traced;
        stats->ms = ms;
    }
    *out = m;
    return RT_OK;
}

}  // extern "C"
