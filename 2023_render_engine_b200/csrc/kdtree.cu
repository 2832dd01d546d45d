// The photon map's kd-tree built on the GPU: the same implicit balanced tree as the host build
// (kd_build, photon.cu; kdtree.h:78-108): the middle element of a range, by the axis of largest
// extent, is its node.
//
// The points are sorted once per axis. Every range of the tree is then a range of positions of
// all three orders, so that its extent is the difference of its ends, its node is the middle
// element of the order of its axis, and its halves come from a stable partition of the other two
// orders. Ranges are split a level at a time over the whole arrays (a prefix sum over "goes to the
// left / right half") until they fit a block, which finishes its range in shared memory.
//
// What bounds it: launches and latency; each level moves some 50 bytes per point. The host's
// recursion over std::nth_element took 40 ms for 413,000 photons on one core, with the copies to the
// host and back; this build 0.6 ms.
//
// Equal coordinates: the tree is the host's, bit for bit, unless a node's coordinate also occurs
// next to it in its range. Which of the equal elements becomes the node, and on which side the
// others go, is then a matter of std::nth_element's internals there, and of the elements'
// indices here; the build reports it (kKdTies) and counts such nodes.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>

#include "rt_internal.h"

namespace rtb {
namespace {

constexpr int kT = 256;
// Largest range a block finishes: one position per thread, 24 bytes of shared memory each.
constexpr uint32_t kLocal = 1024;

__host__ __device__ __forceinline__ uint32_t kd_middle(uint32_t l, uint32_t r) { return (uint32_t)(((uint64_t)l + r) >> 1); }

// The range at `level` below [l, r) that holds position p; false: p became a node above.
__device__ __forceinline__ bool kd_range(uint32_t p, uint32_t &l, uint32_t &r, int level)
{
    for (int d = 0; d < level; d++) {
        const uint32_t m = kd_middle(l, r);
        if (p == m) return false;
        if (p < m)
            r = m;
        else
            l = m + 1;
    }
    return true;
}

// Unsigned keys that order like the floats (-0 as +0).
__device__ __forceinline__ uint32_t kd_key(float x)
{
    const uint32_t b = __float_as_uint(x + 0.f);
    return b ^ ((b >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}

__global__ void __launch_bounds__(kT) k_kd_keys(const rt_photon *__restrict__ ph, uint32_t n, float *__restrict__ xyz,
                                                uint32_t *__restrict__ keys, uint32_t *__restrict__ ids,
                                                uint32_t *__restrict__ report)
{
    const uint32_t i = blockIdx.x * kT + threadIdx.x;
    if (i >= n) return;
    const float4 p = *reinterpret_cast<const float4 *>(ph[i].pos);
    const float c[3] = {p.x, p.y, p.z};
    bool finite = true;
    for (int a = 0; a < 3; a++) {
        xyz[(size_t)a * n + i] = c[a];
        keys[(size_t)a * n + i] = kd_key(c[a]);
        finite &= isfinite(c[a]);
    }
    ids[i] = i;
    if (!finite) atomicOr(report, kKdNotFinite);
}

// Axis of largest extent of a range whose ends in the order of axis a are lo[a], hi[a] (the first
// axis on ties).
__device__ __forceinline__ int kd_axis(const float lo[3], const float hi[3])
{
    int ax = 0;
    float mx = __fsub_rn(hi[0], lo[0]);
    for (int a = 1; a < 3; a++) {
        const float e = __fsub_rn(hi[a], lo[a]);
        if (e > mx) {
            ax = a;
            mx = e;
        }
    }
    return ax;
}

// Side of every element of its range: 0 left of the node, 1 the node, 2 right. The nodes get their
// axis. report: kKdNotFinite, number of nodes with an equal coordinate beside them.
__global__ void __launch_bounds__(kT) k_kd_side(const float *__restrict__ xyz, const uint32_t *__restrict__ order, uint32_t n,
                                                int level, uint8_t *__restrict__ side, uint8_t *__restrict__ axis,
                                                uint32_t *__restrict__ report)
{
    const uint32_t p = blockIdx.x * kT + threadIdx.x;
    uint32_t l = 0, r = n;
    if (p >= n || !kd_range(p, l, r, level)) return;
    float lo[3], hi[3];
    for (int a = 0; a < 3; a++) {
        const uint32_t *o = order + (size_t)a * n;
        lo[a] = xyz[(size_t)a * n + o[l]];
        hi[a] = xyz[(size_t)a * n + o[r - 1]];
    }
    const int ax = kd_axis(lo, hi);
    const uint32_t *o = order + (size_t)ax * n;
    const uint32_t m = kd_middle(l, r);
    side[o[p]] = p < m ? 0 : (p == m ? 1 : 2);
    if (p == m) {
        const float *x = xyz + (size_t)ax * n;
        const float c = x[o[m]];
        axis[m] = r - l > 1 ? (uint8_t)ax : 0;
        if ((m > l && x[o[m - 1]] == c) || (m + 1 < r && x[o[m + 1]] == c)) atomicAdd(report + 1, 1u);
    }
}

// Per position of the three orders: goes left (low word), goes right (high word).
__global__ void __launch_bounds__(kT) k_kd_flags(const uint32_t *__restrict__ order, uint64_t n3,
                                                 const uint8_t *__restrict__ side, uint64_t *__restrict__ flags)
{
    const uint64_t j = (uint64_t)blockIdx.x * kT + threadIdx.x;
    if (j >= n3) return;
    const uint32_t s = side[order[j]];
    flags[j] = (uint64_t)(s == 0) | ((uint64_t)(s == 2) << 32);
}

// Stable partition of every range of the three orders (sums: the exclusive sums of the flags).
__global__ void __launch_bounds__(kT) k_kd_split(const uint32_t *__restrict__ order, uint32_t n, int level,
                                                 const uint8_t *__restrict__ side, const uint64_t *__restrict__ sums,
                                                 uint32_t *__restrict__ out)
{
    const uint32_t p = blockIdx.x * kT + threadIdx.x;
    const size_t base = (size_t)blockIdx.y * n;
    if (p >= n) return;
    const uint32_t id = order[base + p];
    uint32_t l = 0, r = n, to = p;
    if (kd_range(p, l, r, level)) {
        const uint32_t m = kd_middle(l, r), s = side[id];
        const uint64_t before = sums[base + p] - sums[base + l];
        to = s == 0 ? l + (uint32_t)before : (s == 1 ? m : m + 1 + (uint32_t)(before >> 32));
    }
    out[base + to] = id;
}

// One block per range at `level` (the b-th from the left; at most kLocal positions): all levels
// below, with the three orders in shared memory as indices into the block's points. local: scratch,
// by element.
__global__ void __launch_bounds__(kLocal) k_kd_local(const float *__restrict__ xyz, const uint32_t *__restrict__ order,
                                                     uint32_t n, int level, uint32_t *__restrict__ local,
                                                     uint32_t *__restrict__ out, uint8_t *__restrict__ axis,
                                                     uint32_t *__restrict__ report)
{
    __shared__ float x[3][kLocal];
    __shared__ uint16_t ord[2][3][kLocal];
    __shared__ uint32_t sums[3][kLocal];  // left (low half) and right elements before a position
    __shared__ uint32_t wsum[3][kLocal / 32];
    __shared__ uint8_t side[kLocal];
    uint32_t l0 = 0, r0 = n;
    for (int d = level - 1; d >= 0; d--) {
        const uint32_t m = kd_middle(l0, r0);
        if ((blockIdx.x >> d) & 1u)
            l0 = m + 1;
        else
            r0 = m;
    }
    const uint32_t len = r0 - l0, t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    if (len == 0) return;  // the whole block
    const bool on = t < len;
    uint32_t id = 0;
    if (on) {
        id = order[l0 + t];
        local[id] = t;
        for (int a = 0; a < 3; a++) x[a][t] = xyz[(size_t)a * n + id];
        ord[0][0][t] = (uint16_t)t;
    }
    __syncthreads();
    if (on)
        for (int a = 1; a < 3; a++) ord[0][a][t] = (uint16_t)local[order[(size_t)a * n + l0 + t]];
    __syncthreads();
    int b = 0;
    bool ties = false;
    // a level halves the ranges: 32 - clz(len) of them leave none
    const int levels = 32 - __clz(len);
    for (int d = 0; d < levels; d++, b ^= 1) {
        uint32_t l = 0, r = len;
        const bool live = on && kd_range(t, l, r, d);
        const uint32_t m = kd_middle(l, r);
        if (live) {
            float lo[3], hi[3];
            for (int a = 0; a < 3; a++) {
                lo[a] = x[a][ord[b][a][l]];
                hi[a] = x[a][ord[b][a][r - 1]];
            }
            const int ax = kd_axis(lo, hi);
            side[ord[b][ax][t]] = t < m ? 0 : (t == m ? 1 : 2);
            if (t == m) {
                const float c = x[ax][ord[b][ax][m]];
                axis[l0 + m] = r - l > 1 ? (uint8_t)ax : 0;
                ties |= (m > l && x[ax][ord[b][ax][m - 1]] == c) || (m + 1 < r && x[ax][ord[b][ax][m + 1]] == c);
            }
        }
        __syncthreads();
        uint32_t mine[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const uint32_t s = on ? side[ord[b][a][t]] : 1u;
            const uint32_t below = (1u << lane) - 1u;
            const unsigned left = __ballot_sync(0xFFFFFFFFu, s == 0), right = __ballot_sync(0xFFFFFFFFu, s == 2);
            mine[a] = (uint32_t)__popc(left & below) | ((uint32_t)__popc(right & below) << 16);
            if (lane == 0) wsum[a][warp] = (uint32_t)__popc(left) | ((uint32_t)__popc(right) << 16);
        }
        __syncthreads();
        if (warp < 3) {
            uint32_t v = wsum[warp][lane], incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            wsum[warp][lane] = incl - v;
        }
        __syncthreads();
        for (int a = 0; a < 3; a++) sums[a][t] = mine[a] + wsum[a][warp];
        __syncthreads();
        if (on)
            for (int a = 0; a < 3; a++) {
                const uint32_t e = ord[b][a][t];
                uint32_t to = t;
                if (live) {
                    const uint32_t s = side[e], before = sums[a][t] - sums[a][l];
                    to = s == 0 ? l + (before & 0xFFFFu) : (s == 1 ? m : m + 1 + (before >> 16));
                }
                ord[b ^ 1][a][to] = (uint16_t)e;
            }
        __syncthreads();
    }
    // every range has been split down to single elements: the orders agree
    sums[0][t] = id;
    __syncthreads();
    if (on) out[l0 + t] = sums[0][ord[b][0][t]];
    const int all = __syncthreads_count(ties);
    if (all && t == 0) atomicAdd(report + 1, (uint32_t)all);
}

// The nodes in tree order: position and axis, shape and photon index.
__global__ void __launch_bounds__(kT) k_kd_nodes(const rt_photon *__restrict__ photons, const uint32_t *__restrict__ order,
                                                 const uint8_t *__restrict__ axis, uint32_t n, float4 *__restrict__ pos,
                                                 int2 *__restrict__ aux)
{
    const uint32_t i = blockIdx.x * kT + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = order[i];
    const float4 p = *reinterpret_cast<const float4 *>(photons[id].pos);  // xyz, shape id
    pos[i] = make_float4(p.x, p.y, p.z, __uint_as_float((uint32_t)axis[i]));
    aux[i] = make_int2(__float_as_int(p.w), (int)id);
}

unsigned blocks_for(uint64_t n) { return (unsigned)((n + kT - 1) / kT); }

}  // namespace

int kd_build_device(rt_context *ctx, const rt_photon *photons, uint64_t n64, float4 *node_pos, int2 *node_aux,
                    uint32_t *report, uint32_t *ties)
{
    cudaStream_t st = ctx->stream;
    *report = *ties = 0;
    if (n64 == 0) return RT_OK;
    if (n64 > kKdDeviceMax) return fail(RT_ERR_CAPACITY, "kd_build_device: too many points");
    const uint32_t n = (uint32_t)n64;
    const uint64_t n3 = 3 * n64;
    int level = 0;  // ranges at this level hold at most kLocal positions (they differ by at most one)
    while ((n >> level) > kLocal) level++;
    size_t sort_bytes = 0, scan_bytes = 0;
    uint32_t *none = nullptr;
    uint64_t *none64 = nullptr;
    RTB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, none, none, none, none, (int)n, 0, 32, st));
    if (level) RTB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, none64, none64, (int64_t)n3, st));
    DevBuf work(ctx);
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) / 256 * 256;
        return o;
    };
    const size_t o_xyz = take(4 * n3), o_keys = take(4 * n3), o_keys2 = take(4 * n64), o_ids = take(4 * n64),
                 o_ord = take(4 * n3), o_ord2 = take(4 * n3), o_side = take(n64), o_axis = take(n64),
                 o_flags = take(level ? 8 * n3 : 0), o_sums = take(level ? 8 * n3 : 0),
                 o_tmp = take(std::max(sort_bytes, scan_bytes)), o_rep = take(8);
    RTB_CHECK(work.reserve(at));
    char *w = work.as<char>();
    float *xyz = reinterpret_cast<float *>(w + o_xyz);
    uint32_t *keys = reinterpret_cast<uint32_t *>(w + o_keys), *keys2 = reinterpret_cast<uint32_t *>(w + o_keys2),
             *ids = reinterpret_cast<uint32_t *>(w + o_ids), *ord = reinterpret_cast<uint32_t *>(w + o_ord),
             *ord2 = reinterpret_cast<uint32_t *>(w + o_ord2), *rep = reinterpret_cast<uint32_t *>(w + o_rep);
    uint8_t *side = reinterpret_cast<uint8_t *>(w + o_side), *axis = reinterpret_cast<uint8_t *>(w + o_axis);
    uint64_t *flags = reinterpret_cast<uint64_t *>(w + o_flags), *sums = reinterpret_cast<uint64_t *>(w + o_sums);
    RTB_CUDA(cudaMemsetAsync(rep, 0, 8, st));
    k_kd_keys<<<blocks_for(n), kT, 0, st>>>(photons, n, xyz, keys, ids, rep);
    RTB_CUDA(cudaGetLastError());
    for (int a = 0; a < 3; a++)  // stable: equal coordinates in index order
        RTB_CUDA(cub::DeviceRadixSort::SortPairs(w + o_tmp, sort_bytes, keys + (size_t)a * n, keys2, ids,
                                                 ord + (size_t)a * n, (int)n, 0, 32, st));
    for (int d = 0; d < level; d++) {
        k_kd_side<<<blocks_for(n), kT, 0, st>>>(xyz, ord, n, d, side, axis, rep);
        k_kd_flags<<<blocks_for(n3), kT, 0, st>>>(ord, n3, side, flags);
        RTB_CUDA(cub::DeviceScan::ExclusiveSum(w + o_tmp, scan_bytes, flags, sums, (int64_t)n3, st));
        k_kd_split<<<dim3(blocks_for(n), 3), kT, 0, st>>>(ord, n, d, side, sums, ord2);
        RTB_CUDA(cudaGetLastError());
        std::swap(ord, ord2);
    }
    // nodes of the levels above keep their positions
    RTB_CUDA(cudaMemcpyAsync(ord2, ord, 4 * n64, cudaMemcpyDeviceToDevice, st));
    k_kd_local<<<1u << level, kLocal, 0, st>>>(xyz, ord, n, level, keys2, ord2, axis, rep);
    k_kd_nodes<<<blocks_for(n), kT, 0, st>>>(photons, ord2, axis, n, node_pos, node_aux);
    RTB_CUDA(cudaGetLastError());
    uint32_t found[2];
    RTB_CUDA(cudaMemcpyAsync(found, rep, 8, cudaMemcpyDeviceToHost, st));
    RTB_CUDA(cudaStreamSynchronize(st));
    *report = found[0] | (found[1] ? kKdTies : 0u);
    *ties = found[1];
    return RT_OK;
}

}  // namespace rtb
