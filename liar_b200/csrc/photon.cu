// photon.cu -- photon-map build and k-nearest gather on sm_100a.
//
// Replaces the Lass KdTree<Photon> that PhotonMapper::buildPhotonMap resets
// (src/liar/tracers/photon_mapper.cpp:798-835, photon_mapper.h:153) and its rangeSearch(point,
// maxRadius, maxCount) calls (photon_mapper.cpp:1097, 1257, 1312, 1352): the up to k photons
// nearest to a point, all closer than r_max, the farthest first in the reference's heap.
//
// Build (spatial hashing, Teschner et al. 2003): a bounding-box reduction fixes the grid origin;
// the cell width follows the photons' density (map_build_impl: about 140 photons per cell on
// surfaces, 9 in volumes, between r_max and r_max / 8), cell = floor((p - origin) / cell_size),
// bucket = hash(cell) mod 2^m; a counting sort (histogram, exclusive scan, scatter) orders the photons by
// bucket into float4 (x, y, z, original index) records (their cells follow from the positions).
// Gather: one warp per query visits the cells around the query in rings of growing Chebyshev
// distance R until k candidates are found or R cell widths reach r_max, then the cells left of the
// box around the k-th of them -- the grid form of the kd-tree search that shrinks its radius as it
// finds neighbours. Candidates are filtered by their cell key, so buckets shared by colliding cells
// never yield a photon twice. Candidates are 64-bit keys (d^2 bits << 32 | photon index), appended to
// a list in shared memory while they are below the limit, the list's k-th as of the last cut; the
// list is sorted once, at the end.
// Distances use explicitly rounded IEEE operations in a fixed order, so every (query, photon) key
// and therefore the neighbour set, ties included (equal d^2: lower index first), equals the CPU
// restatement's.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "../../include/liar_gpu.h"
#include "ctx.h"

using namespace liar_gpu;

struct liar_gpu_photon_map {
    int device = -1;
    size_t n = 0;
    float r_max = 0.0f, cell = 0.0f;
    float origin[3] = {0, 0, 0};
    float extent = 0.0f;
    uint32_t bucket_bits = 0;
    float4* sorted = nullptr;          // bucket order: x, y, z, original index bits
    uint32_t* bucket_start = nullptr;  // 2^bits + 1
    void* scratch = nullptr;           // build scratch (ranks, counts, bounds), kept for rebuilds
    size_t scratch_bytes = 0;
    size_t cap_n = 0, cap_buckets = 0; // capacities of sorted and of bucket_start
};

namespace {

constexpr int kGatherK = 64;
constexpr float kRefine = 4.0f;              // cells per r_max
constexpr int kCellLimit = (1 << 21) - 2;     // largest cell index per axis
constexpr uint32_t kStatusBadBucket = 1u << 4;  // device status bit of the photon kernels

__host__ __device__ __forceinline__ uint32_t bucket_of(int ix, int iy, int iz, uint32_t mask) {
    const uint32_t h = ((uint32_t)ix * 73856093u) ^ ((uint32_t)iy * 19349663u) ^ ((uint32_t)iz * 83492791u);
    return h & mask;
}
__device__ __forceinline__ int cell_coord(float p, float o, float inv) { return (int)floorf((p - o) * inv); }

// squared distance with fixed IEEE roundings (the CPU restatement performs the same operations)
__device__ __forceinline__ float dist2_exact(float px, float py, float pz, float qx, float qy, float qz) {
    const float dx = __fsub_rn(px, qx), dy = __fsub_rn(py, qy), dz = __fsub_rn(pz, qz);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

struct BuildParams {
    float ox, oy, oz, inv;
    uint32_t mask;
};

// ---- bounding box (min x, y, z then max x, y, z as order-preserving integer keys)
__device__ __forceinline__ uint32_t fkey(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float fkey_inv(uint32_t k) {
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, 4);
    return f;
#endif
}
// Bound by its loads in flight and, for small maps, by the atomics on six words: blocks reduce first
// and a thread reads four photons a turn (100k photons: 14.5 -> 4 us with an atomic per block instead
// of one per warp).
__global__ void __launch_bounds__(256) k_bounds(const float* __restrict__ pos, uint32_t n, uint32_t* __restrict__ bounds) {
    __shared__ uint32_t s_b[6][8];
    uint32_t lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4u * step) {
        float v[4][3];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const size_t i = min((size_t)i0 + (size_t)u * step, (size_t)n - 1);
#pragma unroll
            for (int a = 0; a < 3; ++a) v[u][a] = __ldg(pos + 3 * i + a);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const uint32_t k = fkey(v[u][a]);
                lo[a] = min(lo[a], k);
                hi[a] = max(hi[a], k);
            }
    }
    const uint32_t warp = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
        hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
        if ((threadIdx.x & 31u) == 0) {
            s_b[a][warp] = lo[a];
            s_b[3 + a][warp] = hi[a];
        }
    }
    __syncthreads();
    if (threadIdx.x < 3u) {
        uint32_t m = 0xffffffffu;
        for (int w = 0; w < 8; ++w) m = min(m, s_b[threadIdx.x][w]);
        atomicMin(bounds + threadIdx.x, m);
    } else if (threadIdx.x < 6u) {
        uint32_t m = 0u;
        for (int w = 0; w < 8; ++w) m = max(m, s_b[threadIdx.x][w]);
        atomicMax(bounds + threadIdx.x, m);
    }
}

// One photon of every `stride` counted into the buckets of two trial grids, cells of widths c0 and c1
// (the density estimate of map_build_impl); the grids' origins follow from the bounds on the device.
__global__ void k_trial_count(const float* __restrict__ pos, uint32_t n, uint32_t stride, const uint32_t* __restrict__ bounds,
                              float c0, float c1, uint32_t mask, uint32_t* __restrict__ counts0, uint32_t* __restrict__ counts1) {
    const uint64_t i = (uint64_t)(blockIdx.x * blockDim.x + threadIdx.x) * stride;
    if (i >= n) return;
    float d[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) d[a] = __ldg(pos + 3 * i + a) - fkey_inv(bounds[a]);
    const float i0 = 1.0f / c0, i1 = 1.0f / c1;
    // (one cell of margin below the lowest photon, as in the map's own grid)
    atomicAdd(counts0 + bucket_of((int)floorf((d[0] + c0) * i0), (int)floorf((d[1] + c0) * i0), (int)floorf((d[2] + c0) * i0), mask), 1u);
    atomicAdd(counts1 + bucket_of((int)floorf((d[0] + c1) * i1), (int)floorf((d[1] + c1) * i1), (int)floorf((d[2] + c1) * i1), mask), 1u);
}

// The photon's place in its bucket, and the buckets' counts.
__global__ void k_bucket_rank(const float* __restrict__ pos, uint32_t n, BuildParams P, uint32_t* __restrict__ ranks,
                              uint32_t* __restrict__ counts) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = pos[3 * (size_t)i], y = pos[3 * (size_t)i + 1], z = pos[3 * (size_t)i + 2];
    const uint32_t b = bucket_of(cell_coord(x, P.ox, P.inv), cell_coord(y, P.oy, P.inv), cell_coord(z, P.oz, P.inv), P.mask);
    ranks[i] = atomicAdd(counts + b, 1u);
}

// sum over buckets of count^2 (the photon-weighted bucket occupancy times n) of two count arrays
// (nb each, a multiple of 4)
__global__ void __launch_bounds__(256) k_sumsq(const uint32_t* __restrict__ counts0, const uint32_t* __restrict__ counts1,
                                               uint32_t nb, unsigned long long* __restrict__ out) {
    const uint4* c = reinterpret_cast<const uint4*>(blockIdx.y ? counts1 : counts0);
    unsigned long long s = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb / 4; i += gridDim.x * blockDim.x) {
        const uint4 v = c[i];
        s += (unsigned long long)v.x * v.x + (unsigned long long)v.y * v.y + (unsigned long long)v.z * v.z +
             (unsigned long long)v.w * v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31u) == 0 && s) atomicAdd(out + blockIdx.y, s);
}

// exclusive scan of `counts` (n_buckets + 1 entries written to `start`), one block per 1024 x 4 entries
constexpr int kScanBlock = 1024;
constexpr int kScanItems = 4;

__global__ void k_scan_local(const uint32_t* __restrict__ in, uint32_t n, uint32_t* __restrict__ out,
                             uint32_t* __restrict__ block_sums) {
    __shared__ uint32_t warp_sums[32];
    const uint32_t base = blockIdx.x * kScanBlock * kScanItems + threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
    if (base + kScanItems <= n) {
        const uint4 q = *reinterpret_cast<const uint4*>(in + base);
        v[0] = q.x;
        v[1] = q.y;
        v[2] = q.z;
        v[3] = q.w;
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) v[k] = base + k < n ? in[base + k] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) s += v[k];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (kScanBlock / 32) ? warp_sums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= (uint32_t)o) w += t;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    uint32_t run = incl - s + (warp > 0 ? warp_sums[warp - 1] : 0u);
    uint32_t e[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        e[k] = run;
        run += v[k];
    }
    if (base + kScanItems <= n) {
        *reinterpret_cast<uint4*>(out + base) = make_uint4(e[0], e[1], e[2], e[3]);
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (base + k < n) out[base + k] = e[k];
    }
    if (threadIdx.x == kScanBlock - 1) block_sums[blockIdx.x] = run;
}

// (in and out of the scan are 16-byte aligned)
__global__ void k_scan_add(uint32_t* __restrict__ out, uint32_t n, const uint32_t* __restrict__ block_offsets) {
    const uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) * kScanItems;
    if (base >= n) return;
    const uint32_t o = block_offsets[base / (kScanBlock * kScanItems)];
    if (base + kScanItems <= n) {
        uint4* p = reinterpret_cast<uint4*>(out + base);
        const uint4 v = *p;
        *p = make_uint4(v.x + o, v.y + o, v.z + o, v.w + o);
    } else {
        for (uint32_t i = base; i < n; ++i) out[i] += o;
    }
}

// ---- spatial order of gather queries: a counting sort by the Morton code of a 64^3 grid over the
// map, so that the warps running at the same time gather from overlapping cells
constexpr int kOrderBits = 6;
constexpr uint32_t kOrderCells = 1u << (3 * kOrderBits);

__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // bit k of v to bit 3k
    uint32_t r = 0;
#pragma unroll
    for (int k = 0; k < kOrderBits; ++k) r |= ((v >> k) & 1u) << (3 * k);
    return r;
}

__device__ __forceinline__ uint32_t order_key(float x, float y, float z, float ox, float oy, float oz, float inv) {
    const float c[3] = {(x - ox) * inv, (y - oy) * inv, (z - oz) * inv};
    uint32_t k = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float f = fminf(fmaxf(c[a], 0.0f), (float)((1 << kOrderBits) - 1));  // NaN -> 0
        k |= spread3((uint32_t)f) << a;
    }
    return k;
}

// the query's place in its cell, and the cells' counts
__global__ void k_order_rank(const float* __restrict__ q, uint32_t n, float ox, float oy, float oz, float inv,
                             uint32_t* __restrict__ ranks, uint32_t* __restrict__ counts) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t j = 3 * (size_t)i;
    ranks[i] = atomicAdd(counts + order_key(q[j], q[j + 1], q[j + 2], ox, oy, oz, inv), 1u);
}

__global__ void k_order_scatter(const float* __restrict__ q, uint32_t n, float ox, float oy, float oz, float inv,
                                const uint32_t* __restrict__ ranks, const uint32_t* __restrict__ start,
                                float4* __restrict__ ordered, uint32_t* __restrict__ status) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t j = 3 * (size_t)i;
    const float x = q[j], y = q[j + 1], z = q[j + 2];
    const uint32_t slot = start[order_key(x, y, z, ox, oy, oz, inv)] + ranks[i];
    if (slot >= n) {  // cannot happen with consistent counts: record, write nothing
        atomicOr(status, kStatusBadBucket);
        return;
    }
    ordered[slot] = make_float4(x, y, z, __uint_as_float(i));
}

// Bound by its random 16-byte writes; the places come from k_bucket_rank, so that no atomic is waited
// for here.
__global__ void k_scatter(const float* __restrict__ pos, uint32_t n, BuildParams P, const uint32_t* __restrict__ ranks,
                          const uint32_t* __restrict__ start, float4* __restrict__ sorted, uint32_t* __restrict__ status) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = pos[3 * (size_t)i], y = pos[3 * (size_t)i + 1], z = pos[3 * (size_t)i + 2];
    const uint32_t b = bucket_of(cell_coord(x, P.ox, P.inv), cell_coord(y, P.oy, P.inv), cell_coord(z, P.oz, P.inv), P.mask);
    const uint32_t slot = start[b] + ranks[i];
    if (slot >= n) {  // a bucket range past the photon array: record it, write nothing
        atomicOr(status, kStatusBadBucket);
        return;
    }
    sorted[slot] = make_float4(x, y, z, __uint_as_float(i));
}

// bit 31 of a bucket's start marks a bucket that holds photons of more than one cell (hash
// collisions): the photons of a bucket are contiguous, so two neighbours in the same bucket with
// different cells mark it; the gather checks the cells of such buckets photon by photon and those of
// the other buckets once
constexpr uint32_t kBucketMixed = 0x80000000u;
__global__ void k_mark_mixed(const float4* __restrict__ sorted, uint32_t n, BuildParams P, uint32_t* __restrict__ start) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0 || i >= n) return;
    const float4 a = sorted[i - 1], b = sorted[i];
    const int ax = cell_coord(a.x, P.ox, P.inv), ay = cell_coord(a.y, P.oy, P.inv), az = cell_coord(a.z, P.oz, P.inv);
    const int bx = cell_coord(b.x, P.ox, P.inv), by = cell_coord(b.y, P.oy, P.inv), bz = cell_coord(b.z, P.oz, P.inv);
    if (ax == bx && ay == by && az == bz) return;
    const uint32_t ba = bucket_of(ax, ay, az, P.mask), bb = bucket_of(bx, by, bz, P.mask);
    if (ba == bb) atomicOr(start + bb, kBucketMixed);
}

// ---- warp sorting helpers on 64-bit keys
__device__ __forceinline__ uint64_t shfl_xor64(uint64_t v, int m) {
    return __shfl_xor_sync(0xffffffffu, (unsigned long long)v, m);
}
// compare-exchange of lanes l and l^j; ascending where `up` holds for the pair's lower lane
__device__ __forceinline__ uint64_t cmpx(uint64_t v, int j, bool up) {
    const uint64_t o = shfl_xor64(v, j);
    const bool lower = ((threadIdx.x & 31u) & (uint32_t)j) == 0u;
    const bool take_min = lower == up;
    return take_min ? (v < o ? v : o) : (v > o ? v : o);
}
// the same on 32-bit keys
__device__ __forceinline__ uint32_t warp_sort32u(uint32_t v) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const uint32_t o = __shfl_xor_sync(0xffffffffu, v, j);
            const bool lower = (lane & (uint32_t)j) == 0u;
            const bool take_min = lower == ((lane & (uint32_t)k) == 0u);
            v = take_min ? min(v, o) : max(v, o);
        }
    }
    return v;
}

// full ascending bitonic sort of one key per lane
__device__ __forceinline__ uint64_t warp_sort32(uint64_t v) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) v = cmpx(v, j, (lane & (uint32_t)k) == 0u);
    }
    return v;
}
// sorts a bitonic sequence of one key per lane ascending
__device__ __forceinline__ uint64_t warp_bitonic_merge32(uint64_t v) {
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) v = cmpx(v, j, true);
    return v;
}
__device__ __forceinline__ uint64_t reverse_lanes(uint64_t v) {
    return __shfl_sync(0xffffffffu, (unsigned long long)v, 31 - (threadIdx.x & 31u));
}

// i / d for 0 <= i < 2^22, 0 < d, through a float reciprocal with one correction step
__device__ __forceinline__ int div_small(int i, int d, float inv_d) {
    int q = (int)(((float)i + 0.5f) * inv_d);
    if (q * d > i) --q;
    else if ((q + 1) * d <= i) ++q;
    return q;
}

// (div_small's correction step and the cell bound's slack cover the last bits of these)
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// cell i of the shell at Chebyshev distance R >= 2 around a cell ((2R+1)^3 - (2R-1)^3 cells): the
// two z faces, then the square rings of the levels between them
__device__ __forceinline__ void shell_cell(int i, int R, int& dx, int& dy, int& dz) {
    const int side = 2 * R + 1, face = side * side;
    if (i < 2 * face) {
        const int j = i < face ? i : i - face;
        dz = i < face ? -R : R;
        const int y = div_small(j, side, rcp_approx((float)side));
        dy = y - R;
        dx = j - y * side - R;
    } else {
        const int per = 8 * R, i2 = i - 2 * face;
        const int level = div_small(i2, per, rcp_approx((float)per));
        dz = level - R + 1;
        const int p = i2 - level * per;
        const int k = div_small(p, 2 * R, rcp_approx((float)(2 * R))), t = p - k * 2 * R;
        dx = k == 0 ? -R + t : k == 1 ? R : k == 2 ? R - t : -R;
        dy = k == 0 ? -R : k == 1 ? -R + t : k == 2 ? R : R - t;
    }
}

struct GatherParams {
    BuildParams B;
    float r2max;
    float cell;
    float slack;      // cell-assignment round-off allowance in the ring stopping rule
    int max_ring;
    uint32_t n_photons;
};

// The nearest candidates of a warp's query, unordered, in shared memory: every candidate whose key is
// below `limit` is appended; once kCandSpare more than k are held, all but the k nearest (and up to
// kCandSlack more) are dropped and the limit falls to the farthest kept.
constexpr int kCandCap = kGatherK + 96, kCandSpare = 64, kCandSlack = 8;
constexpr int kCandRegs = kCandCap / 32;

// Drops all but the k smallest of the n >= k keys at buf, and up to `slack` more; returns the number
// kept and in `limit` a key with exactly those below it. The threshold is searched in the
// distance bits: by interpolation (on surfaces the number of photons grows linearly with d^2), key by
// key once it is a few short, and by bisection if neither ends it; among equal distances at the
// threshold, in the index bits.
__device__ __forceinline__ int keep_nearest(uint64_t* buf, int n, int k, int slack, uint64_t& limit) {
    const uint32_t lane = threadIdx.x & 31u;
    uint64_t key[kCandRegs];
    uint32_t top = 0, bottom = 0xffffffffu;
#pragma unroll
    for (int r = 0; r < kCandRegs; ++r) {
        const int j = 32 * r + (int)lane;
        key[r] = j < n ? buf[j] : ~0ull;
        bottom = min(bottom, (uint32_t)(key[r] >> 32));
        if (j < n) top = max(top, (uint32_t)(key[r] >> 32));
    }
    uint32_t lo = __reduce_min_sync(0xffffffffu, bottom), hi = __reduce_max_sync(0xffffffffu, top);  // count(<= hi) = n
    int c_lo = 0, c_hi = n;
    const auto count = [&](uint32_t d) {
        int c = 0;
#pragma unroll
        for (int r = 0; r < kCandRegs; ++r) c += (uint32_t)(key[r] >> 32) <= d;
        return __reduce_add_sync(0xffffffffu, c);
    };
    // count(lo) = c_lo < k from here on, below the smallest distance or, where that is zero, counted
    if (lo != 0u) {
        --lo;
    } else {
        c_lo = count(0u);
        if (c_lo >= k) hi = 0u, c_hi = c_lo;
    }
    for (int it = 0; c_hi > k + slack && hi - lo > 1u; ++it) {
        uint32_t mid = lo + ((hi - lo) >> 1);
        if (k - c_lo <= 4 && it > 1) {
            // a few keys short: the next distance above (ties make it more than one key); there is one
            // up to hi, so that this ends within k - c_lo steps and one more
            uint32_t next = 0xffffffffu;
#pragma unroll
            for (int r = 0; r < kCandRegs; ++r) {
                const uint32_t d = (uint32_t)(key[r] >> 32);
                if (d > lo) next = min(next, d);
            }
            mid = min(__reduce_min_sync(0xffffffffu, next), hi - 1u);
        } else if (it < 8) {
            const float f = ((float)(k - c_lo) + 0.5f * (float)slack) * rcp_approx((float)(c_hi - c_lo));
            const float a = __uint_as_float(lo), b = __uint_as_float(hi);
            mid = min(max(__float_as_uint(fmaf(b - a, f, a)), lo + 1u), hi - 1u);
        }
        const int c = count(mid);
        if (c >= k) {
            hi = mid;
            c_hi = c;
        } else {
            lo = mid;
            c_lo = c;
        }
    }
    uint32_t low = 0xffffffffu;  // the threshold's index bits
    if (c_hi > k + slack) {
        // more than that at one distance: the lowest indices of them
        uint32_t i_lo = 0, i_hi = 0xffffffffu;  // count(<= (hi, i_hi)) = c_hi
        const auto count_low = [&](uint32_t i) {
            const uint64_t t = ((uint64_t)hi << 32) | i;
            int c = 0;
#pragma unroll
            for (int r = 0; r < kCandRegs; ++r) c += key[r] <= t;
            return __reduce_add_sync(0xffffffffu, c);
        };
        if (count_low(0u) >= k) i_hi = 0u;
        while (i_hi - i_lo > 1u && i_hi != 0u) {
            const uint32_t mid = i_lo + ((i_hi - i_lo) >> 1);
            if (count_low(mid) >= k) i_hi = mid;
            else i_lo = mid;
        }
        low = i_hi;
    }
    const uint64_t last = ((uint64_t)hi << 32) | low;
    limit = last + 1ull;
    int kept = 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kCandRegs; ++r) {
        const bool keep = key[r] <= last && 32 * r + (int)lane < n;
        const uint32_t m = __ballot_sync(0xffffffffu, keep);
        if (keep) buf[kept + __popc(m & ((1u << lane) - 1u))] = key[r];
        kept += __popc(m);
    }
    __syncwarp();
    return kept;
}

// One warp per query. Bound by issue slots (73% of them, with the candidates' distances a small part):
// merging every batch of 32 candidates into a sorted list took 3,900 warp instructions a query on 4M
// photons on surfaces (1M queries, k = 64: 4.96 ms). Here candidates are only filtered by distance and
// appended, the list is cut to the k nearest two or three times, and sorted once, at the end (2.6 ms,
// with about seven batches of 32 candidates a query).
__global__ void __launch_bounds__(256, 4) k_gather(const float4* __restrict__ sorted,
                                                const uint32_t* __restrict__ start, GatherParams G,
                                                const float* __restrict__ queries, uint32_t nq, int k_out,
                                                int32_t* __restrict__ out_idx, float* __restrict__ out_d2,
                                                int32_t* __restrict__ out_count, uint32_t* __restrict__ status,
                                                const float4* __restrict__ ordered) {
    __shared__ uint64_t s_cand[8][kCandCap];
    const uint32_t lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
    const uint32_t warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    uint64_t* cand = s_cand[threadIdx.x >> 5];
    constexpr uint64_t INF = ~0ull;
    const BuildParams& P = G.B;
    for (uint32_t w = warp_global; w < nq; w += n_warps) {
        // ordered: the queries in spatial order, each with its own index in w (results go there)
        uint32_t q = w;
        float qx, qy, qz;
        if (ordered) {
            const float4 o = ordered[w];
            qx = o.x;
            qy = o.y;
            qz = o.z;
            q = __float_as_uint(o.w);
            if (q >= nq) {  // a slot the reorder pass did not fill: record it, write nothing
                if (lane == 0) atomicOr(status, kStatusBadBucket);
                continue;
            }
        } else {
            qx = queries[3 * q];
            qy = queries[3 * q + 1];
            qz = queries[3 * q + 2];
        }
        const int cx = cell_coord(qx, P.ox, P.inv), cy = cell_coord(qy, P.oy, P.inv), cz = cell_coord(qz, P.oz, P.inv);
        int n = 0;            // candidates held
        int at_limit = 0;     // candidates held when the limit was last set, 0 while it is that of r_max
        uint64_t limit = (uint64_t)__float_as_uint(G.r2max) << 32;
        // rings of cells at Chebyshev distance R, the query's own cell with R = 1, until k candidates are
        // found; then the cells of the box around their limit that the rings have not covered
        bool box = false;
        int bx0 = 0, by0 = 0, bz0 = 0, bnx = 0, bny = 0;  // the box's first cell (relative) and sizes
        float bix = 0.0f, biy = 0.0f;                     // 1 / (bnx bny), 1 / bnx
        int R = 1, shell = 27;
        while (true) {
            // 32 cells at a time (lane: one cell)
            for (int c0 = 0; c0 < shell; c0 += 32) {
                const int c = c0 + (int)lane;
                int dx = 0, dy = 0, dz = 0;
                bool mine = c < shell;
                if (box) {
                    dz = div_small(c, bnx * bny, bix);
                    const int l = c - dz * bnx * bny;
                    dy = div_small(l, bnx, biy);
                    dx = l - dy * bnx + bx0;
                    dy += by0;
                    dz += bz0;
                    mine = mine && max(abs(dx), max(abs(dy), abs(dz))) > R;
                } else if (R == 1) {
                    dz = (int)(lane * 57u >> 9) - 1;  // lane / 9
                    const uint32_t l9 = lane - 9u * (uint32_t)(dz + 1);
                    dy = (int)(l9 * 11u >> 5) - 1;  // l9 / 3
                    dx = (int)l9 - 3 * (dy + 1) - 1;
                } else if (mine) {
                    shell_cell(c, R, dx, dy, dz);
                }
                const int ix = cx + dx, iy = cy + dy, iz = cz + dz;
                mine = mine && ix >= 0 && iy >= 0 && iz >= 0 && ix <= kCellLimit && iy <= kCellLimit && iz <= kCellLimit;
                float md2 = 0.0f;
                if (mine) {
                    // the query's distance to the cell's box, less the cell-assignment round-off: a
                    // cell beyond the limit cannot contribute and is skipped; the others are taken
                    // nearest first, so that the limit falls early
                    const float lx = P.ox + (float)ix * G.cell, ly = P.oy + (float)iy * G.cell, lz = P.oz + (float)iz * G.cell;
                    const float ex = fmaxf(fmaxf(lx - qx, qx - (lx + G.cell)), 0.0f);
                    const float ey = fmaxf(fmaxf(ly - qy, qy - (ly + G.cell)), 0.0f);
                    const float ez = fmaxf(fmaxf(lz - qz, qz - (lz + G.cell)), 0.0f);
                    const float md = fmaxf(sqrt_approx(ex * ex + ey * ey + ez * ez) * 0.999999f - G.slack, 0.0f);
                    md2 = md * md;
                    mine = md2 <= __uint_as_float((uint32_t)(limit >> 32));
                }
                uint32_t s0 = 0, cnt = 0;
                bool mixed = false;
                const auto holds = [&](const float4& p, int x, int y, int z) {  // photon p lies in cell (x, y, z)
                    return cell_coord(p.x, P.ox, P.inv) == x && cell_coord(p.y, P.oy, P.inv) == y && cell_coord(p.z, P.oz, P.inv) == z;
                };
                if (mine) {
                    const uint32_t b = bucket_of(ix, iy, iz, P.mask);
                    const uint32_t r0 = __ldg(start + b);
                    s0 = r0 & ~kBucketMixed;
                    const uint32_t s1 = __ldg(start + b + 1) & ~kBucketMixed;
                    if (s0 > s1 || s1 > G.n_photons) {  // corrupt bucket range: record it, skip the cell
                        atomicOr(status, kStatusBadBucket);
                    } else {
                        cnt = s1 - s0;
                        mixed = (r0 & kBucketMixed) != 0u;
                        // a single-cell bucket: its first photon tells whether it is this cell's
                        if (cnt && !mixed && !holds(__ldg(sorted + s0), ix, iy, iz)) cnt = 0;
                    }
                }
                uint32_t live = __ballot_sync(0xffffffffu, cnt > 0u);
                if (live == 0u) continue;
                uint32_t n_live = __popc(live);
                // mixed buckets are taken one by one, with the cell checked photon by photon (and
                // so are, for the 32-bit prefix sums, buckets of 2^27 photons)
                const uint32_t slow = __ballot_sync(0xffffffffu, mixed && cnt > 0u) | __ballot_sync(0xffffffffu, cnt >> 27);
                while (live) {
                    const bool check = (live & ~slow) == 0u;
                    const uint32_t take = check ? live & (0u - live) : live & ~slow;
                    live &= ~take;
                    // the cells taken, nearest first, in lanes 0 .. n_live - 1: sorted by the distance
                    // bound with its 5 low bits cleared (a lower bound still) and the lane in them
                    n_live = __popc(take);
                    const uint32_t ck = n_live == 1u ? (uint32_t)__ffs(take) - 1u
                                                     : warp_sort32u((take >> lane) & 1u ? ((__float_as_uint(md2) & ~31u) | lane) : 0xffffffffu);
                    const int src = (int)(ck & 31u);
                    const float a_d2 = __uint_as_float(ck & ~31u);
                    const uint32_t a_s0 = __shfl_sync(0xffffffffu, s0, src), c_src = __shfl_sync(0xffffffffu, cnt, src);
                    const uint32_t a_cnt = lane < n_live ? c_src : 0u;
                    int tx = 0, ty = 0, tz = 0;
                    if (check) {
                        tx = __shfl_sync(0xffffffffu, ix, src);
                        ty = __shfl_sync(0xffffffffu, iy, src);
                        tz = __shfl_sync(0xffffffffu, iz, src);
                    }
                    // their photons as one list: lane j's cell owns items [excl_j, excl_j + cnt_j), so
                    // that a batch of 32 candidates spans as many cells as it takes
                    uint32_t incl = a_cnt;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                        if ((int)lane >= o) incl += t;
                    }
                    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31), excl = incl - a_cnt, from = a_s0 - excl;
                    for (uint32_t base = 0; base < total; base += 32) {
                        const uint32_t item = base + lane;
                        // the owning cell: the last lane whose list starts at or before the item
                        uint32_t owner = 0;
                        if (n_live > 1u) {
#pragma unroll
                            for (uint32_t step = 16; step > 0; step >>= 1) {
                                const uint32_t e = __shfl_sync(0xffffffffu, excl, (int)(owner + step));
                                if (e <= item && owner + step < n_live) owner += step;
                            }
                            // ascending distances: once the batch's first cell lies beyond the limit,
                            // so do all that follow
                            const float first = __shfl_sync(0xffffffffu, a_d2, (int)__shfl_sync(0xffffffffu, owner, 0));
                            if (first > __uint_as_float((uint32_t)(limit >> 32))) break;
                        }
                        const uint32_t i = __shfl_sync(0xffffffffu, from, (int)owner) + item;
                        uint64_t key = INF;
                        if (item < total) {
                            const float4 p = __ldg(sorted + i);
                            const float d2 = dist2_exact(p.x, p.y, p.z, qx, qy, qz);
                            key = ((uint64_t)__float_as_uint(d2) << 32) | (uint64_t)__float_as_uint(p.w);
                            if (check && !holds(p, tx, ty, tz)) key = INF;
                        }
                        const bool better = key < limit;
                        const uint32_t m = __ballot_sync(0xffffffffu, better);
                        if (m == 0u) continue;
                        if (better) cand[n + __popc(m & lt_mask)] = key;
                        n += __popc(m);
                        if (n >= k_out + kCandSpare) {
                            __syncwarp();
                            at_limit = n = keep_nearest(cand, n, k_out, kCandSlack, limit);
                        }
                    }
                }
            }
            if (box) break;
            // every photon outside rings 0..R is farther than R cells (minus round-off)
            const float reach = fmaxf((float)R * G.cell - G.slack, 0.0f);
            if (reach * reach >= G.r2max) break;
            if (n >= k_out && n != at_limit) {
                __syncwarp();
                at_limit = n = keep_nearest(cand, n, k_out, kCandSlack, limit);
            }
            if (at_limit) {
                // the cells that a photon below the limit can lie in
                const float rho = sqrt_approx(__uint_as_float((uint32_t)(limit >> 32))) * 1.000001f + G.slack;
                bx0 = cell_coord(qx - rho, P.ox, P.inv) - cx;
                by0 = cell_coord(qy - rho, P.oy, P.inv) - cy;
                bz0 = cell_coord(qz - rho, P.oz, P.inv) - cz;
                const int bx1 = cell_coord(qx + rho, P.ox, P.inv) - cx, by1 = cell_coord(qy + rho, P.oy, P.inv) - cy,
                          bz1 = cell_coord(qz + rho, P.oz, P.inv) - cz;
                if (min(bx0, min(by0, bz0)) >= -R && max(bx1, max(by1, bz1)) <= R) break;
                box = true;
                bnx = bx1 - bx0 + 1;
                bny = by1 - by0 + 1;
                shell = bnx * bny * (bz1 - bz0 + 1);
                bix = rcp_approx((float)(bnx * bny));
                biy = rcp_approx((float)bnx);
                continue;
            }
            if (++R > G.max_ring) break;
            shell = (2 * R + 1) * (2 * R + 1) * (2 * R + 1) - (2 * R - 1) * (2 * R - 1) * (2 * R - 1);
        }
        __syncwarp();
        if (n > k_out) n = keep_nearest(cand, n, k_out, 0, limit);
        // the nearest k in ascending order: slot `lane` in lo, slot `32 + lane` in hi. Sorted by 32-bit
        // keys, the distance in 2^26 steps of the limit with the place in cand: exchanges of one
        // shuffle and one minimum; where two distances share a step the order shows it (about one
        // query in 30,000), and the full keys are sorted
        const float step = 67108864.0f / __uint_as_float((uint32_t)(limit >> 32));
        const auto short_key = [&](uint32_t j) {
            if ((int)j >= n) return 0xffffffffu;
            const float d2 = __uint_as_float((uint32_t)(cand[j] >> 32));
            return (min((uint32_t)(d2 * step), 67108862u) << 6) | j;  // below the empty key
        };
        uint32_t s_lo = warp_sort32u(short_key(lane)), s_hi = 0xffffffffu;
        if (n > 32) {
            s_hi = warp_sort32u(short_key(32u + lane));
            const uint32_t r_hi = __shfl_sync(0xffffffffu, s_hi, 31 - (int)lane);
            s_hi = max(s_lo, r_hi);
            s_lo = min(s_lo, r_hi);
#pragma unroll
            for (int j = 16; j > 0; j >>= 1) {
                const uint32_t a = __shfl_xor_sync(0xffffffffu, s_lo, j), b = __shfl_xor_sync(0xffffffffu, s_hi, j);
                const bool lower = (lane & (uint32_t)j) == 0u;
                s_lo = lower ? min(s_lo, a) : max(s_lo, a);
                s_hi = lower ? min(s_hi, b) : max(s_hi, b);
            }
        }
        uint64_t lo = s_lo != 0xffffffffu ? cand[s_lo & 63u] : INF, hi = s_hi != 0xffffffffu ? cand[s_hi & 63u] : INF;
        const uint64_t lo_next = __shfl_down_sync(0xffffffffu, (unsigned long long)lo, 1),
                       hi_next = __shfl_down_sync(0xffffffffu, (unsigned long long)hi, 1),
                       hi_first = __shfl_sync(0xffffffffu, (unsigned long long)hi, 0);
        if (__any_sync(0xffffffffu, lo > (lane == 31u ? hi_first : lo_next) || (lane < 31u && hi > hi_next))) {
            lo = (int)lane < n ? cand[lane] : INF;
            hi = (int)(32 + lane) < n ? cand[32 + lane] : INF;
            lo = warp_sort32(lo);
            hi = reverse_lanes(warp_sort32(hi));
            const uint64_t a = lo < hi ? lo : hi, b = lo < hi ? hi : lo;
            lo = warp_bitonic_merge32(a);
            hi = warp_bitonic_merge32(b);
        }
        __syncwarp();
        int32_t* oi = out_idx + (size_t)q * k_out;
        float* od = out_d2 + (size_t)q * k_out;
        if ((int)lane < k_out) {
            oi[lane] = lo != INF ? (int32_t)(uint32_t)lo : -1;
            od[lane] = lo != INF ? __uint_as_float((uint32_t)(lo >> 32)) : INFINITY;
        }
        if ((int)(32 + lane) < k_out) {
            oi[32 + lane] = hi != INF ? (int32_t)(uint32_t)hi : -1;
            od[32 + lane] = hi != INF ? __uint_as_float((uint32_t)(hi >> 32)) : INFINITY;
        }
        if (lane == 0 && out_count) out_count[q] = min(n, k_out);
    }
}

// PhotonMapper::estimateIrradianceImpl (photon_mapper.cpp:1254-1279): sum of the powers of the
// neighbours arriving from the normal's side, over pi r^2 with r the farthest neighbour's distance
//
// W lanes per query, a neighbour to a lane (two at k > 32). Bound by L1 wavefronts and, with a thread
// per query (303,000 queries in flight, their photons spread over more than the L2), by DRAM: 5.5 GB
// read for 96 MB of photons. Lanes share a query, so that the queries in flight are fewer and their
// neighbours, which overlap, are found in L1 and L2; and a 12-byte record is read as the one or two
// aligned 16-byte words that hold it.
__device__ __forceinline__ float3 load_record(const float* __restrict__ p, uint32_t i, uint32_t n, bool aligned) {
    if (!aligned || i + 2u > n) return make_float3(__ldg(p + 3 * (size_t)i), __ldg(p + 3 * (size_t)i + 1), __ldg(p + 3 * (size_t)i + 2));
    const uint32_t m = i & 3u;  // the record starts m * 12 bytes after a 48-byte boundary
    const float4* v = reinterpret_cast<const float4*>(p + 12 * (size_t)(i >> 2)) + (m == 0u ? 0u : m - 1u);
    const float4 a = __ldg(v);
    float4 b = a;
    if (m == 1u || m == 2u) b = __ldg(v + 1);
    return make_float3(m == 0u ? a.x : m == 1u ? a.w : m == 2u ? a.z : a.y, m == 0u ? a.y : m == 1u ? b.x : m == 2u ? a.w : a.z,
                       m == 0u ? a.z : m == 1u ? b.y : m == 2u ? b.x : a.w);
}

template <int W>
__global__ void __launch_bounds__(256) k_estimate(const float* __restrict__ power, const float* __restrict__ omega_in,
                                                  const float* __restrict__ normals, uint32_t nq, int k,
                                                  const int32_t* __restrict__ idx, const float* __restrict__ d2,
                                                  const int32_t* __restrict__ count, float power_scale, uint32_t n_photons,
                                                  float* __restrict__ out, uint32_t* __restrict__ status) {
    const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) / W, sub = threadIdx.x % W;
    if (q >= nq) return;
    const bool al_p = ((uintptr_t)power & 15u) == 0u, al_o = ((uintptr_t)omega_in & 15u) == 0u;
    const int c = count[q];
    float x = 0.0f, y = 0.0f, z = 0.0f;
    const float nx = normals[3 * (size_t)q], ny = normals[3 * (size_t)q + 1], nz = normals[3 * (size_t)q + 2];
    for (int j = (int)sub; j < c && j < k; j += W) {
        const int32_t i = idx[(size_t)q * k + j];
        if (i < 0 || (uint32_t)i >= n_photons) {
            atomicOr(status, kStatusBadBucket);
            continue;
        }
        const float3 o = load_record(omega_in, (uint32_t)i, n_photons, al_o);
        if (o.x * nx + o.y * ny + o.z * nz > 0.0f) {
            const float3 p = load_record(power, (uint32_t)i, n_photons, al_p);
            x += p.x;
            y += p.y;
            z += p.z;
        }
    }
    const uint32_t group = W == 32 ? 0xffffffffu : ((1u << (W & 31)) - 1u) << ((threadIdx.x & 31u) / W * W);
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) {
        x += __shfl_xor_sync(group, x, o);
        y += __shfl_xor_sync(group, y, o);
        z += __shfl_xor_sync(group, z, o);
    }
    if (sub == 0) {
        float s = 0.0f;
        if (c > 0) {
            const float r2 = d2[(size_t)q * k + (c < k ? c : k) - 1];
            s = r2 > 0.0f ? power_scale / (3.14159265358979323846f * r2) : 0.0f;
        }
        out[3 * (size_t)q] = x * s;
        out[3 * (size_t)q + 1] = y * s;
        out[3 * (size_t)q + 2] = z * s;
    }
}

int map_build_impl(liar_gpu_ctx* ctx, liar_gpu_photon_map* m, const float* d_pos, size_t n, cudaStream_t st) {
    // buckets: the next power of two >= 2n, at most 2^23 (the two-level scan covers 2^24 entries); fewer
    // below, once the photons are known to lie on surfaces
    uint32_t bits = 10;
    while (bits < 23 && (1ull << bits) < 2ull * n) ++bits;
    size_t nb = (size_t)1 << bits;
    size_t scan_blocks = (nb + 1 + kScanBlock * kScanItems - 1) / (kScanBlock * kScanItems);
    // the density estimate counts one photon in `stride` into at most 2^21 buckets
    const size_t nb_trial = std::min<size_t>(nb, (size_t)1 << 21);
    const uint32_t stride = (uint32_t)std::max<size_t>(1, n >> 20);
    const size_t n_trial = (n + stride - 1) / stride;
    const size_t need = n * 4 + nb_trial * 4 + (((nb + 1) * 4 + 255) / 256) * 256 + (scan_blocks + 1) * 8 + 4096;
    if (m->scratch_bytes < need) {
        if (m->scratch) cudaFree(m->scratch);
        m->scratch = nullptr;
        m->scratch_bytes = 0;
        cudaError_t e = cudaMalloc(&m->scratch, need);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return ctx_cuda(ctx, e, "photon map build scratch");
        }
        m->scratch_bytes = need;
    }
    cudaError_t e = cudaSuccess;
    if (m->cap_n < std::max<size_t>(n, 1)) {
        // photons beyond the buffers' capacity (a first build, or a rebuild with more photons)
        if (m->sorted) cudaFree(m->sorted);
        m->sorted = nullptr;
        m->cap_n = 0;
        e = cudaMalloc((void**)&m->sorted, std::max<size_t>(n, 1) * sizeof(float4));
        if (e == cudaSuccess) m->cap_n = std::max<size_t>(n, 1);
    }
    if (e == cudaSuccess && m->cap_buckets < nb + 1) {
        if (m->bucket_start) cudaFree(m->bucket_start);
        m->bucket_start = nullptr;
        m->cap_buckets = 0;
        e = cudaMalloc((void**)&m->bucket_start, (nb + 1) * sizeof(uint32_t));
        if (e == cudaSuccess) m->cap_buckets = nb + 1;
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return ctx_cuda(ctx, e, "photon map");
    }
    char* p = static_cast<char*>(m->scratch);
    uint32_t* ranks = reinterpret_cast<uint32_t*>(p);
    p += ((n * 4 + 255) / 256) * 256;
    uint32_t* counts1 = reinterpret_cast<uint32_t*>(p);  // the second trial grid's, before `counts`
    p += nb_trial * 4;
    uint32_t* counts = reinterpret_cast<uint32_t*>(p);
    p += (((nb + 1) * 4 + 255) / 256) * 256;
    uint32_t* bounds = reinterpret_cast<uint32_t*>(p);
    p += 256;
    uint32_t* block_sums = reinterpret_cast<uint32_t*>(p);
    uint32_t* block_offs = block_sums + ((scan_blocks + 4) & ~(size_t)3);  // 16-byte aligned for the scan
    // grid origin and extent from the photons' bounding box
    m->origin[0] = m->origin[1] = m->origin[2] = 0.0f;
    m->extent = 0.0f;
    m->cell = m->r_max / kRefine;
    float lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    // one cell of margin below the lowest photon keeps every cell index positive
    auto set_grid = [&](float cell) -> bool {
        m->cell = cell;
        m->extent = 0.0f;
        for (int a = 0; a < 3; ++a) {
            m->origin[a] = lo[a] - cell;
            m->extent = std::max(m->extent, hi[a] - m->origin[a]);
        }
        return m->extent / cell <= (float)(kCellLimit - 4);
    };
    if (n) {
        // the bounds and the counts of the density estimate (below) in one go, with one wait for both
        unsigned long long* d_sum = reinterpret_cast<unsigned long long*>(bounds + 8);
        e = cudaMemsetAsync(bounds, 0xff, 12, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(bounds + 3, 0, 36, st);
        if (e == cudaSuccess && n >= 1024) e = cudaMemsetAsync(counts1, 0, nb_trial * 8, st);
        if (e != cudaSuccess) return ctx_cuda(ctx, e, "photon bounds");
        const unsigned blocks = (unsigned)std::min<size_t>((n + 1023) / 1024, (size_t)ctx->num_sms * 4);
        k_bounds<<<blocks, 256, 0, st>>>(d_pos, (uint32_t)n, bounds);
        if (n >= 1024) {
            k_trial_count<<<(unsigned)((n_trial + 255) / 256), 256, 0, st>>>(d_pos, (uint32_t)n, stride, bounds,
                                                                            m->r_max / 2.0f, m->r_max / 4.0f,
                                                                            (uint32_t)(nb_trial - 1), counts, counts1);
            const unsigned sum_blocks = (unsigned)std::min<size_t>((nb_trial / 4 + 255) / 256, (size_t)ctx->num_sms * 4);
            k_sumsq<<<dim3(sum_blocks, 2), 256, 0, st>>>(counts, counts1, (uint32_t)nb_trial, d_sum);
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return ctx_cuda(ctx, e, "photon density");
        uint32_t hb[12];
        e = cudaMemcpyAsync(hb, bounds, sizeof(hb), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return ctx_cuda(ctx, e, "photon bounds");
        unsigned long long hs[2];
        std::memcpy(hs, hb + 8, sizeof(hs));
        for (int a = 0; a < 3; ++a) {
            lo[a] = fkey_inv(hb[a]);
            hi[a] = fkey_inv(hb[3 + a]);
            if (!std::isfinite(lo[a]) || !std::isfinite(hi[a]))
                return ctx_fail(ctx, LIAR_ERR_INVALID, "photon position is not finite");
        }
        // the cell width from the photons' density: the photon-weighted number of other photons
        // sharing a photon's cell, lambda(c) (a bucket's count squared summed over the buckets, over
        // n, less the photon itself and the expected share of colliding cells n / nb), at r_max / 2
        // and r_max / 4 gives the local dimension D = log2(lambda1 / lambda2) (2 for photons on
        // surfaces, 3 in volumes) and the width at which lambda = T(D), 140 on surfaces and 9 in
        // volumes (geometric in between), measured optima of the gather's cost: the bucket lookups of
        // the cells visited against the candidates tested. Rebuild, gather and estimate at (60, 4),
        // (120, 8), (180, 12), (240, 16): 4M photons on surfaces, 1M queries, k = 64: 4.98, 4.12,
        // 4.02, 4.18 ms; 1M photons in a volume, 500k queries, k = 32: 1.93, 1.62, 1.58, 1.61 ms;
        // 50k photons, 3,000 queries, k = 50: 156, 169, 178, 186 us; cells r_max / 1 .. r_max / 8
        if (n >= 1024) {
            double lam[2] = {0.0, 0.0};
            for (int t = 0; t < 2; ++t) {
                if (!set_grid(m->r_max / (t == 0 ? 2.0f : 4.0f))) break;
                lam[t] = ((double)hs[t] / (double)n_trial - 1.0 - (double)n_trial / (double)nb_trial) * (double)stride;
            }
            float refine = kRefine;
            if (lam[0] > 0.0 && lam[1] > 0.0) {
                const double D = std::min(3.0, std::max(1.5, std::log2(lam[0] / lam[1])));
                const double target = 140.0 * std::pow(9.0 / 140.0, D - 2.0);
                refine = (float)std::min(8.0, std::max(1.0, 2.0 * std::pow(lam[0] / target, 1.0 / D)));
                // surfaces: cells of many photons, so that a quarter of the buckets keeps collisions as rare
                if (target >= 60.0)
                    while (bits > 10 && (1ull << bits) >= (unsigned long long)n) --bits;
            }
            while (!set_grid(m->r_max / refine) && refine > 1.0f) refine = std::max(1.0f, refine * 0.5f);
        }
        if (!set_grid(m->cell))
            return ctx_fail(ctx, LIAR_ERR_UNSUPPORTED, "photons span more than %d grid cells per axis; raise r_max",
                            kCellLimit - 4);
    }
    m->bucket_bits = bits;
    nb = (size_t)1 << bits;
    scan_blocks = (nb + 1 + kScanBlock * kScanItems - 1) / (kScanBlock * kScanItems);
    BuildParams P{m->origin[0], m->origin[1], m->origin[2], 1.0f / m->cell, (uint32_t)(nb - 1)};
    e = cudaMemsetAsync(counts, 0, (nb + 1) * 4, st);
    if (e != cudaSuccess) return ctx_cuda(ctx, e, "photon map counts");
    if (n) k_bucket_rank<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d_pos, (uint32_t)n, P, ranks, counts);
    // exclusive scan of counts[0 .. nb] -> bucket_start (start[nb] = n)
    k_scan_local<<<(unsigned)scan_blocks, kScanBlock, 0, st>>>(counts, (uint32_t)(nb + 1), m->bucket_start, block_sums);
    if (scan_blocks > 1) {
        const size_t blocks2 = (scan_blocks + kScanBlock * kScanItems - 1) / (kScanBlock * kScanItems);
        if (blocks2 > 1) return ctx_fail(ctx, LIAR_ERR_UNSUPPORTED, "photon map too large to scan");
        k_scan_local<<<1, kScanBlock, 0, st>>>(block_sums, (uint32_t)scan_blocks, block_offs, block_sums + scan_blocks);
        k_scan_add<<<(unsigned)((nb + 1 + 1023) / 1024), 256, 0, st>>>(m->bucket_start, (uint32_t)(nb + 1), block_offs);
    }
    if (n) {
        k_scatter<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d_pos, (uint32_t)n, P, ranks, m->bucket_start, m->sorted,
                                                              ctx->d_scratch + kStatusWord);
        k_mark_mixed<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(m->sorted, (uint32_t)n, P, m->bucket_start);
    }
    m->n = n;
    return ctx_cuda(ctx, cudaGetLastError(), "photon map build");
}

}  // namespace

extern "C" int liar_gpu_photon_map_build_device(liar_gpu_ctx* ctx, const float* d_positions, size_t n, float r_max,
                                                liar_gpu_photon_map** out, void* stream) {
    if (!ctx || !out) return LIAR_ERR_INVALID;
    *out = nullptr;
    if (n && !d_positions) return ctx_fail(ctx, LIAR_ERR_INVALID, "null photon positions");
    if (!(r_max > 0.0f) || !std::isfinite(r_max)) return ctx_fail(ctx, LIAR_ERR_INVALID, "r_max must be positive");
    if (n >= (1ull << 31)) return ctx_fail(ctx, LIAR_ERR_INVALID, "too many photons (limit 2^31)");
    int rc = ctx_activate(ctx);
    if (rc) return rc;
    liar_gpu_photon_map* m = new (std::nothrow) liar_gpu_photon_map();
    if (!m) return ctx_fail(ctx, LIAR_ERR_OOM, "host allocation");
    m->device = ctx->device;
    m->r_max = r_max;
    m->cell = r_max / kRefine;
    rc = map_build_impl(ctx, m, d_positions, n, stream ? (cudaStream_t)stream : ctx->stream);
    if (rc) {
        liar_gpu_photon_map_destroy(m);
        return rc;
    }
    *out = m;
    return LIAR_OK;
}

extern "C" int liar_gpu_photon_map_rebuild_device(liar_gpu_ctx* ctx, liar_gpu_photon_map* m, const float* d_positions,
                                                  size_t n, float r_max, void* stream) {
    if (!ctx || !m) return LIAR_ERR_INVALID;
    if (n && !d_positions) return ctx_fail(ctx, LIAR_ERR_INVALID, "null photon positions");
    if (!(r_max > 0.0f) || !std::isfinite(r_max)) return ctx_fail(ctx, LIAR_ERR_INVALID, "r_max must be positive");
    if (n >= (1ull << 31)) return ctx_fail(ctx, LIAR_ERR_INVALID, "too many photons (limit 2^31)");
    if (m->device != ctx->device) return ctx_fail(ctx, LIAR_ERR_INVALID, "photon map belongs to another device");
    int rc = ctx_activate(ctx);
    if (rc) return rc;
    m->r_max = r_max;
    m->cell = r_max / kRefine;
    return map_build_impl(ctx, m, d_positions, n, stream ? (cudaStream_t)stream : ctx->stream);
}

extern "C" int liar_gpu_photon_map_build(liar_gpu_ctx* ctx, const float* positions, size_t n, float r_max,
                                         liar_gpu_photon_map** out) {
    if (!ctx || !out) return LIAR_ERR_INVALID;
    *out = nullptr;
    if (n && !positions) return ctx_fail(ctx, LIAR_ERR_INVALID, "null photon positions");
    for (size_t i = 0; i < 3 * n; ++i)
        if (!std::isfinite(positions[i])) return ctx_fail(ctx, LIAR_ERR_INVALID, "photon position is not finite");
    int rc = ctx_activate(ctx);
    if (rc) return rc;
    float* d = nullptr;
    cudaError_t e = cudaMalloc((void**)&d, std::max<size_t>(n, 1) * 12);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return ctx_cuda(ctx, e, "photon upload");
    }
    e = cudaMemcpyAsync(d, positions, n * 12, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) rc = liar_gpu_photon_map_build_device(ctx, d, n, r_max, out, ctx->stream);
    else rc = ctx_cuda(ctx, e, "photon upload");
    if (!rc) rc = ctx_cuda(ctx, cudaStreamSynchronize(ctx->stream), "photon map build");
    cudaFree(d);
    if (rc && *out) {
        liar_gpu_photon_map_destroy(*out);
        *out = nullptr;
    }
    if (!rc) rc = ctx_check_status(ctx);
    return rc;
}

extern "C" void liar_gpu_photon_map_destroy(liar_gpu_photon_map* m) {
    if (!m) return;
    int cur = -1;
    cudaGetDevice(&cur);
    if (m->device >= 0) cudaSetDevice(m->device);
    if (m->sorted) cudaFree(m->sorted);
    if (m->bucket_start) cudaFree(m->bucket_start);
    if (m->scratch) cudaFree(m->scratch);
    if (cur >= 0) cudaSetDevice(cur);
    delete m;
}

namespace {

constexpr size_t kOrderMinQueries = 1u << 15;  // below this the sort costs more than it saves

struct GatherOrder {
    void* mem = nullptr;
    size_t cap = 0;
    // end of the last gather that read the buffer: a gather on another stream waits for it, since
    // the buffer's entries decide where k_gather writes its results
    cudaEvent_t last_use = nullptr;
    bool used = false;
};

// the queries as float4 (x, y, z, own index) in the Morton order of a 64^3 grid over the map
int order_queries(liar_gpu_ctx* ctx, const liar_gpu_photon_map* m, const float* d_q, uint32_t n, cudaStream_t st,
                  const float4** out, GatherOrder** order) {
    GatherOrder* g = nullptr;
    for (auto& ext : ctx->extensions)
        if (ext.first == "gather_order") g = static_cast<GatherOrder*>(ext.second);
    if (!g) {
        g = new GatherOrder();
        ctx->extensions.emplace_back("gather_order", g);
        ctx->on_destroy.push_back([g]() {
            if (g->mem) cudaFree(g->mem);
            if (g->last_use) cudaEventDestroy(g->last_use);
            delete g;
        });
    }
    if (!g->last_use) {
        cudaError_t e = cudaEventCreateWithFlags(&g->last_use, cudaEventDisableTiming);
        if (e != cudaSuccess) return ctx_cuda(ctx, e, "gather order event");
    }
    if (g->used) {
        cudaError_t e = cudaStreamWaitEvent(st, g->last_use, 0);
        if (e != cudaSuccess) return ctx_cuda(ctx, e, "gather order wait");
    }
    const size_t nb = kOrderCells;
    const size_t scan_blocks = (nb + 1 + kScanBlock * kScanItems - 1) / (kScanBlock * kScanItems);
    const size_t a_ord = ((size_t)n * 16 + 255) / 256 * 256, a_keys = ((size_t)n * 4 + 255) / 256 * 256;
    const size_t a_cnt = ((nb + 1) * 4 + 255) / 256 * 256;
    int rc = ctx_grow(ctx, &g->mem, &g->cap, a_ord + a_keys + 2 * a_cnt + (scan_blocks + 1) * 8 + 256, "gather order");
    if (rc) return rc;
    char* p = static_cast<char*>(g->mem);
    float4* ordered = reinterpret_cast<float4*>(p);
    uint32_t* ranks = reinterpret_cast<uint32_t*>(p + a_ord);
    uint32_t* counts = reinterpret_cast<uint32_t*>(p + a_ord + a_keys);
    uint32_t* start = reinterpret_cast<uint32_t*>(p + a_ord + a_keys + a_cnt);
    uint32_t* block_sums = reinterpret_cast<uint32_t*>(p + a_ord + a_keys + 2 * a_cnt);
    uint32_t* block_offs = block_sums + ((scan_blocks + 4) & ~(size_t)3);  // 16-byte aligned for the scan
    cudaError_t e = cudaMemsetAsync(counts, 0, (nb + 1) * 4, st);
    if (e != cudaSuccess) return ctx_cuda(ctx, e, "gather order");
    const float inv = (float)(1 << kOrderBits) / std::max(m->extent, 1e-30f);
    const unsigned blocks = (n + 255) / 256;
    k_order_rank<<<blocks, 256, 0, st>>>(d_q, n, m->origin[0], m->origin[1], m->origin[2], inv, ranks, counts);
    k_scan_local<<<(unsigned)scan_blocks, kScanBlock, 0, st>>>(counts, (uint32_t)(nb + 1), start, block_sums);
    if (scan_blocks > 1) {
        k_scan_local<<<1, kScanBlock, 0, st>>>(block_sums, (uint32_t)scan_blocks, block_offs, block_sums + scan_blocks);
        k_scan_add<<<(unsigned)((nb + 1 + 1023) / 1024), 256, 0, st>>>(start, (uint32_t)(nb + 1), block_offs);
    }
    k_order_scatter<<<blocks, 256, 0, st>>>(d_q, n, m->origin[0], m->origin[1], m->origin[2], inv, ranks, start, ordered,
                                            ctx->d_scratch + kStatusWord);
    e = cudaGetLastError();
    if (e != cudaSuccess) return ctx_cuda(ctx, e, "gather order");
    *out = ordered;
    *order = g;
    return LIAR_OK;
}

}  // namespace

extern "C" int liar_gpu_photon_gather_device(liar_gpu_ctx* ctx, const liar_gpu_photon_map* m, const float* d_queries,
                                             size_t n_queries, int k, int32_t* d_idx, float* d_d2, int32_t* d_count,
                                             void* stream) {
    if (!ctx) return LIAR_ERR_INVALID;
    if (!m || (n_queries && (!d_queries || !d_idx || !d_d2))) return ctx_fail(ctx, LIAR_ERR_INVALID, "null map or buffer");
    if (k < 1 || k > kGatherK) return ctx_fail(ctx, LIAR_ERR_INVALID, "k must be 1..%d", kGatherK);
    if (m->device != ctx->device) return ctx_fail(ctx, LIAR_ERR_INVALID, "photon map lives on another device");
    if (n_queries >= (1ull << 31)) return ctx_fail(ctx, LIAR_ERR_INVALID, "too many queries");
    if (n_queries == 0) return LIAR_OK;
    int rc = ctx_activate(ctx);
    if (rc) return rc;
    cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
    GatherParams G;
    G.B = BuildParams{m->origin[0], m->origin[1], m->origin[2], 1.0f / m->cell,
                      (uint32_t)(((size_t)1 << m->bucket_bits) - 1)};
    G.r2max = m->r_max * m->r_max;
    G.cell = m->cell;
    G.slack = std::max(1e-3f * m->cell, 8.0f * 1.1920929e-07f * std::max(m->extent, 1.0f));
    G.max_ring = (int)std::ceil(m->r_max / m->cell) + 1;
    G.n_photons = (uint32_t)m->n;
    const float4* ordered = nullptr;
    GatherOrder* order = nullptr;
    if (n_queries >= kOrderMinQueries && m->n > 0) {
        rc = order_queries(ctx, m, d_queries, (uint32_t)n_queries, st, &ordered, &order);
        if (rc) return rc;
    }
    const unsigned blocks = (unsigned)std::min<size_t>((n_queries + 7) / 8, (size_t)ctx->num_sms * 8);
    k_gather<<<blocks, 256, 0, st>>>(m->sorted, m->bucket_start, G, d_queries, (uint32_t)n_queries, k, d_idx,
                                     d_d2, d_count, ctx->d_scratch + kStatusWord, ordered);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && order) {
        e = cudaEventRecord(order->last_use, st);
        order->used = e == cudaSuccess;
    }
    return ctx_cuda(ctx, e, "photon gather launch");
}

extern "C" int liar_gpu_photon_gather(liar_gpu_ctx* ctx, const liar_gpu_photon_map* m, const float* queries,
                                      size_t n_queries, int k, int32_t* idx, float* d2, int32_t* count) {
    if (!ctx) return LIAR_ERR_INVALID;
    if (!m || (n_queries && (!queries || !idx || !d2))) return ctx_fail(ctx, LIAR_ERR_INVALID, "null map or buffer");
    if (k < 1 || k > kGatherK) return ctx_fail(ctx, LIAR_ERR_INVALID, "k must be 1..%d", kGatherK);
    if (n_queries == 0) return LIAR_OK;
    for (size_t i = 0; i < 3 * n_queries; ++i)
        if (!std::isfinite(queries[i])) return ctx_fail(ctx, LIAR_ERR_INVALID, "query position is not finite");
    int rc = ctx_activate(ctx);
    if (rc) return rc;
    const size_t qb = n_queries * 12, ob = n_queries * (size_t)k * 4, cb = n_queries * 4;
    char* d = nullptr;
    cudaError_t e = cudaMalloc((void**)&d, qb + 2 * ob + cb + 64);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return ctx_cuda(ctx, e, "gather buffers");
    }
    float* dq = reinterpret_cast<float*>(d);
    int32_t* di = reinterpret_cast<int32_t*>(d + qb);
    float* dd = reinterpret_cast<float*>(d + qb + ob);
    int32_t* dc = reinterpret_cast<int32_t*>(d + qb + 2 * ob);
    e = cudaMemcpyAsync(dq, queries, qb, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) rc = liar_gpu_photon_gather_device(ctx, m, dq, n_queries, k, di, dd, dc, ctx->stream);
    else rc = ctx_cuda(ctx, e, "query upload");
    if (!rc) {
        e = cudaMemcpyAsync(idx, di, ob, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(d2, dd, ob, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess && count) e = cudaMemcpyAsync(count, dc, cb, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) rc = ctx_cuda(ctx, e, "gather results");
    }
    cudaFree(d);
    if (!rc) rc = ctx_check_status(ctx);
    return rc;
}

extern "C" int liar_gpu_photon_estimate_device(liar_gpu_ctx* ctx, const float* d_power, const float* d_omega_in,
                                               size_t n_photons, const float* d_normals, size_t n_queries, int k,
                                               const int32_t* d_idx, const float* d_d2, const int32_t* d_count,
                                               float power_scale, float* d_out, void* stream) {
    if (!ctx) return LIAR_ERR_INVALID;
    if (n_queries && (!d_power || !d_omega_in || !d_normals || !d_idx || !d_d2 || !d_count || !d_out))
        return ctx_fail(ctx, LIAR_ERR_INVALID, "null buffer");
    if (k < 1 || k > kGatherK) return ctx_fail(ctx, LIAR_ERR_INVALID, "k must be 1..%d", kGatherK);
    if (n_queries >= (1ull << 31) || n_photons >= (1ull << 31)) return ctx_fail(ctx, LIAR_ERR_INVALID, "too many items");
    if (n_queries == 0) return LIAR_OK;
    int rc = ctx_activate(ctx);
    if (rc) return rc;
    cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
    // lanes per query: k of them up to a warp (fewer queries in flight at once read photons nearer to
    // one another, see k_estimate)
    const auto launch = [&](auto kern, int w) {
        kern<<<(unsigned)((n_queries * (size_t)w + 255) / 256), 256, 0, st>>>(
            d_power, d_omega_in, d_normals, (uint32_t)n_queries, k, d_idx, d_d2, d_count, power_scale, (uint32_t)n_photons,
            d_out, ctx->d_scratch + kStatusWord);
    };
    if (k <= 8) launch(k_estimate<8>, 8);
    else if (k <= 16) launch(k_estimate<16>, 16);
    else launch(k_estimate<32>, 32);
    return ctx_cuda(ctx, cudaGetLastError(), "photon estimate launch");
}
