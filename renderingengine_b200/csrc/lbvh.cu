// GPU LBVH build: scene bounds, 30-bit Morton codes, a stable LSD radix sort
// on (code, stable primitive ID), the Karras hierarchy and its boxes, all on
// the device.  Semantics follow the reference's CPU mirror
// (src/rt/software_gpu/SoftwareGpu.cpp):
//   - MortonCode / QuantizeMortonAxis / ExpandMortonBits   :184-207, 814-838
//   - centroid = midpoint of the primitive bounds         :92-98
//   - StableRadixSortMorton: lexicographic (code, ID)      :840-884
//   - FindKarrasSplit on the 64-bit key code << 32 | ID    :540-571
//   - one primitive per leaf; RefitBottomUp                 :1265-1527
// and the GPU passes software_lbvh_{morton,radix,hierarchy,bounds}.hlsl.
// The hierarchy is identical to the reference's (the split of a key range is
// the first differing bit of its end keys, a unique position); the device
// nodes carry Karras numbers, and the reference's pre-order numbering is made
// when the flattened records are exported (host_flat).
//
// How the passes map to the device:
//   - a node's box is the union of a contiguous range of leaf boxes, so the
//     boxes come from a binary reduction tree over the leaves (k_seg_build) and
//     one range query per node inside k_karras: no bottom-up walk, whose
//     arrival counters and fences made it a chain of memory round trips as
//     long as the hierarchy is deep;
//   - up to 65,536 keys are sorted by one cluster of eight CTAs, keys and
//     values in shared memory through every pass (k_cluster_sort); more by
//     8-bit passes over global memory;
//   - IDs that already increase with the record index (the usual case) leave
//     only the four passes over the code, since the sort is stable.
#include <algorithm>
#include <chrono>
#include <cooperative_groups.h>
#include <cstring>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "runtime.h"
#include "traverse.cuh"

namespace re {

re_status upload_scene_nodes(re_scene* sc);

namespace {

namespace cg = cooperative_groups;

// Order-preserving float <-> uint mapping for atomic min / max.
__device__ __forceinline__ uint32_t f2o(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}


// Triangle positions (three float4 per triangle, `stride` float4 apart) and
// stable IDs (`id_stride` words apart): separate arrays, or the fields of
// CanonicalTraversalTriangle records.
struct TriangleView {
    const float4* pos;
    const uint32_t* ids;
    uint32_t stride, id_stride;
    __device__ __forceinline__ const float4* at(uint32_t i) const { return pos + size_t(i) * stride; }
    __device__ __forceinline__ uint32_t id(uint32_t i) const { return ids[size_t(i) * id_stride]; }
};

// Union of the boxes of a 256-thread CTA into out (6 words: minima, maxima):
// one atomic per CTA and bound.
__device__ __forceinline__ void block_bounds(float (&lo)[3], float (&hi)[3], uint32_t* out) {
    __shared__ float part[8][6];
    for (int a = 0; a < 3; ++a) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    }
    if ((threadIdx.x & 31) == 0) {
        for (int a = 0; a < 3; ++a) {
            part[threadIdx.x >> 5][a] = lo[a];
            part[threadIdx.x >> 5][3 + a] = hi[a];
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        float v = part[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) v = fminf(v, part[w][threadIdx.x]);
        atomicMin(out + threadIdx.x, f2o(v));
    } else if (threadIdx.x < 6) {
        float v = part[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) v = fmaxf(v, part[w][threadIdx.x]);
        atomicMax(out + threadIdx.x, f2o(v));
    }
}

__device__ __forceinline__ void grow(float (&lo)[3], float (&hi)[3], float4 p) {
    lo[0] = fminf(lo[0], p.x); lo[1] = fminf(lo[1], p.y); lo[2] = fminf(lo[2], p.z);
    hi[0] = fmaxf(hi[0], p.x); hi[1] = fmaxf(hi[1], p.y); hi[2] = fmaxf(hi[2], p.z);
}

// What the passes before the sort report (a word of flags).
constexpr uint32_t kBadFinite = 1u, kBadDegenerate = 2u, kBadNoId = 4u, kBadIdRange = 8u, kBadIdDup = 16u;
constexpr uint32_t kHasAlphaMask = 32u;  // not an error: some record is alpha-masked
constexpr uint32_t kIdsUnordered = 64u;  // not an error: IDs do not increase with the record index

// Header of a build's scratch: scene bounds and the flags.
struct BuildHeader {
    uint32_t bounds[6];
    uint32_t flags;
    uint32_t pad;
};

__global__ void k_init(BuildHeader* h) {
    if (threadIdx.x < 6) h->bounds[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
    if (threadIdx.x == 6) h->flags = 0u;
}

// Scene bounds and whether the IDs increase with the record index.
__global__ void __launch_bounds__(256) k_bounds(TriangleView v, uint32_t n, BuildHeader* h) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    bool unordered = false;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4* p = v.at(i);
        grow(lo, hi, p[0]);
        grow(lo, hi, p[1]);
        grow(lo, hi, p[2]);
        unordered |= i > 0 && v.id(i) <= v.id(i - 1);
    }
    if (unordered) atomicOr(&h->flags, kIdsUnordered);
    block_bounds(lo, hi, h->bounds);
}

__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
    v &= 0x000003ffu;
    v = (v | (v << 16u)) & 0x030000ffu;
    v = (v | (v << 8u)) & 0x0300f00fu;
    v = (v | (v << 4u)) & 0x030c30c3u;
    v = (v | (v << 2u)) & 0x09249249u;
    return v;
}

// QuantizeMortonAxis in double precision.
__device__ __forceinline__ uint32_t quantize(float v, float lo, float hi) {
    const double extent = double(hi) - double(lo);
    const double nrm = extent > 0.0 ? (double(v) - double(lo)) / extent : 0.5;
    const double c = fmin(fmax(nrm, 0.0), 1.0);
    return min(uint32_t(c * 1024.0), 1023u);
}

__device__ __forceinline__ float midpoint(float a, float b) {
    // std::midpoint for finite floats of normal magnitude: (a + b) / 2.
    return (a + b) / 2.0f;
}

__global__ void k_morton(TriangleView v, uint32_t n, const BuildHeader* h, unsigned long long* keys, uint32_t* vals) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = o2f(h->bounds[a]);
        hi[a] = o2f(h->bounds[3 + a]);
    }
    const float4* p = v.at(i);
    const float4 p0 = p[0], p1 = p[1], p2 = p[2];
    const float c[3] = {midpoint(fminf(p0.x, fminf(p1.x, p2.x)), fmaxf(p0.x, fmaxf(p1.x, p2.x))),
                        midpoint(fminf(p0.y, fminf(p1.y, p2.y)), fmaxf(p0.y, fmaxf(p1.y, p2.y))),
                        midpoint(fminf(p0.z, fminf(p1.z, p2.z)), fmaxf(p0.z, fmaxf(p1.z, p2.z)))};
    const uint32_t code = (expand_bits(quantize(c[0], lo[0], hi[0])) << 2u) |
                          (expand_bits(quantize(c[1], lo[1], hi[1])) << 1u) | expand_bits(quantize(c[2], lo[2], hi[2]));
    keys[i] = (static_cast<unsigned long long>(code) << 32) | v.id(i);
    if (vals != nullptr) vals[i] = i;
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (key, value) by the 62 significant key bits (30-bit
// code above a 32-bit ID), 8 bits a pass.  A pass whose digit is the same in
// every key is left out where that is known: the ID's passes when the IDs
// already increase with the input index (stability keeps their order).
// ---------------------------------------------------------------------------
constexpr uint32_t kBins = 256;

// Lanes of the warp (of those with `in`) whose 8-bit digit equals this lane's:
// one ballot per bit.  (__match_any_sync on 32 distinct digits is served a
// value at a time: with it a cluster pass took 16 us.)
__device__ __forceinline__ uint32_t same_digit(uint32_t digit, bool in) {
    uint32_t mask = __ballot_sync(0xffffffffu, in);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (digit >> b) & 1u;
        const uint32_t with = __ballot_sync(0xffffffffu, bit);
        mask &= bit ? with : ~with;
    }
    return mask;
}

// One cluster of eight CTAs, the keys in their shared memory: CTA r holds
// positions [r * per, (r + 1) * per), per = items * 1024.  A pass ranks each
// warp's keys among equal digits (32 consecutive positions at a time, per-warp
// counts), puts its CTA's keys in digit order in the other
// buffer, exchanges the CTAs' digit counts through the cluster's shared memory,
// and sends each run of a digit to the CTA that owns its target positions, so
// the remote stores of a warp are a few contiguous pieces.  Bound by the latency of a
// pass's barriers, two of the cluster and five of the CTA (the largest stall), and
// its ranking: issue in 32 % of the cycles; 50,003 keys with ordered IDs:
// 61 us in four passes, where 16 four-bit passes of three launches over global
// memory took most of the static build's 628.  The line to the global-memory
// passes is what eight CTAs' shared memory holds.
constexpr uint32_t kClusterCtas = 8, kClusterThreads = 1024, kClusterItems = 8;
constexpr uint32_t kClusterKeys = kClusterCtas * kClusterThreads * kClusterItems;
struct ClusterShared {
    unsigned long long key[2][kClusterThreads * kClusterItems];
    uint32_t val[2][kClusterThreads * kClusterItems];
    uint16_t warp_count[32][kBins];
    uint32_t cta_total[kClusterCtas][kBins];
    unsigned long long cta_varying[kClusterCtas];
    uint32_t base[kBins];
    uint32_t start[kBins];
    uint32_t part[8];
    uint32_t varying[2];
};

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads, 1)
    k_cluster_sort(const unsigned long long* keys_in, uint32_t n, uint32_t items, const BuildHeader* h,
                   unsigned long long* keys_out, uint32_t* vals_out) {
    extern __shared__ __align__(16) unsigned char smem[];
    ClusterShared& S = *reinterpret_cast<ClusterShared*>(smem);
    cg::cluster_group cluster = cg::this_cluster();
    // Another CTA's shared memory may only be accessed once that CTA has
    // started, which a cluster barrier shows; the key loads cover its wait.
    auto started = cluster.barrier_arrive();
    const uint32_t rank = cluster.block_rank(), t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint32_t per = items * kClusterThreads;
    const uint32_t first = warp * 32u * items + lane;  // this lane's slots: first + 32 j
    if (t < 2) S.varying[t] = 0u;
    __syncthreads();
    const unsigned long long ref = keys_in[0];
    unsigned long long vary = 0ull;
    for (uint32_t j = 0; j < items; ++j) {
        const uint32_t slot = first + 32u * j, g = rank * per + slot;
        // Positions past the end sort last: their key is above every code.
        const unsigned long long k = g < n ? keys_in[g] : ~0ull;
        S.key[0][slot] = k;
        S.val[0][slot] = g;
        if (g < n) vary |= k ^ ref;
    }
    atomicOr(&S.varying[0], __reduce_or_sync(0xffffffffu, uint32_t(vary)));
    atomicOr(&S.varying[1], __reduce_or_sync(0xffffffffu, uint32_t(vary >> 32)));
    __syncthreads();
    cluster.barrier_wait(std::move(started));
    if (t < kClusterCtas)
        cluster.map_shared_rank(S.cta_varying, t)[rank] =
            (static_cast<unsigned long long>(S.varying[1]) << 32) | S.varying[0];
    cluster.sync();
    vary = 0ull;
    for (uint32_t r = 0; r < kClusterCtas; ++r) vary |= S.cta_varying[r];
    const bool ordered = (h->flags & kIdsUnordered) == 0u;
    const uint32_t buf = 0;
    for (uint32_t shift = ordered ? 32u : 0u; shift < 64u; shift += 8u) {
        if (((vary >> shift) & 0xffull) == 0ull) continue;  // the same in every CTA
        for (uint32_t b = lane; b < kBins; b += 32u) S.warp_count[warp][b] = 0;
        __syncwarp();
        uint32_t place[kClusterItems];  // digit | rank within the warp << 8
#pragma unroll
        for (uint32_t j = 0; j < kClusterItems; ++j) {
            if (j >= items) break;
            const uint32_t dgt = uint32_t(S.key[buf][first + 32u * j] >> shift) & 0xffu;
            const uint32_t same = same_digit(dgt, true);
            const uint32_t before = S.warp_count[warp][dgt];
            place[j] = dgt | ((before + __popc(same & ((1u << lane) - 1u))) << 8);
            __syncwarp();
            if (int(lane) == __ffs(same) - 1) S.warp_count[warp][dgt] = uint16_t(before + __popc(same));
            __syncwarp();
        }
        __syncthreads();
        // Counts over warps; the digit's first place in this CTA; its total to
        // every CTA.
        uint32_t mine = 0, incl = 0;
        if (t < kBins) {
            for (uint32_t w = 0; w < 32u; ++w) {
                const uint32_t c = S.warp_count[w][t];
                S.warp_count[w][t] = uint16_t(mine);
                mine += c;
            }
            for (uint32_t r = 0; r < kClusterCtas; ++r)
                cluster.map_shared_rank(&S.cta_total[0][0], r)[rank * kBins + t] = mine;
            incl = mine;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= uint32_t(o)) incl += v;
            }
            if (lane == 31u) S.part[warp] = incl;
        }
        __syncthreads();
        if (t < kBins) {
            uint32_t head = incl - mine;
            for (uint32_t w = 0; w < warp; ++w) head += S.part[w];
            S.start[t] = head;
        }
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < kClusterItems; ++j) {
            if (j >= items) break;
            const uint32_t dgt = place[j] & 0xffu;
            const uint32_t at = S.start[dgt] + S.warp_count[warp][dgt] + (place[j] >> 8);
            S.key[buf ^ 1u][at] = S.key[buf][first + 32u * j];
            S.val[buf ^ 1u][at] = S.val[buf][first + 32u * j];
        }
        cluster.sync();  // totals are in, and no CTA reads its old buffer any more
        uint32_t before = 0, all = 0;
        if (t < kBins) {
            for (uint32_t r = 0; r < kClusterCtas; ++r) {
                const uint32_t c = S.cta_total[r][t];
                if (r < rank) before += c;
                all += c;
            }
            incl = all;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= uint32_t(o)) incl += v;
            }
            if (lane == 31u) S.part[warp] = incl;
        }
        __syncthreads();
        if (t < kBins) {
            uint32_t head = incl - all + before - S.start[t];
            for (uint32_t w = 0; w < warp; ++w) head += S.part[w];
            S.base[t] = head;  // target position minus place in this CTA
        }
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < kClusterItems; ++j) {
            if (j >= items) break;
            const uint32_t at = j * kClusterThreads + t;
            const unsigned long long k = S.key[buf ^ 1u][at];
            const uint32_t g = S.base[uint32_t(k >> shift) & 0xffu] + at;
            const uint32_t r = (g >> 10) / items, slot = g - r * per;
            cluster.map_shared_rank(S.key[buf], r)[slot] = k;
            cluster.map_shared_rank(S.val[buf], r)[slot] = S.val[buf ^ 1u][at];
        }
        cluster.sync();
    }
    for (uint32_t slot = t; slot < per; slot += kClusterThreads) {
        const uint32_t g = rank * per + slot;
        if (g < n) {
            keys_out[g] = S.key[buf][slot];
            vals_out[g] = S.val[buf][slot];
        }
    }
}

cudaError_t cluster_sort(const unsigned long long* keys_in, uint32_t n, const BuildHeader* h,
                         unsigned long long* keys_out, uint32_t* vals_out, cudaStream_t s) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_cluster_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(ClusterShared)));
    if (e != cudaSuccess) return e;
    const uint32_t items = (n + kClusterCtas * kClusterThreads - 1u) / (kClusterCtas * kClusterThreads);
    k_cluster_sort<<<kClusterCtas, kClusterThreads, sizeof(ClusterShared), s>>>(keys_in, n, items, h, keys_out,
                                                                                vals_out);
    return cudaGetLastError();
}

// Global-memory pass: per-tile digit counts (digit-major rows of `tiles`), an
// exclusive scan of each digit's row, and the scatter, which sorts its tile in
// shared memory first so that keys of one digit leave as one run.
constexpr uint32_t kTileThreads = 256, kTileItems = 16, kTile = kTileThreads * kTileItems;

__global__ void __launch_bounds__(kTileThreads) k_sort_count(const unsigned long long* keys, uint32_t n, uint32_t shift,
                                                             uint32_t* rows, uint32_t tiles) {
    __shared__ uint32_t count[kBins];
    count[threadIdx.x] = 0u;
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < kTileItems; ++j) {
        const uint32_t i = blockIdx.x * kTile + j * kTileThreads + threadIdx.x;
        if (i < n) atomicAdd(&count[uint32_t(keys[i] >> shift) & 0xffu], 1u);
    }
    __syncthreads();
    rows[size_t(threadIdx.x) * tiles + blockIdx.x] = count[threadIdx.x];
}

// One CTA per digit: its row becomes an exclusive scan over the tiles, its sum
// goes to total[digit].
__global__ void __launch_bounds__(kTileThreads) k_sort_rows(uint32_t* rows, uint32_t tiles, uint32_t* total) {
    __shared__ uint32_t part[8];
    uint32_t* row = rows + size_t(blockIdx.x) * tiles;
    uint32_t carry = 0;
    for (uint32_t b = 0; b < tiles; b += kTileThreads) {
        const uint32_t i = b + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
        const uint32_t v = i < tiles ? row[i] : 0u;
        uint32_t incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= uint32_t(o)) incl += u;
        }
        if (lane == 31u) part[warp] = incl;
        __syncthreads();
        uint32_t head = carry, sum = 0;
        for (uint32_t w = 0; w < 8u; ++w) {
            if (w < warp) head += part[w];
            sum += part[w];
        }
        if (i < tiles) row[i] = head + incl - v;
        carry += sum;
        __syncthreads();
    }
    if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(kTileThreads)
    k_sort_scatter(const unsigned long long* keys_in, const uint32_t* vals_in, unsigned long long* keys_out,
                   uint32_t* vals_out, uint32_t n, uint32_t shift, const uint32_t* rows, const uint32_t* total,
                   uint32_t tiles) {
    __shared__ unsigned long long skey[kTile];
    __shared__ uint32_t sval[kTile / 4];  // values go through in quarters
    __shared__ uint32_t warp_count[8][kBins];
    __shared__ uint32_t start[kBins];   // the digit's first place in the tile
    __shared__ uint32_t target[kBins];  // ... and in the output, minus that
    __shared__ uint32_t part[2][8];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    for (uint32_t b = lane; b < kBins; b += 32u) warp_count[warp][b] = 0u;
    __syncwarp();
    // Warp w owns 512 consecutive keys, 32 at a time, so ranks follow the
    // input order.
    const uint32_t first = blockIdx.x * kTile + warp * 32u * kTileItems + lane;
    unsigned long long key[kTileItems];
    uint32_t place[kTileItems];
#pragma unroll
    for (uint32_t j = 0; j < kTileItems; ++j) {
        const uint32_t i = first + 32u * j;
        key[j] = i < n ? keys_in[i] : ~0ull;
    }
#pragma unroll
    for (uint32_t j = 0; j < kTileItems; ++j) {
        const bool in = first + 32u * j < n;
        const uint32_t dgt = uint32_t(key[j] >> shift) & 0xffu;
        const uint32_t same = same_digit(dgt, in);
        const uint32_t before = in ? warp_count[warp][dgt] : 0u;
        place[j] = before + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (in && int(lane) == __ffs(same) - 1) warp_count[warp][dgt] = before + __popc(same);
        __syncwarp();
    }
    __syncthreads();
    uint32_t mine = 0;
    for (uint32_t w = 0; w < 8u; ++w) {
        const uint32_t c = warp_count[w][t];
        warp_count[w][t] = mine;
        mine += c;
    }
    const uint32_t all = total[t];
    uint32_t incl = mine, gincl = all;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o), v = __shfl_up_sync(0xffffffffu, gincl, o);
        if (lane >= uint32_t(o)) {
            incl += u;
            gincl += v;
        }
    }
    if (lane == 31u) {
        part[0][warp] = incl;
        part[1][warp] = gincl;
    }
    __syncthreads();
    for (uint32_t w = 0; w < warp; ++w) {
        incl += part[0][w];
        gincl += part[1][w];
    }
    start[t] = incl - mine;
    target[t] = (gincl - all) + rows[size_t(t) * tiles + blockIdx.x] - (incl - mine);
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < kTileItems; ++j) {
        if (first + 32u * j >= n) continue;
        const uint32_t dgt = uint32_t(key[j] >> shift) & 0xffu;
        place[j] += start[dgt] + warp_count[warp][dgt];
        skey[place[j]] = key[j];
    }
    __syncthreads();
    const uint32_t count = min(kTile, n - blockIdx.x * kTile);
    for (uint32_t k = t; k < count; k += kTileThreads) {
        const unsigned long long x = skey[k];
        keys_out[target[uint32_t(x >> shift) & 0xffu] + k] = x;
    }
    for (uint32_t q = 0; q < kTile; q += kTile / 4) {
#pragma unroll
        for (uint32_t j = 0; j < kTileItems; ++j) {
            const uint32_t i = first + 32u * j;
            if (i < n && place[j] - q < kTile / 4) sval[place[j] - q] = vals_in[i];
        }
        __syncthreads();
        for (uint32_t k = q + t; k < min(count, q + kTile / 4); k += kTileThreads)
            vals_out[target[uint32_t(skey[k] >> shift) & 0xffu] + k] = sval[k - q];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Boxes of leaf ranges.  Level k holds the union of leaves [j 2^k, (j + 1) 2^k)
// for every j whose leaves all exist; level 0 is the leaf boxes.  A box is two
// float4 (minimum, maximum).  Minima and maxima do not depend on the order
// they are taken in, so a range's box is the one a bottom-up refit gives.
// ---------------------------------------------------------------------------
struct RangeBoxes {
    float4* box;
    uint32_t top;  // twice the smallest power of two >= n
    __host__ __device__ __forceinline__ uint32_t level(uint32_t k) const { return top - (top >> k); }
    static uint32_t span(uint32_t n) {
        uint32_t p = 1u;
        while (p < n) p <<= 1;
        return 2u * p;
    }
};

struct Box {
    float lo[3], hi[3];
};
__device__ __forceinline__ void merge(Box& b, float4 lo, float4 hi) {
    b.lo[0] = fminf(b.lo[0], lo.x); b.lo[1] = fminf(b.lo[1], lo.y); b.lo[2] = fminf(b.lo[2], lo.z);
    b.hi[0] = fmaxf(b.hi[0], hi.x); b.hi[1] = fmaxf(b.hi[1], hi.y); b.hi[2] = fmaxf(b.hi[2], hi.z);
}

// Union of leaves [a, b): at most 2 log2(b - a) aligned blocks, whose loads do
// not depend on each other.
__device__ __forceinline__ Box range_box(const RangeBoxes& r, uint32_t a, uint32_t b) {
    Box out{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
    while (a < b) {
        const uint32_t fit = 31u - uint32_t(__clz(b - a));
        const uint32_t k = a == 0u ? fit : min(uint32_t(__ffs(a)) - 1u, fit);
        const float4* q = r.box + 2 * size_t(r.level(k) + (a >> k));
        merge(out, __ldg(q), __ldg(q + 1));
        a += 1u << k;
    }
    return out;
}

// Levels base + 1 .. base + 8 from level base, 256 of its boxes per CTA.
__global__ void __launch_bounds__(256) k_seg_build(RangeBoxes r, uint32_t n, uint32_t base) {
    __shared__ float4 part[8][2];
    const uint32_t have = n >> base, i = blockIdx.x * 256u + threadIdx.x, lane = threadIdx.x & 31u;
    Box b{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
    if (i < have) {
        const float4* q = r.box + 2 * size_t(r.level(base) + i);
        merge(b, q[0], q[1]);
    }
    auto step = [&](int o) {
        for (int a = 0; a < 3; ++a) {
            b.lo[a] = fminf(b.lo[a], __shfl_xor_sync(0xffffffffu, b.lo[a], o));
            b.hi[a] = fmaxf(b.hi[a], __shfl_xor_sync(0xffffffffu, b.hi[a], o));
        }
    };
    auto put = [&](uint32_t k, uint32_t j) {  // block j of level base + k, when complete
        if (((j + 1u) << k) > have) return;
        float4* q = r.box + 2 * size_t(r.level(base + k) + j);
        q[0] = make_float4(b.lo[0], b.lo[1], b.lo[2], 0.f);
        q[1] = make_float4(b.hi[0], b.hi[1], b.hi[2], 0.f);
    };
    for (uint32_t k = 1; k <= 5u; ++k) {
        step(1 << (k - 1u));
        if ((lane & ((1u << k) - 1u)) == 0u) put(k, i >> k);
    }
    if (lane == 0u) {
        part[threadIdx.x >> 5][0] = make_float4(b.lo[0], b.lo[1], b.lo[2], 0.f);
        part[threadIdx.x >> 5][1] = make_float4(b.hi[0], b.hi[1], b.hi[2], 0.f);
    }
    __syncthreads();
    if (threadIdx.x >= 32u) return;
    b = Box{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
    if (lane < 8u) merge(b, part[lane][0], part[lane][1]);
    for (uint32_t k = 6; k <= 8u; ++k) {
        step(1 << (k - 6u));
        if (lane < 8u && (lane & ((1u << (k - 5u)) - 1u)) == 0u) put(k, (blockIdx.x * 8u + lane) >> (k - 5u));
    }
}

cudaError_t seg_build(const RangeBoxes& r, uint32_t n, cudaStream_t s) {
    for (uint32_t base = 0; (n >> base) > 1u; base += 8u)
        k_seg_build<<<((n >> base) + 255u) / 256u, 256, 0, s>>>(r, n, base);
    return cudaGetLastError();
}

// Leaf boxes (level 0) of separate position arrays in sorted order.
__global__ void k_leaf_boxes(TriangleView v, const uint32_t* order, uint32_t n, RangeBoxes r) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4* p = v.at(order[i]);
    const float4 p0 = p[0], p1 = p[1], p2 = p[2];
    r.box[2 * size_t(i)] = make_float4(fminf(p0.x, fminf(p1.x, p2.x)), fminf(p0.y, fminf(p1.y, p2.y)),
                                       fminf(p0.z, fminf(p1.z, p2.z)), 0.f);
    r.box[2 * size_t(i) + 1] = make_float4(fmaxf(p0.x, fmaxf(p1.x, p2.x)), fmaxf(p0.y, fmaxf(p1.y, p2.y)),
                                           fmaxf(p0.z, fmaxf(p1.z, p2.z)), 0.f);
}

// Common-prefix length of sorted keys i and j (-1 outside the array).  With
// kIndexTieBreak, equal keys compare by their sorted positions instead
// (64 + the common prefix of i and j, Karras 2012 section 4), so duplicate
// keys still give every node exactly one parent; without it the keys must be
// unique, which the scene builds check before they get here.
template <bool kIndexTieBreak>
__device__ __forceinline__ int delta(const unsigned long long* k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const unsigned long long x = k[i] ^ k[j];
    if (kIndexTieBreak && x == 0ull) return 64 + __clz(uint32_t(i) ^ uint32_t(j));
    return __clzll(x);
}

// Karras hierarchy (Karras 2012, "Maximizing parallelism in the construction
// of BVHs, octrees, and k-d trees"): internal node i covers leaves [first,
// last] and splits after gamma.  Child codes: bit 31 set = leaf.
struct KarrasNode {
    uint32_t first, last, gamma, left, right;
};
template <bool kIndexTieBreak>
__device__ __forceinline__ KarrasNode karras_node(const unsigned long long* k, int n, int i) {
    auto dl = [&](int j) { return delta<kIndexTieBreak>(k, n, i, j); };
    const int d = (dl(i + 1) - dl(i - 1)) >= 0 ? 1 : -1;
    const int dmin = dl(i - d);
    int lmax = 2;
    while (dl(i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (dl(i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = dl(j);
    int s = 0;
    int t = l;
    do {
        t = (t + 1) >> 1;
        if (dl(i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int first = min(i, j), last = max(i, j);
    return {uint32_t(first), uint32_t(last), uint32_t(gamma),
            (first == gamma) ? (0x80000000u | uint32_t(gamma)) : uint32_t(gamma),
            (last == gamma + 1) ? (0x80000000u | uint32_t(gamma + 1)) : uint32_t(gamma + 1)};
}

// The caller's 32-byte nodes of the allocation-free build.
__global__ void k_karras_static(const unsigned long long* k, int n, RangeBoxes r, re_lbvh_node* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const KarrasNode kn = karras_node<true>(k, n, i);
    const Box b = range_box(r, kn.first, kn.last + 1u);
    float4* o = reinterpret_cast<float4*>(out + i);
    o[0] = make_float4(b.lo[0], b.lo[1], b.lo[2], __uint_as_float(kn.left));
    o[1] = make_float4(b.hi[0], b.hi[1], b.hi[2], __uint_as_float(kn.right));
}

// A scene's child-pair nodes, by Karras number (root 0, a node's interior
// children next to each other).
__global__ void k_karras_nodes(const unsigned long long* k, int n, RangeBoxes r, DeviceNode* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const KarrasNode kn = karras_node<false>(k, n, i);
    const Box a = range_box(r, kn.first, kn.gamma + 1u), b = range_box(r, kn.gamma + 1u, kn.last + 1u);
    float4* o = reinterpret_cast<float4*>(out + i);
    o[0] = make_float4(a.lo[0], a.hi[0], a.lo[1], a.hi[1]);
    o[1] = make_float4(a.lo[2], a.hi[2], b.lo[0], b.hi[0]);
    o[2] = make_float4(b.lo[1], b.hi[1], b.lo[2], b.hi[2]);
    reinterpret_cast<uint4*>(o)[3] =
        make_uint4(kn.left & 0x7fffffffu, kn.right & 0x7fffffffu, kn.left >> 31, kn.right >> 31);
}

// Scene bounds of CanonicalTraversalTriangle records and, with CHECK, the
// primitive checks of re_scene_create (finite vertices, the degenerate-area
// rule, traversal IDs present and unique -- here they must also be below the
// triangle count, so a bitmap checks uniqueness).
template <bool CHECK>
__global__ void __launch_bounds__(256) k_scan_records(const re_canonical_triangle* t, uint32_t n, uint32_t* seen,
                                                      BuildHeader* h) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    uint32_t bad = 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4* q = reinterpret_cast<const float4*>(t + i);  // 11 float4 a record
        const float4 p0 = __ldg(q), p1 = __ldg(q + 1), p2 = __ldg(q + 2);
        const uint4 meta = __ldg(reinterpret_cast<const uint4*>(q + 10));
        const uint32_t id = meta.z;
        if (i > 0 && id <= __ldg(&t[i - 1].metadata.z)) bad |= kIdsUnordered;
        if ((meta.x & RE_GEOMETRY_FLAG_ALPHA_MASK) != 0u || (meta.y & RE_MATERIAL_FLAG_ALPHA_MASK) != 0u)
            bad |= kHasAlphaMask;
        grow(lo, hi, p0);
        grow(lo, hi, p1);
        grow(lo, hi, p2);
        if (!CHECK) continue;
        if (!(isfinite(p0.x) && isfinite(p0.y) && isfinite(p0.z) && isfinite(p1.x) && isfinite(p1.y) &&
              isfinite(p1.z) && isfinite(p2.x) && isfinite(p2.y) && isfinite(p2.z))) {
            bad |= kBadFinite;
        } else {
            const float e0x = __fsub_rn(p1.x, p0.x), e0y = __fsub_rn(p1.y, p0.y), e0z = __fsub_rn(p1.z, p0.z);
            const float e1x = __fsub_rn(p2.x, p0.x), e1y = __fsub_rn(p2.y, p0.y), e1z = __fsub_rn(p2.z, p0.z);
            const float cx = __fsub_rn(__fmul_rn(e0y, e1z), __fmul_rn(e0z, e1y));
            const float cy = __fsub_rn(__fmul_rn(e0z, e1x), __fmul_rn(e0x, e1z));
            const float cz = __fsub_rn(__fmul_rn(e0x, e1y), __fmul_rn(e0y, e1x));
            const float area2 = __fadd_rn(__fadd_rn(__fmul_rn(cx, cx), __fmul_rn(cy, cy)), __fmul_rn(cz, cz));
            const float l0 = __fadd_rn(__fadd_rn(__fmul_rn(e0x, e0x), __fmul_rn(e0y, e0y)), __fmul_rn(e0z, e0z));
            const float l1 = __fadd_rn(__fadd_rn(__fmul_rn(e1x, e1x), __fmul_rn(e1y, e1y)), __fmul_rn(e1z, e1z));
            const float scale = l0 > l1 ? l0 : l1;
            if (!isfinite(area2) || !(area2 > __fmul_rn(__fmul_rn(scale, scale), 1.0e-14f))) bad |= kBadDegenerate;
        }
        if (id == 0xffffffffu) bad |= kBadNoId;
        else if (id >= n) bad |= kBadIdRange;
        else if (atomicOr(seen + (id >> 5), 1u << (id & 31u)) & (1u << (id & 31u))) bad |= kBadIdDup;
    }
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0 && bad != 0u) atomicOr(&h->flags, bad);
    block_bounds(lo, hi, h->bounds);
}

// Leaf-ordered triangle and attribute records (as upload_scene_triangles packs
// them on the host) and the leaf boxes.
__global__ void k_pack_leaf_order(const re_canonical_triangle* t, const uint32_t* order, uint32_t n,
                                  DeviceTriangle* tris, DeviceAttr* attrs, float4* alpha_tc, RangeBoxes boxes) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t src = order[i];
    const float4* q = reinterpret_cast<const float4*>(t + src);  // 11 float4 a record
    const float4 p0 = __ldg(q), p1 = __ldg(q + 1), p2 = __ldg(q + 2);
    const float4 n0 = __ldg(q + 3), n1 = __ldg(q + 4), n2 = __ldg(q + 5);
    const uint4 id = __ldg(reinterpret_cast<const uint4*>(q + 9)), meta = __ldg(reinterpret_cast<const uint4*>(q + 10));
    const bool double_sided = (meta.x & RE_GEOMETRY_FLAG_DOUBLE_SIDED) != 0u ||
                              (meta.y & RE_MATERIAL_FLAG_DOUBLE_SIDED) != 0u;
    const bool casts = (meta.w & RE_INSTANCE_FLAG_CASTS_SHADOW) != 0u;
    const bool masked = (meta.x & RE_GEOMETRY_FLAG_ALPHA_MASK) != 0u || (meta.y & RE_MATERIAL_FLAG_ALPHA_MASK) != 0u;
    const uint32_t flags = (double_sided ? kTriDoubleSided : 0u) | (casts ? kTriCastsShadow : 0u) |
                           (masked ? kTriAlphaMask : 0u);
    if (alpha_tc != nullptr) {
        const float4 t0 = __ldg(q + 6), t1 = __ldg(q + 7), t2 = __ldg(q + 8);
        alpha_tc[2 * size_t(i)] = make_float4(t0.x, t0.y, t1.x, t1.y);
        alpha_tc[2 * size_t(i) + 1] = make_float4(t2.x, t2.y, __uint_as_float(id.w), 0.f);
    }
    float4* d = reinterpret_cast<float4*>(tris + i);
    d[0] = make_float4(p0.x, p0.y, p0.z, __uint_as_float(flags));
    d[1] = make_float4(__fsub_rn(p1.x, p0.x), __fsub_rn(p1.y, p0.y), __fsub_rn(p1.z, p0.z), __uint_as_float(id.x));
    d[2] = make_float4(__fsub_rn(p2.x, p0.x), __fsub_rn(p2.y, p0.y), __fsub_rn(p2.z, p0.z), __uint_as_float(id.y));
    reinterpret_cast<uint4*>(d)[3] = make_uint4(id.x, id.y, meta.z, src);
    float4* a = reinterpret_cast<float4*>(attrs + i);
    a[0] = make_float4(n0.x, n0.y, n0.z, 0.f);
    a[1] = make_float4(n1.x, n1.y, n1.z, 0.f);
    a[2] = make_float4(n2.x, n2.y, n2.z, 0.f);
    reinterpret_cast<uint4*>(a)[3] = id;
    boxes.box[2 * size_t(i)] = make_float4(fminf(p0.x, fminf(p1.x, p2.x)), fminf(p0.y, fminf(p1.y, p2.y)),
                                           fminf(p0.z, fminf(p1.z, p2.z)), 0.f);
    boxes.box[2 * size_t(i) + 1] = make_float4(fmaxf(p0.x, fmaxf(p1.x, p2.x)), fmaxf(p0.y, fmaxf(p1.y, p2.y)),
                                               fmaxf(p0.z, fmaxf(p1.z, p2.z)), 0.f);
}

// ---------------------------------------------------------------------------
// Four-wide nodes from the child-pair nodes, one level of wide nodes per
// launch.  A wide node takes its binary node's two children and opens the
// interior child of the largest surface area until it has four children or
// only leaves (build_wide_layout's rule and order of children); its interior
// children get consecutive numbers on the next level.  The numbers of a level
// follow the order its threads reach the counter, which no result depends on.
// ---------------------------------------------------------------------------
constexpr uint32_t kMaxWideLevels = 128;
struct WideState {
    uint32_t count[kMaxWideLevels + 1];  // wide nodes per level
    uint32_t stack_bound, max_depth, overflow;
};
struct WideItem {
    uint32_t binary;         // the child-pair node to collapse
    uint32_t stack, depth;   // stack entries held above it; its binary depth (root 1)
};

__global__ void k_wide_init(WideState* st, WideItem* items) {
    for (uint32_t k = threadIdx.x; k <= kMaxWideLevels; k += blockDim.x) st->count[k] = k == 0u ? 1u : 0u;
    if (threadIdx.x == 0) {
        st->stack_bound = 0u;
        st->max_depth = 0u;
        st->overflow = 0u;
        items[0] = {0u, 0u, 1u};
    }
}

__global__ void __launch_bounds__(128) k_wide_level(const DeviceNode* nodes, WideItem* items, WideNode* wide,
                                                    uint32_t capacity, uint32_t level, WideState* st) {
    uint32_t start = 0;
    for (uint32_t k = 0; k < level; ++k) start += st->count[k];
    const uint32_t count = st->count[level];
    for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
        const bool live = base + threadIdx.x < count;
        const uint32_t w = start + base + threadIdx.x;
        float4 ka[4], kb[4];  // (lo.xyz, reference), (hi.xyz, leaf count) per child
        uint32_t kd[4];       // binary depth
        uint32_t kids = 0, inner = 0, stack = 0;
        if (live) {
            const WideItem it = items[w];
            auto load = [&](uint32_t node, float4& a0, float4& b0, float4& a1, float4& b1) {
                const float4* q = reinterpret_cast<const float4*>(nodes + node);
                const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2), d = __ldg(q + 3);
                a0 = make_float4(a.x, a.z, b.x, d.x);
                b0 = make_float4(a.y, a.w, b.y, d.z);
                a1 = make_float4(b.z, c.x, c.z, d.y);
                b1 = make_float4(b.w, c.y, c.w, d.w);
            };
            load(it.binary, ka[0], kb[0], ka[1], kb[1]);
            kd[0] = kd[1] = it.depth + 1u;
            kids = 2;
            while (kids < 4u) {
                int pick = -1;
                float best = -1.0f;
                for (uint32_t k = 0; k < kids; ++k) {
                    if (__float_as_uint(kb[k].w) != 0u) continue;
                    const float dx = kb[k].x - ka[k].x, dy = kb[k].y - ka[k].y, dz = kb[k].z - ka[k].z;
                    const float area = dx * dy + dy * dz + dz * dx;
                    if (area > best) {
                        best = area;
                        pick = int(k);
                    }
                }
                if (pick < 0) break;
                for (uint32_t k = kids; k > uint32_t(pick) + 1u; --k) {
                    ka[k] = ka[k - 1];
                    kb[k] = kb[k - 1];
                    kd[k] = kd[k - 1];
                }
                kd[pick] += 1u;
                kd[pick + 1] = kd[pick];
                load(__float_as_uint(ka[pick].w), ka[pick], kb[pick], ka[pick + 1], kb[pick + 1]);
                ++kids;
            }
            // A traversal at this node pushes all but its nearest child.
            stack = it.stack + kids - 1u;
            for (uint32_t k = 0; k < kids; ++k) inner += __float_as_uint(kb[k].w) == 0u ? 1u : 0u;
        }
        // Numbers of the interior children: one atomic per warp.
        uint32_t incl = inner;
        const uint32_t lane = threadIdx.x & 31u;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= uint32_t(o)) incl += v;
        }
        uint32_t first = 0;
        if (lane == 31u && incl != 0u) first = atomicAdd(&st->count[level + 1u], incl);
        first = start + count + __shfl_sync(0xffffffffu, first, 31) + incl - inner;
        const uint32_t deepest = __reduce_max_sync(0xffffffffu, [&] {
            uint32_t m = 0u;
            for (uint32_t k = 0; k < kids; ++k)
                if (__float_as_uint(kb[k].w) != 0u) m = max(m, kd[k]);
            return m;
        }());
        const uint32_t most = __reduce_max_sync(0xffffffffu, stack);
        if (lane == 0u) {
            atomicMax(&st->max_depth, deepest);
            atomicMax(&st->stack_bound, most);
        }
        if (!live) continue;
        if (w >= capacity || (inner != 0u && first + inner > capacity)) {
            atomicOr(&st->overflow, 1u);
            continue;
        }
        float lo[3][4], hi[3][4];
        uint32_t entry[4], cnt[4];
        uint32_t next = first;
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            const bool has = k < kids;
            lo[0][k] = has ? ka[k].x : INFINITY; hi[0][k] = has ? kb[k].x : INFINITY;
            lo[1][k] = has ? ka[k].y : INFINITY; hi[1][k] = has ? kb[k].y : INFINITY;
            lo[2][k] = has ? ka[k].z : INFINITY; hi[2][k] = has ? kb[k].z : INFINITY;
            cnt[k] = has ? __float_as_uint(kb[k].w) : kWideEmpty;
            entry[k] = kWideEmpty;
            if (!has) continue;
            if (cnt[k] != 0u) {
                entry[k] = __float_as_uint(ka[k].w) | (cnt[k] << kWideLeafShift);
            } else {
                items[next] = {__float_as_uint(ka[k].w), stack, kd[k]};
                entry[k] = next++;
            }
        }
        float4* o = reinterpret_cast<float4*>(wide + w);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            o[2 * a] = make_float4(lo[a][0], lo[a][1], lo[a][2], lo[a][3]);
            o[2 * a + 1] = make_float4(hi[a][0], hi[a][1], hi[a][2], hi[a][3]);
        }
        reinterpret_cast<uint4*>(o)[6] = make_uint4(entry[0], entry[1], entry[2], entry[3]);
        reinterpret_cast<uint4*>(o)[7] = make_uint4(cnt[0], cnt[1], cnt[2], cnt[3]);
    }
}

constexpr size_t align256(size_t v) { return (v + 255) / 256 * 256; }

}  // namespace

// Wide nodes a tree of `interior` child pairs can take.  A wide node has four
// children, or only leaves (two or three): with A of the first kind, B of the
// second and n leaves, 4 A + 2 B <= A + B - 1 + n and B <= 3 A + 1, so
// A + B <= 2 n / 3 + 1.
static uint32_t wide_capacity(uint32_t interior) { return uint32_t((uint64_t(interior) + 1u) * 2u / 3u + 2u); }

size_t wide_scratch_bytes(uint32_t interior) {
    const size_t capacity = wide_capacity(interior);
    return align256(sizeof(WideState)) + align256(capacity * sizeof(WideItem)) +
           align256(capacity * sizeof(WideNode));
}

// Builds sc's four-wide nodes (and reports its binary depth in max_depth) from
// its child-pair nodes on the device.  `scratch` holds wide_scratch_bytes; the
// nodes are made there and copied, as their number is only known then.
re_status build_wide_on_device(re_scene* sc, void* scratch, uint32_t* max_depth) {
    const uint32_t interior = sc->device_node_count, capacity = wide_capacity(interior);
    char* base = static_cast<char*>(scratch);
    auto* st = reinterpret_cast<WideState*>(base);
    auto* items = reinterpret_cast<WideItem*>(base + align256(sizeof(WideState)));
    auto* wide = reinterpret_cast<WideNode*>(base + align256(sizeof(WideState)) +
                                             align256(size_t(capacity) * sizeof(WideItem)));
    k_wide_init<<<1, 128>>>(st, items);
    // Levels in rounds (a balanced tree of 2^28 leaves needs about 15, and a
    // level without nodes costs its launch only), the count read back after each.
    WideState host;
    uint32_t level = 0;
    do {
        for (uint32_t k = 0; k < 20u && level < kMaxWideLevels; ++k, ++level)
            k_wide_level<<<std::min<uint32_t>(148u * 8u, (interior + 127u) / 128u), 128>>>(
                static_cast<const DeviceNode*>(sc->nodes.ptr), items, wide, capacity, level, st);
        RE_CUDA_TRY(cudaGetLastError());
        RE_CUDA_TRY(cudaMemcpy(&host, st, sizeof(host), cudaMemcpyDeviceToHost));
    } while (host.count[level] != 0u && level < kMaxWideLevels);
    if (host.overflow != 0u || host.count[level] != 0u)
        return set_error(RE_RECORDING_FAILED, "four-wide layout exceeds its bound");
    uint32_t total = 0;
    for (uint32_t k = 0; k < level; ++k) total += host.count[k];
    RE_CUDA_TRY(sc->wide_nodes.reserve(size_t(total) * sizeof(WideNode)));
    RE_CUDA_TRY(cudaMemcpyAsync(sc->wide_nodes.ptr, wide, size_t(total) * sizeof(WideNode), cudaMemcpyDeviceToDevice));
    sc->wide_node_count = total;
    sc->wide_stack_bound = host.stack_bound;
    if (max_depth != nullptr) *max_depth = host.max_depth;
    return RE_SUCCESS;
}

namespace {

// Quad node of every child-pair node (trace_quad): its grandchildren, or a
// child itself where that is a leaf.
__global__ void k_quad_nodes(const DeviceNode* nodes, uint32_t count, WideNode* quads) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const DeviceNode nd = nodes[i];
    float lo[3][4], hi[3][4];
    uint32_t entry[4];
    auto put = [&](int slot, const DeviceNode& d, int side) {
        lo[0][slot] = side == 0 ? d.a[0] : d.b[2]; hi[0][slot] = side == 0 ? d.a[1] : d.b[3];
        lo[1][slot] = side == 0 ? d.a[2] : d.c[0]; hi[1][slot] = side == 0 ? d.a[3] : d.c[1];
        lo[2][slot] = side == 0 ? d.b[0] : d.c[2]; hi[2][slot] = side == 0 ? d.b[1] : d.c[3];
        entry[slot] = d.d[side] | (d.d[2 + side] << kWideLeafShift);
    };
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        if (nd.d[2 + side] == 0u) {
            const DeviceNode c = nodes[nd.d[side]];
            put(2 * side, c, 0);
            put(2 * side + 1, c, 1);
        } else {
            put(2 * side, nd, side);
            for (int a = 0; a < 3; ++a) {
                lo[a][2 * side + 1] = INFINITY;
                hi[a][2 * side + 1] = -INFINITY;
            }
            entry[2 * side + 1] = kWideEmpty;
        }
    }
    float4* o = reinterpret_cast<float4*>(quads + i);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        o[2 * a] = make_float4(lo[a][0], lo[a][1], lo[a][2], lo[a][3]);
        o[2 * a + 1] = make_float4(hi[a][0], hi[a][1], hi[a][2], hi[a][3]);
    }
    reinterpret_cast<uint4*>(o)[6] = make_uint4(entry[0], entry[1], entry[2], entry[3]);
    reinterpret_cast<uint4*>(o)[7] = make_uint4(0u, 0u, 0u, 0u);
}

}  // namespace

bool make_quad_nodes(re_scene* sc, cudaStream_t stream) {
    const uint32_t n = sc->device_node_count;
    bool ok = sc->quad_event != nullptr ||
              cudaEventCreateWithFlags(&sc->quad_event, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && sc->quad_nodes.reserve_on(size_t(n) * sizeof(WideNode), stream) == cudaSuccess;
    if (ok) {
        k_quad_nodes<<<(n + 127u) / 128u, 128, 0, stream>>>(static_cast<const DeviceNode*>(sc->nodes.ptr), n,
                                                            static_cast<WideNode*>(sc->quad_nodes.ptr));
        ok = cudaGetLastError() == cudaSuccess && cudaEventRecord(sc->quad_event, stream) == cudaSuccess;
        if (!ok) {
            cudaStreamSynchronize(stream);
            sc->quad_nodes.release();
        }
    }
    if (!ok) cudaGetLastError();
    return ok;
}

// The scene from CanonicalTraversalTriangle records in device memory: the
// checks, the LBVH passes, the leaf-ordered records and the four-wide nodes,
// all on the device; the host reads the flags and bounds once and the wide
// layout's counts once.
re_status build_lbvh_from_device_records(re_scene* sc, const re_canonical_triangle* d_tris, bool check) {
    const uint32_t n = sc->triangle_count;
    const auto t0 = std::chrono::steady_clock::now();
    // The passes read records as 16-byte lanes; records that start elsewhere
    // are moved first.
    BuildBuffer moved;
    if ((reinterpret_cast<uintptr_t>(d_tris) & 15u) != 0u) {
        RE_CUDA_TRY(moved.reserve(size_t(n) * sizeof(re_canonical_triangle)));
        RE_CUDA_TRY(cudaMemcpyAsync(moved.ptr, d_tris, size_t(n) * sizeof(re_canonical_triangle),
                                    cudaMemcpyDeviceToDevice));
        d_tris = static_cast<const re_canonical_triangle*>(moved.ptr);
    }
    const uint32_t tiles = (n + kTile - 1u) / kTile;
    const uint32_t span = RangeBoxes::span(n);
    // One allocation: header | ID bitmap | keys and values twice | digit rows |
    // totals | range boxes; the wide layout's scratch lies over the part that
    // is no longer read by then.
    size_t bytes = 0;
    auto slot = [&](size_t b) {
        const size_t off = bytes;
        bytes += align256(b);
        return off;
    };
    const size_t o_head = slot(sizeof(BuildHeader)), o_seen = slot((size_t(n) + 31) / 32 * 4), o_reuse = bytes;
    const size_t o_keys_a = slot(size_t(n) * 8), o_keys_b = slot(size_t(n) * 8), o_vals_a = slot(size_t(n) * 4),
                 o_vals_b = slot(size_t(n) * 4), o_rows = slot(size_t(tiles) * kBins * 4), o_total = slot(kBins * 4),
                 o_box = slot(size_t(span) * 2 * sizeof(float4));
    BuildBuffer scratch;
    RE_CUDA_TRY(scratch.reserve(std::max(bytes, o_reuse + wide_scratch_bytes(n))));
    char* base = static_cast<char*>(scratch.ptr);
    auto* head = reinterpret_cast<BuildHeader*>(base + o_head);
    auto* seen = reinterpret_cast<uint32_t*>(base + o_seen);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    struct Events {
        cudaEvent_t &a, &b;
        ~Events() {
            if (a) cudaEventDestroy(a);
            if (b) cudaEventDestroy(b);
        }
    } events{e0, e1};
    cudaEventRecord(e0);
    k_init<<<1, 32>>>(head);
    const uint32_t scan_grid = std::min<uint32_t>(148u * 8u, (n + 255u) / 256u);
    if (check) {
        RE_CUDA_TRY(cudaMemsetAsync(seen, 0, (size_t(n) + 31) / 32 * 4));
        k_scan_records<true><<<scan_grid, 256>>>(d_tris, n, seen, head);
    } else {
        k_scan_records<false><<<scan_grid, 256>>>(d_tris, n, nullptr, head);
    }
    RE_CUDA_TRY(cudaGetLastError());
    BuildHeader hh;
    RE_CUDA_TRY(cudaMemcpy(&hh, head, sizeof(hh), cudaMemcpyDeviceToHost));
    if (hh.flags & kBadFinite) return set_error(RE_INVALID_ARGUMENT, "A BVH cannot contain a non-finite triangle");
    if (hh.flags & kBadDegenerate) return set_error(RE_INVALID_ARGUMENT, "scene contains a degenerate triangle");
    if (hh.flags & kBadNoId) return set_error(RE_INVALID_ARGUMENT, "triangle has no traversal ID");
    if (hh.flags & kBadIdRange)
        return set_error(RE_INVALID_ARGUMENT, "traversal IDs of device records must be below the triangle count");
    if (hh.flags & kBadIdDup) return set_error(RE_INVALID_ARGUMENT, "traversal IDs must be unique");

    TriangleView view;
    view.pos = reinterpret_cast<const float4*>(d_tris);
    view.stride = uint32_t(sizeof(re_canonical_triangle) / sizeof(float4));
    view.ids = &d_tris->metadata.z;  // an address only
    view.id_stride = uint32_t(sizeof(re_canonical_triangle) / 4);
    auto* keys_a = reinterpret_cast<unsigned long long*>(base + o_keys_a);
    auto* keys_b = reinterpret_cast<unsigned long long*>(base + o_keys_b);
    auto* vals_a = reinterpret_cast<uint32_t*>(base + o_vals_a);
    auto* vals_b = reinterpret_cast<uint32_t*>(base + o_vals_b);
    auto* rows = reinterpret_cast<uint32_t*>(base + o_rows);
    auto* total = reinterpret_cast<uint32_t*>(base + o_total);
    k_morton<<<(n + 255) / 256, 256>>>(view, n, head, keys_a, n <= kClusterKeys ? nullptr : vals_a);
    if (n <= kClusterKeys) {
        RE_CUDA_TRY(cluster_sort(keys_a, n, head, keys_b, vals_b, nullptr));
        std::swap(keys_a, keys_b);
        std::swap(vals_a, vals_b);
    } else {
        // Device records' IDs are below n; a host scene's may be any.
        uint32_t id_bits = 32;
        if (check) {
            id_bits = 0;
            while ((uint64_t(1) << id_bits) < n) ++id_bits;
        }
        for (uint32_t shift = 0; shift < 64u; shift += 8u) {
            if (shift < 32u && ((hh.flags & kIdsUnordered) == 0u || shift >= id_bits)) continue;
            k_sort_count<<<tiles, kTileThreads>>>(keys_a, n, shift, rows, tiles);
            k_sort_rows<<<kBins, kTileThreads>>>(rows, tiles, total);
            k_sort_scatter<<<tiles, kTileThreads>>>(keys_a, vals_a, keys_b, vals_b, n, shift, rows, total, tiles);
            std::swap(keys_a, keys_b);
            std::swap(vals_a, vals_b);
        }
    }
    RE_CUDA_TRY(cudaGetLastError());
    RE_CUDA_TRY(sc->tris.reserve(size_t(n) * sizeof(DeviceTriangle)));
    RE_CUDA_TRY(sc->attrs.reserve(size_t(n) * sizeof(DeviceAttr)));
    RE_CUDA_TRY(sc->leaf_order.reserve(size_t(n) * 4));
    sc->alpha_masked = (hh.flags & kHasAlphaMask) != 0u;
    if (sc->alpha_masked) RE_CUDA_TRY(sc->alpha_tc.reserve(size_t(n) * 2 * sizeof(float4)));
    const RangeBoxes boxes{reinterpret_cast<float4*>(base + o_box), span};
    k_pack_leaf_order<<<(n + 255) / 256, 256>>>(d_tris, vals_a, n, static_cast<DeviceTriangle*>(sc->tris.ptr),
                                                static_cast<DeviceAttr*>(sc->attrs.ptr),
                                                sc->alpha_masked ? static_cast<float4*>(sc->alpha_tc.ptr) : nullptr,
                                                boxes);
    RE_CUDA_TRY(cudaMemcpyAsync(sc->leaf_order.ptr, vals_a, size_t(n) * 4, cudaMemcpyDeviceToDevice));
    auto bound = [](uint32_t u) {
        const uint32_t v = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
        float f;
        std::memcpy(&f, &v, 4);
        return f;
    };
    for (int a = 0; a < 3; ++a) {
        sc->root_lo[a] = bound(hh.bounds[a]);
        sc->root_hi[a] = bound(hh.bounds[3 + a]);
    }
    sc->flat = FlatBvh{};
    sc->flat.leaf_count = n;
    sc->flat_node_count = 2u * n - 1u;
    if (n > 1u) {
        RE_CUDA_TRY(sc->nodes.reserve(size_t(n - 1u) * sizeof(DeviceNode)));
        RE_CUDA_TRY(seg_build(boxes, n, nullptr));
        k_karras_nodes<<<(n - 1 + 255) / 256, 256>>>(keys_a, int(n), boxes, static_cast<DeviceNode*>(sc->nodes.ptr));
        RE_CUDA_TRY(cudaGetLastError());
        sc->device_node_count = n - 1u;
        sc->layout_meta.root_is_leaf = 0;
        sc->layout_meta.node_original.clear();
        cudaEventRecord(e1);
        // Keys are unique, so a level consumes at least one of their 62 bits
        // and the depth stays below 64.
        const re_status st = build_wide_on_device(sc, base + o_reuse, &sc->flat.max_depth);
        if (st != RE_SUCCESS) return st;
    } else {
        cudaEventRecord(e1);
        sc->flat.max_depth = 1u;
        re_software_node leaf{};
        leaf.bounds_min = re_float4{sc->root_lo[0], sc->root_lo[1], sc->root_lo[2], 0.f};
        leaf.bounds_max = re_float4{sc->root_hi[0], sc->root_hi[1], sc->root_hi[2], 0.f};
        leaf.links = re_uint4{0u, 1u, 0xffffffffu, 0xffffffffu};
        sc->flat.nodes.push_back(leaf);
        sc->flat.leaf_order.push_back(0u);
        const re_status st = upload_scene_nodes(sc);
        if (st != RE_SUCCESS) return st;
    }
    RE_CUDA_TRY(cudaDeviceSynchronize());
    float gpu_ms = 0.f;
    cudaEventElapsedTime(&gpu_ms, e0, e1);
    sc->lbvh_gpu_ms = gpu_ms;
    sc->lbvh_total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return RE_SUCCESS;
}

// The same build from host records (validated by the caller).
re_status build_lbvh_on_device(re_scene* sc, const re_canonical_triangle* tris) {
    const size_t bytes = size_t(sc->triangle_count) * sizeof(re_canonical_triangle);
    BuildBuffer records;
    RE_CUDA_TRY(records.reserve(bytes));
    RE_CUDA_TRY(cudaMemcpy(records.ptr, tris, bytes, cudaMemcpyHostToDevice));
    return build_lbvh_from_device_records(sc, static_cast<const re_canonical_triangle*>(records.ptr), false);
}

// The flattened records (the reference's pre-order, BuildKarrasLbvh's
// buildRange order) and leaf order of a scene whose tree was built on the
// device, from its child-pair nodes; made once, on the first request.
re_status host_flat(const re_scene* csc) {
    re_scene* sc = const_cast<re_scene*>(csc);
    std::lock_guard<std::mutex> lock(sc->flat_mutex);
    if (!sc->flat.nodes.empty()) return RE_SUCCESS;
    const uint32_t n = sc->triangle_count;
    std::vector<DeviceNode> dev(n - 1u);
    std::vector<uint32_t> order(n);
    // The caller may be capturing, and its current device stays.
    {
        DeviceScope on(sc->device);
        RelaxedCaptureScope relaxed;
        cudaStream_t stream = nullptr;
        RE_CUDA_TRY(scene_pool_stream(sc->device, &stream));
        RE_CUDA_TRY(cudaMemcpyAsync(dev.data(), sc->nodes.ptr, dev.size() * sizeof(DeviceNode),
                                    cudaMemcpyDeviceToHost, stream));
        RE_CUDA_TRY(cudaMemcpyAsync(order.data(), sc->leaf_order.ptr, size_t(n) * 4, cudaMemcpyDeviceToHost, stream));
        RE_CUDA_TRY(cudaStreamSynchronize(stream));
    }
    std::vector<re_software_node> nodes;
    nodes.reserve(2u * size_t(n) - 1u);
    struct Item {
        uint32_t ref, leaf, parent, is_right;
        float lo[3], hi[3];
    };
    std::vector<Item> todo;
    Item root{0u, 0u, 0xffffffffu, 0u, {}, {}};
    for (int a = 0; a < 3; ++a) {
        root.lo[a] = sc->root_lo[a];
        root.hi[a] = sc->root_hi[a];
    }
    todo.push_back(root);
    while (!todo.empty()) {
        const Item it = todo.back();
        todo.pop_back();
        const uint32_t pre = uint32_t(nodes.size());
        if (it.is_right) nodes[it.parent].links.z = pre;
        re_software_node rec;
        rec.bounds_min = re_float4{it.lo[0], it.lo[1], it.lo[2], 0.f};
        rec.bounds_max = re_float4{it.hi[0], it.hi[1], it.hi[2], 0.f};
        if (it.leaf) rec.links = re_uint4{it.ref, 1u, 0xffffffffu, it.parent};
        else rec.links = re_uint4{pre + 1u, 0u, 0u, it.parent};
        nodes.push_back(rec);
        if (it.leaf) continue;
        const DeviceNode& d = dev[it.ref];
        const Item left{d.d[0], d.d[2], pre, 0u, {d.a[0], d.a[2], d.b[0]}, {d.a[1], d.a[3], d.b[1]}};
        const Item right{d.d[1], d.d[3], pre, 1u, {d.b[2], d.c[0], d.c[2]}, {d.b[3], d.c[1], d.c[3]}};
        todo.push_back(right);
        todo.push_back(left);
    }
    sc->flat.leaf_order = std::move(order);
    sc->flat.nodes = std::move(nodes);
    return RE_SUCCESS;
}

// ---------------------------------------------------------------------------
// Allocation-free LBVH build (re_lbvh_build_static).  The same passes with
// every intermediate array carved out of one file-scope device array instead
// of a cudaMalloc'd one, launched on the caller's stream, with the Karras
// hierarchy written to caller buffers.  50,003 triangles:
// 628 us with 52 launches, 98 us now, bound by the serial chain of its passes
// (61 us of it the sort).
// ---------------------------------------------------------------------------
namespace {

constexpr uint32_t kStaticMaxTris = RE_LBVH_STATIC_MAX_TRIANGLES;
static_assert(kStaticMaxTris <= kClusterKeys, "the allocation-free build sorts in one cluster");
constexpr size_t kStaticScratchBytes =
    align256(sizeof(BuildHeader)) +
    2 * align256(size_t(kStaticMaxTris) * 8) +                  // keys before and after the sort
    align256(2 * size_t(kStaticMaxTris) * 2 * sizeof(float4));  // range boxes

// Scratch of re_lbvh_build_static: about 5.3 MB per device the library is
// loaded on.  Nothing in it needs an initial value: each call re-initialises
// the scene bounds and flags before using them.
static __device__ __align__(256) unsigned char g_lbvh_static_scratch[kStaticScratchBytes];

// Device address of g_lbvh_static_scratch per device, resolved once with that
// device current.
std::mutex g_static_mutex;
void* g_static_addr[64] = {};

}  // namespace

}  // namespace re

extern "C" RE_API re_status re_lbvh_build_static(const re_float4* positions, const uint32_t* stable_ids,
                                                 uint32_t count, uint32_t* order_out, re_lbvh_node* nodes_out,
                                                 void* stream) {
    using namespace re;
    if (positions == nullptr || stable_ids == nullptr || order_out == nullptr || (count > 1 && nodes_out == nullptr))
        return set_error(RE_INVALID_ARGUMENT, "null argument");
    if (count == 0) return set_error(RE_INVALID_ARGUMENT, "LBVH build of zero triangles");
    if (count > kStaticMaxTris)
        return set_error(RE_INVALID_ARGUMENT, "re_lbvh_build_static: " + std::to_string(count) +
                                                  " triangles exceed the static scratch capacity of " +
                                                  std::to_string(kStaticMaxTris));
    if ((reinterpret_cast<uintptr_t>(positions) & 15u) != 0 || (reinterpret_cast<uintptr_t>(nodes_out) & 15u) != 0 ||
        (reinterpret_cast<uintptr_t>(stable_ids) & 3u) != 0 || (reinterpret_cast<uintptr_t>(order_out) & 3u) != 0)
        return set_error(RE_INVALID_ARGUMENT, "re_lbvh_build_static: misaligned buffer");
    // A launch error left by the caller's earlier work would otherwise be
    // picked up by the check after this call's launches and reported as this
    // build's failure: report it as what it is, before launching anything.
    const cudaError_t pending = cudaGetLastError();
    if (pending != cudaSuccess)
        return set_error(RE_CUDA_ERROR, std::string("re_lbvh_build_static: CUDA error pending from earlier work: ") +
                                            cudaGetErrorString(pending));
    int device = 0;
    RE_CUDA_TRY(cudaGetDevice(&device));
    if (device < 0 || device >= 64) return set_error(RE_INVALID_ARGUMENT, "device ordinal out of range");
    char* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_static_mutex);
        if (g_static_addr[device] == nullptr) {
            void* addr = nullptr;
            RE_CUDA_TRY(cudaGetSymbolAddress(&addr, g_lbvh_static_scratch));
            g_static_addr[device] = addr;
        }
        base = static_cast<char*>(g_static_addr[device]);
    }
    const uint32_t n = count;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base + off;
        off += align256(bytes);
        return p;
    };
    auto* head = reinterpret_cast<BuildHeader*>(take(sizeof(BuildHeader)));
    auto* keys = reinterpret_cast<unsigned long long*>(take(size_t(kStaticMaxTris) * 8));
    auto* sorted = reinterpret_cast<unsigned long long*>(take(size_t(kStaticMaxTris) * 8));
    const RangeBoxes boxes{reinterpret_cast<float4*>(take(2 * size_t(kStaticMaxTris) * 2 * sizeof(float4))),
                           RangeBoxes::span(n)};
    if (off > kStaticScratchBytes) return set_error(RE_FATAL_QUEUE, "static LBVH scratch layout overflow");

    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const TriangleView view{reinterpret_cast<const float4*>(positions), stable_ids, 3u, 1u};
    k_init<<<1, 32, 0, st>>>(head);
    k_bounds<<<std::min<uint32_t>(148u, (n + 255) / 256), 256, 0, st>>>(view, n, head);
    k_morton<<<(n + 255) / 256, 256, 0, st>>>(view, n, head, keys, nullptr);
    RE_CUDA_TRY(cluster_sort(keys, n, head, sorted, order_out, st));
    if (n > 1) {
        k_leaf_boxes<<<(n + 255) / 256, 256, 0, st>>>(view, order_out, n, boxes);
        RE_CUDA_TRY(seg_build(boxes, n, st));
        // Stable IDs are not checked for uniqueness here (that would need a
        // read-back): equal (code, ID) keys are split by sorted position.
        k_karras_static<<<(n - 1 + 255) / 256, 256, 0, st>>>(sorted, int(n), boxes, nodes_out);
    }
    RE_CUDA_TRY(cudaGetLastError());
    return clear_error();
}
