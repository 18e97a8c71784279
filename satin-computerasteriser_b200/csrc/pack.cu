// pack.cu — the GPU packer: raw points -> Morton-ordered, LOD-bucketed,
// split-precision batches written straight into a cloud's slot pool.
//
// Restates GPUPacker.encodePack (GPUPacker.swift:204-392) and its kernels
// (Pipelines/GPUPacker/Shaders.metal:41-414), which in turn mirror the CPU
// PackedPointCloudFixtures.pack (PackedPointCloudFixtures.swift:30-344):
//   1 load, bounds  raw input to 16-byte records {x, y, z, rgba8} (records on
//                   the device are read in place), and the AABB of every
//                   segment (order-preserving flipped-bit min/max), read back
//                   once for the Morton scales and the LOD grids
//   2 morton        10 bits/axis (30-bit key) or 21 bits/axis (63-bit key),
//                   with the histograms of every 8-bit digit
//   3 sort          stable LSD radix of (key, input index), one single-sweep
//                   pass per digit (decoupled look-back; the first pass
//                   makes the input indices)                     [radix.cu]
//   4 gather        positions in Morton order, levels = maxLevel
//   5 LOD           per level, coarsest first: dense voxel grid, atomicMin
//                   of the Morton position claims a voxel for the first
//                   eligible point in sorted order (the CPU's "first point
//                   to occupy an empty voxel"); the claims of a level ride
//                   in the kernel before (the gather, or the previous
//                   level's assignment), the last level's assignment in the
//                   batch kernel
//   6-7 batches     one CTA per batch, a contiguous segment per warp:
//                   AABB, level counts, RasterBatch with the cumulative LOD
//                   counts; stable level-ascending scatter (warp ballots, no
//                   block barrier) of the points, quantised to 30 bits an
//                   axis in three 10-bit/axis words, with colours, levels
//                   and source indices.
// Every stage is one launch over all segments of a run (the chunks of one
// cr_pack_chunks call, or the one cloud of cr_pack): a streamed node of 140
// thousand points fills a quarter of the GPU, and launches and read-backs
// took longer than its kernels (ten nodes: 2.04 ms one after the other, 0.45
// ms together).
// Host-side float math (scale, voxel sizes, grid dims) is compiled without
// contraction and uses the same operation order as the CPU oracle.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "cr_device.cuh"
#include "cr_internal.h"
#include "cr_pack.h"

namespace {

constexpr int kThreads = 256;
constexpr uint64_t kLodCellCap = 1ull << 28;  // 1 GiB of uint32 voxels

__host__ __device__ __forceinline__ uint32_t flip(float f) {
#ifdef __CUDA_ARCH__
    const uint32_t b = __float_as_uint(f);
#else
    uint32_t b;
    std::memcpy(&b, &f, 4);
#endif
    return b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
}
__host__ __device__ __forceinline__ float unflip(uint32_t u) {
    const uint32_t b = u ^ ((u >> 31) ? 0x80000000u : 0xffffffffu);
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float f;
    std::memcpy(&f, &b, 4);
    return f;
#endif
}

// Ten bits spread to every third place.  The copies do not overlap, so a
// shift and an or are one multiplication.
__device__ __forceinline__ uint32_t spread10(uint32_t v) {
    uint32_t x = v & 0x3ffu;
    x = (x * 0x10001u) & 0x030000ffu;
    x = (x * 0x101u) & 0x0300f00fu;
    x = (x * 0x11u) & 0x030c30c3u;
    x = (x * 0x5u) & 0x09249249u;
    return x;
}

struct LoadArgs {
    const uint8_t *pos;
    uint32_t pos_stride;
    const uint8_t *col;
    uint32_t col_stride;
    int col_format;
};

struct MortonArgs {
    float bmin[3];
    float scale[3];
    float top;
};

struct LodArgs {
    float bmin[3];
    float inv;
    uint32_t dims[3];
    uint32_t *grid;  // this level's voxels
};

constexpr int kMaxLevels = 8;

}  // namespace

// One segment of a run: points packed into slots of their own.  Its keys,
// indices, levels and sorted points are elements [begin, begin + n) of the
// scratch arrays.
struct PackSeg {
    LoadArgs la;
    const float4 *pos;  // the records: the staged copy, or the caller's
    float4 *stage;      // where the load writes them (null: read in place)
    uint64_t begin;
    uint32_t n;
    uint32_t block0;      // first CTA of the per-point kernels (kPointsPerCta each)
    uint32_t batch0;      // first CTA of the batch kernel
    uint32_t first_slot;  // first slot of the pool
    MortonArgs m;
    LodArgs lod[kMaxLevels - 1];
};

namespace {

// The segments of a launch: one rides in the kernel's parameters (ONE), more
// are read from device memory.
struct Segs {
    PackSeg one;
    const PackSeg *list;
    uint32_t n;
};

// Segment of block b among the segments' first blocks.
template <bool ONE, uint32_t PackSeg::*FIRST>
__device__ __forceinline__ uint32_t seg_of(const Segs &s, uint32_t b) {
    uint32_t lo = 0;
    if (!ONE)
        for (uint32_t hi = s.n; hi - lo > 1u;) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s.list[mid].*FIRST <= b)
                lo = mid;
            else
                hi = mid;
        }
    return lo;
}
template <bool ONE>
__device__ __forceinline__ const PackSeg &seg_at(const Segs &s, uint32_t i) {
    if constexpr (ONE)
        return s.one;
    else
        return s.list[i];
}

// Stages 0 and 1: raw input -> float4 positions + packed RGBA8
// (GPUPacker/Shaders.metal:219-235; colour rule: uint(clamp(c, 0, 1) * 255),
// truncating) and the bounds (packBounds, Shaders.metal:71-105).  One 16-byte
// record per point: x, y, z and the packed RGBA8 colour's bits in w (moved,
// never computed on), so the Morton-order gather brings both with one access.
// blockIdx.y = segment.  One set of bounds atomics per CTA (a set per warp
// kept the six words of a 140-thousand-point node busy for 18 us).
constexpr int kLoadRounds = 4;
template <bool ONE>
__global__ void __launch_bounds__(kThreads)
    pack_load_bounds(const __grid_constant__ Segs segs, uint32_t *__restrict__ bounds) {
    const PackSeg &sg = seg_at<ONE>(segs, blockIdx.y);
    const uint32_t n = sg.n;
    const LoadArgs a = sg.la;
    const float4 *pos = sg.pos;
    float4 *stage = sg.stage;
    uint32_t mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
    const uint64_t step = (uint64_t)gridDim.x * kThreads;
    auto widen = [&](const float4 &p) {
        const uint32_t f[3] = {flip(p.x), flip(p.y), flip(p.z)};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            mn[d] = min(mn[d], f[d]);
            mx[d] = max(mx[d], f[d]);
        }
    };
    uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (!stage) {
        for (; i + step * (kLoadRounds - 1) < n; i += step * kLoadRounds) {
            float4 p[kLoadRounds];
#pragma unroll
            for (int k = 0; k < kLoadRounds; ++k) p[k] = pos[i + step * k];
#pragma unroll
            for (int k = 0; k < kLoadRounds; ++k) widen(p[k]);
        }
        for (; i < n; i += step) widen(pos[i]);
    } else {
        for (; i < n; i += step) {
            const float *q = reinterpret_cast<const float *>(a.pos + i * a.pos_stride);
            uint32_t col;
            if (a.col_format == 1) {
                col = *reinterpret_cast<const uint32_t *>(a.col + i * a.col_stride);
            } else {
                const float *c = reinterpret_cast<const float *>(a.col + i * a.col_stride);
                const uint32_t r = (uint32_t)(fminf(fmaxf(c[0], 0.0f), 1.0f) * 255.0f);
                const uint32_t g = (uint32_t)(fminf(fmaxf(c[1], 0.0f), 1.0f) * 255.0f);
                const uint32_t b = (uint32_t)(fminf(fmaxf(c[2], 0.0f), 1.0f) * 255.0f);
                const uint32_t al = (uint32_t)(fminf(fmaxf(c[3], 0.0f), 1.0f) * 255.0f);
                col = r | (g << 8) | (b << 16) | (al << 24);
            }
            const float4 p = make_float4(q[0], q[1], q[2], __uint_as_float(col));
            stage[i] = p;
            widen(p);
        }
    }
    __shared__ uint32_t part[6][kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const uint32_t x = __reduce_min_sync(0xffffffffu, mn[d]);
        const uint32_t y = __reduce_min_sync(0xffffffffu, ~mx[d]);
        if (lane == 0) {
            part[d][warp] = x;
            part[3 + d][warp] = y;
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        uint32_t x = 0xffffffffu;
        for (int w = 0; w < kThreads / 32; ++w) x = min(x, part[threadIdx.x][w]);
        atomicMin(&bounds[8 * blockIdx.y + threadIdx.x], x);
    }
}

// Morton keys.  63 bits: the low ten bits and the high eleven of each axis
// are spread apart as 32-bit words, which the integer pipe does in fewer
// operations than 64-bit shifts and masks.
__device__ __forceinline__ uint32_t interleave10(uint32_t x, uint32_t y, uint32_t z) {
    return (spread10(x) << 2) | (spread10(y) << 1) | spread10(z);
}
__device__ __forceinline__ void morton_key(uint32_t x, uint32_t y, uint32_t z, uint32_t &key) {
    key = interleave10(x, y, z);
}
__device__ __forceinline__ void morton_key(uint32_t x, uint32_t y, uint32_t z,
                                           unsigned long long &key) {
    const uint32_t lo = interleave10(x, y, z);                    // key bits 0..29
    const uint32_t mid = interleave10(x >> 10, y >> 10, z >> 10);  // key bits 30..59
    const uint32_t top = ((x >> 20) << 2) | ((y >> 20) << 1) | (z >> 20);  // key bits 60..62
    key = ((unsigned long long)((top << 28) | (mid >> 2)) << 32) | (lo | (mid << 30));
}

// Stage 2: Morton keys (packMorton, GPUPacker/Shaders.metal:109-126) and the
// histograms of their 8-bit digits (a CTA counts in shared memory and adds
// its counts once); the identity index the reference writes beside the keys
// is made by the sort's first pass instead.  blockIdx.y = segment.  100M
// 63-bit keys: 480 us, where the keys (577 us) and their histograms (362 us,
// reading them again) were two kernels.
template <typename K, bool ONE>
__global__ void __launch_bounds__(kThreads)
    pack_morton(const __grid_constant__ Segs segs, K *__restrict__ keys,
                uint32_t *__restrict__ hist) {
    constexpr int kPasses = sizeof(K) == 8 ? 8 : 4;
    __shared__ uint32_t sh[kPasses * 256];
    for (int i = threadIdx.x; i < kPasses * 256; i += kThreads) sh[i] = 0u;
    __syncthreads();
    const PackSeg &sg = seg_at<ONE>(segs, blockIdx.y);
    const uint32_t n = sg.n;
    const float4 *pos = sg.pos;
    const MortonArgs m = sg.m;
    keys += sg.begin;
    const uint64_t step = (uint64_t)gridDim.x * kThreads;
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += step) {
        const float4 p = pos[i];
        const uint32_t qx = (uint32_t)fminf(fmaxf((p.x - m.bmin[0]) * m.scale[0], 0.0f), m.top);
        const uint32_t qy = (uint32_t)fminf(fmaxf((p.y - m.bmin[1]) * m.scale[1], 0.0f), m.top);
        const uint32_t qz = (uint32_t)fminf(fmaxf((p.z - m.bmin[2]) * m.scale[2], 0.0f), m.top);
        K k;
        morton_key(qx, qy, qz, k);
        keys[i] = k;
#pragma unroll
        for (int d = 0; d < kPasses; ++d)
            atomicAdd(&sh[d * 256 + ((uint32_t)(k >> (8 * d)) & 0xffu)], 1u);
    }
    __syncthreads();
    uint32_t *out = hist + (size_t)blockIdx.y * kRadixMaxPasses * 256;
    for (int i = threadIdx.x; i < kPasses * 256; i += kThreads)
        if (sh[i]) atomicAdd(&out[i], sh[i]);
}

__device__ __forceinline__ uint32_t lod_cell(const float4 &p, const LodArgs &a) {
    const float lx = (p.x - a.bmin[0]) * a.inv;
    const float ly = (p.y - a.bmin[1]) * a.inv;
    const float lz = (p.z - a.bmin[2]) * a.inv;
    const uint32_t cx = min((uint32_t)max(0, (int)floorf(lx)), a.dims[0] - 1u);
    const uint32_t cy = min((uint32_t)max(0, (int)floorf(ly)), a.dims[1] - 1u);
    const uint32_t cz = min((uint32_t)max(0, (int)floorf(lz)), a.dims[2] - 1u);
    return cx + a.dims[0] * (cy + a.dims[1] * cz);  // a grid has at most kLodCellCap cells
}

// Stage 5 (packLODClaim / packLODAssign, GPUPacker/Shaders.metal:337-371).
// The points are in Morton order, so neighbouring lanes often share a cell;
// lanes carry increasing indices, so the lowest lane of each group of lanes
// with the same cell holds the group's minimum and alone does the atomicMin
// (the grid ends the same: min is order-independent).  The claims are fused
// into the kernels that read the Morton-ordered points anyway: the gather
// also claims the coarsest level (every point is still unassigned there),
// and the assignment of level L also claims level L + 1 for the points it
// leaves unassigned (each level has its own grid), so the points are read
// once per level instead of twice.
// MOVED: ties were put in order, so a lane's index may be below that of a lane
// before it.
template <bool MOVED>
__device__ __forceinline__ void lod_claim_one(bool part, const float4 &p, uint32_t i,
                                              const LodArgs &a) {
    const unsigned act = __ballot_sync(0xffffffffu, part);
    if (!part) return;
    const uint32_t cell = lod_cell(p, a);
    const unsigned same = __match_any_sync(act, cell);
    if (MOVED) i = __reduce_min_sync(same, i);
    if ((int)(__ffs(same) - 1) == (int)(threadIdx.x & 31u)) atomicMin(&a.grid[cell], i);
}

// The sort's values of a segment: where its indices ended up (null: the
// input order stands).
__device__ __forceinline__ const uint32_t *sorted_index(const uint32_t *vals0,
                                                        const uint32_t *vals1, uint32_t set,
                                                        uint64_t begin) {
    return set == 0u ? nullptr : ((__popc(set) & 1) ? vals1 : vals0) + begin;
}

// The kernels over the sorted points: four points per thread, a CTA's width
// apart (each load coalesced over the warp), every load of the four issued
// before the first is used: a point a thread waited for its level, its record
// and its voxel one after the other with nothing else in flight (100M points:
// an assignment with claims 604 us, 352 us so).
constexpr int kEach = 4;
constexpr uint32_t kPointsPerCta = kEach * kThreads;

// What the sort left in order (RadixBuffers, RadixScratch).  Where it left out
// low digits (ties), the gather orders the keys that agree above them, and the
// other values buffer holds the final indices.
struct Sorted {
    uint32_t *vals[2];
    const unsigned long long *keys[2];  // 64-bit keys, else unused
    const uint32_t *runs, *ties;
    int want_index;  // the final indices are read (source indices asked for)
};
__device__ __forceinline__ const uint32_t *final_index(const Sorted &so, uint32_t si,
                                                       uint64_t begin) {
    const uint32_t set = so.runs[si];
    if (so.ties[si] != 0u) return ((__popc(set) & 1) ? so.vals[0] : so.vals[1]) + begin;
    return sorted_index(so.vals[0], so.vals[1], set, begin);
}

// Places of a CTA's keys among the keys that agree with them above `low` (at
// most 32) bits: in a run of such keys, which are neighbours, a key stands after
// those with smaller low bits and the equal ones before it.  The CTA's keys are
// staged in shared memory; a run that leaves it is read in place.  Most runs are
// of a few keys, which are looked at one after the other.  A longer run's ends are
// searched for, its keys being sorted above the low bits, and its low words, which
// differ in those bits alone, are counted with nothing to decide between two
// reads.  A pack of 600 thousand points of which 700 agree took 408 us key by key,
// 258 so (310 with every digit sorted); of 100M points of which three thousand
// agree 9.65 ms, 8.99 so (10.9).
__device__ __forceinline__ void tie_places(const unsigned long long *__restrict__ keys, uint32_t n,
                                           uint64_t first, uint32_t low, unsigned long long *skey,
                                           uint32_t (&place)[kEach]) {
    const uint32_t count = (uint32_t)min((uint64_t)n - first, (uint64_t)kPointsPerCta);
    const uint32_t base = (uint32_t)first;
    constexpr uint32_t kNear = 7;
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
        const uint32_t t = threadIdx.x + k * kThreads;
        if (t < count) skey[t] = __ldg(keys + first + t);
    }
    __syncthreads();
    auto key_at = [&](uint32_t i) {
        const uint32_t t = i - base;  // wraps below the CTA's keys
        return t < count ? skey[t] : __ldg(keys + i);
    };
    const unsigned long long mask = (1ull << low) - 1ull;
    uint32_t runs = 0;  // bit k: key k's run goes on past kNear keys on a side
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
        const uint32_t t = threadIdx.x + k * kThreads, i = base + t;
        place[k] = i;
        if (t >= count) continue;
        const unsigned long long mine = skey[t];
        uint32_t at = i, far = 0u;
        for (uint32_t j = i; j > 0u; --j) {
            const unsigned long long other = key_at(j - 1u);
            if ((other ^ mine) & ~mask) break;
            at -= (other & mask) > (mine & mask) ? 1u : 0u;
            if (i - j == kNear) {
                far = 1u;
                break;
            }
        }
        for (uint32_t j = i + 1u; j < n; ++j) {
            const unsigned long long other = key_at(j);
            if ((other ^ mine) & ~mask) break;
            at += (other & mask) < (mine & mask) ? 1u : 0u;
            if (j - i > kNear) {
                far = 1u;
                break;
            }
        }
        place[k] = at;
        if (far) runs |= 1u << k;
    }
    for (; runs; runs &= runs - 1u) {
        const int which = __ffs(runs) - 1;
        const uint32_t i = base + threadIdx.x + which * kThreads;
        const unsigned long long mine = skey[i - base];
        auto agrees = [&](uint32_t j) { return ((key_at(j) ^ mine) >> low) == 0ull; };
        uint32_t s = i, e = i + 1u;  // the run is [s, e)
        uint32_t step = 1u;
        for (; step <= s && agrees(s - step); step <<= 1) s -= step;
        while (step >>= 1)
            if (step <= s && agrees(s - step)) s -= step;
        step = 1u;
        for (; step <= n - e && agrees(e - 1u + step); step <<= 1) e += step;
        while (step >>= 1)
            if (step <= n - e && agrees(e - 1u + step)) e += step;
        const uint32_t my = (uint32_t)mine;
        uint32_t before = 0;
        auto rank = [&](auto low_at) {
#pragma unroll 8
            for (uint32_t j = s; j < i; ++j) before += low_at(j) <= my ? 1u : 0u;
#pragma unroll 8
            for (uint32_t j = i + 1u; j < e; ++j) before += low_at(j) < my ? 1u : 0u;
        };
        if (s >= base && e - base <= count)
            rank([&](uint32_t j) { return (uint32_t)skey[j - base]; });
        else
            rank([&](uint32_t j) {
                return __ldg(reinterpret_cast<const uint32_t *>(keys) + 2 * (size_t)j);
            });
#pragma unroll
        for (int k = 0; k < kEach; ++k)
            if (k == which) place[k] = s + before;
    }
}

// Stage 4: gather into Morton order, all levels at max_level (packLODInit),
// and the coarsest level's claims when there is more than one level.  Bound by
// its random 16-byte reads, of which five CTAs an SM keep more in flight: 400M
// points 36.55 ms a pack with the 64 registers that it would take, 35.83 with 48,
// 10M 1049 and 1020 us.
template <bool ONE>
__global__ void __launch_bounds__(kThreads, 5)
    pack_gather_claim(const __grid_constant__ Segs segs, const __grid_constant__ Sorted so,
                      float4 *__restrict__ sorted, uint8_t *__restrict__ lv, uint32_t max_level) {
    __shared__ unsigned long long skey[ONE ? kPointsPerCta : 1];
    const uint32_t si = seg_of<ONE, &PackSeg::block0>(segs, blockIdx.x);
    const PackSeg &sg = seg_at<ONE>(segs, si);
    const uint64_t i0 = (uint64_t)(blockIdx.x - sg.block0) * kPointsPerCta + threadIdx.x;
    const uint32_t set = so.runs[si];
    const uint32_t *idx = sorted_index(so.vals[0], so.vals[1], set, sg.begin);
    const float4 *pos = sg.pos;
    uint32_t from[kEach], place[kEach];
    float4 p[kEach];
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
        const uint64_t i = i0 + k * kThreads;
        place[k] = (uint32_t)i;
        // Bounded, since a sort that gave up waiting leaves any value.
        from[k] = i < sg.n && idx ? min(__ldg(idx + i), sg.n - 1u) : (uint32_t)i;
    }
#pragma unroll
    for (int k = 0; k < kEach; ++k)
        p[k] = i0 + k * kThreads < sg.n ? __ldg(pos + from[k]) : make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t low = ONE ? so.ties[0] : 0u;  // only a single segment has any
    if (ONE && low != 0u)
        tie_places(so.keys[__popc(set) & 1], sg.n, i0 - threadIdx.x, low, skey, place);
#pragma unroll
    for (int k = 0; k < kEach; ++k)
        if (i0 + k * kThreads < sg.n) {
            sorted[sg.begin + place[k]] = p[k];
            lv[sg.begin + place[k]] = (uint8_t)max_level;
            if (ONE && low != 0u && so.want_index)
                ((__popc(set) & 1) ? so.vals[0] : so.vals[1])[place[k]] = from[k];
        }
    if (max_level > 0u)
#pragma unroll
        for (int k = 0; k < kEach; ++k)
            lod_claim_one<ONE>(i0 + k * kThreads < sg.n, p[k], place[k], sg.lod[0]);
}

// The holder of a voxel sets it back to "empty" when it takes its level (every
// other point of the voxel still reads a value that is not its own index), so
// the grids are empty again after a run and need no clearing before the next.

// Assignment of a level and the claims of the next (the last level's
// assignment rides in the batch kernel).
template <bool ONE>
__global__ void __launch_bounds__(kThreads)
    pack_lod_assign(const __grid_constant__ Segs segs, const float4 *__restrict__ sorted,
                    uint8_t *__restrict__ lv, uint32_t level, uint32_t max_level) {
    const PackSeg &sg = seg_at<ONE>(segs, seg_of<ONE, &PackSeg::block0>(segs, blockIdx.x));
    const uint64_t i0 = (uint64_t)(blockIdx.x - sg.block0) * kPointsPerCta + threadIdx.x;
    const LodArgs &a = sg.lod[level];
    bool left[kEach];
    float4 p[kEach];
    uint32_t cell[kEach], holder[kEach];
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
        const uint64_t i = i0 + k * kThreads;
        left[k] = i < sg.n && lv[sg.begin + i] == max_level;
        // The record is read before its level is known: nearly all are left.
        p[k] = i < sg.n ? __ldg(sorted + sg.begin + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
        cell[k] = lod_cell(p[k], a);
        // Through L1: the claims are the kernel's before, and of what is written
        // now, no value but its own index matters to a point.  A pack of 20M points
        // in one place takes 3.75 ms with the voxels read from L2, 2.41 so; of
        // 100M points of terrain 8.85 and 8.75.
        holder[k] = left[k] ? a.grid[cell[k]] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
        const uint64_t i = i0 + k * kThreads;
        if (left[k] && holder[k] == (uint32_t)i) {
            a.grid[cell[k]] = 0xffffffffu;  // empty again for the next run
            lv[sg.begin + i] = (uint8_t)level;
            left[k] = false;
        }
    }
#pragma unroll
    for (int k = 0; k < kEach; ++k)
        lod_claim_one<false>(left[k], p[k], (uint32_t)(i0 + k * kThreads), sg.lod[level + 1]);
}

// Stages 6 and 7: per batch AABB, RasterBatch and stable level bucketing
// (packBatchAABB + packBucketLOD, GPUPacker/Shaders.metal:243-284, 383-414),
// then final order and quantisation (packQuantize, Shaders.metal:288-309).
// One CTA per batch; each warp owns a contiguous segment of the batch's
// points.  Pass 1: the AABB and the warp's per-level counts (ballots).  The
// counts give every warp its first slot per level (the batch's exclusive
// level prefix plus the counts of the warps before it), so pass 2 needs no
// block barrier: each warp walks its segment in order, 32 points a round,
// places each point after the earlier points of its level (ballot rank) and
// writes it there quantised.  Both passes load kBatchRounds rounds ahead.
// Bound by memory: pass 1 reads the batch from DRAM (17 bytes a point), pass
// 2 reads it again from L2 (two or three 10,240-point batches of 164 KB an
// SM are in flight), and the points of a level land next to each other, so
// the stores of a round fill one run per level.
// NL: the levels there can be (4, the default, or 8): a ballot each in both
// passes.
constexpr int kBatchRounds = 4;
// A warp for every kBatchRounds rounds of the largest batch, up to this many
// threads (5M points in batches of 64: the pack 3180 us with 512 threads to every
// batch, 2000 so).
constexpr uint32_t kBatchThreads = 512;
uint32_t batch_threads(uint32_t ppb) {
    return std::min(kBatchThreads, 32u * ((ppb + 32u * kBatchRounds - 1u) / (32u * kBatchRounds)));
}
template <int NL, bool ONE>
__global__ void __launch_bounds__(kBatchThreads)
    pack_batches(const __grid_constant__ Segs segs, const float4 *__restrict__ sorted,
                 uint8_t *__restrict__ lv, uint32_t max_level, uint32_t ppb,
                 const __grid_constant__ Sorted so, cr_raster_batch *__restrict__ batches,
                 uint32_t *__restrict__ low, uint32_t *__restrict__ med,
                 uint32_t *__restrict__ high, uint32_t *__restrict__ colors,
                 uint8_t *__restrict__ levels, uint32_t *__restrict__ src_out) {
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ uint32_t red[6][kBatchThreads / 32];
    __shared__ uint32_t wcnt[kBatchThreads / 32][NL];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t si = seg_of<ONE, &PackSeg::batch0>(segs, blockIdx.x);
    const PackSeg &sg = seg_at<ONE>(segs, si);
    const uint32_t batch = blockIdx.x - sg.batch0;
    const uint64_t start = (uint64_t)batch * ppb;  // in the segment
    const uint32_t total = (uint32_t)min((uint64_t)sg.n - start, (uint64_t)ppb);
    const uint32_t slot = sg.first_slot + batch;
    const uint64_t pool = (uint64_t)slot * ppb;
    const uint32_t seg = (total + warps - 1u) / warps;
    const uint32_t s0 = min(total, (uint32_t)warp * seg);
    const uint32_t s1 = min(total, (uint32_t)(warp + 1) * seg);
    const float4 *bsorted = sorted + sg.begin + start;
    uint8_t *blv = lv + sg.begin + start;
    // 1. AABB and level counts of the warp's segment.
    uint32_t mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
    uint32_t c[NL] = {};
    for (uint32_t r0 = s0; r0 < s1; r0 += 32u * kBatchRounds) {
        float4 p[kBatchRounds];
        uint32_t l[kBatchRounds];
#pragma unroll
        for (int k = 0; k < kBatchRounds; ++k) {
            const uint32_t i = r0 + 32u * k + lane;
            l[k] = i < s1 ? (blv[i] & 7u) : 8u;
            p[k] = i < s1 ? bsorted[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // The last level's assignment (pass 2 of this thread reads what it
        // stores here).
        if (max_level > 0u) {
            const LodArgs &a = sg.lod[max_level - 1u];
            uint32_t cell[kBatchRounds], holder[kBatchRounds];
#pragma unroll
            for (int k = 0; k < kBatchRounds; ++k) {
                cell[k] = lod_cell(p[k], a);
                holder[k] = l[k] == max_level ? a.grid[cell[k]] : 0xffffffffu;
            }
#pragma unroll
            for (int k = 0; k < kBatchRounds; ++k) {
                const uint32_t i = r0 + 32u * k + lane;
                if (l[k] == max_level && holder[k] == (uint32_t)start + i) {
                    a.grid[cell[k]] = 0xffffffffu;  // empty again for the next run
                    l[k] = max_level - 1u;
                    blv[i] = (uint8_t)l[k];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kBatchRounds; ++k) {
            if (l[k] < 8u) {
                const uint32_t f[3] = {flip(p[k].x), flip(p[k].y), flip(p[k].z)};
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    mn[a] = min(mn[a], f[a]);
                    mx[a] = max(mx[a], f[a]);
                }
            }
#pragma unroll
            for (int L = 0; L < NL; ++L) c[L] += __popc(__ballot_sync(kFull, l[k] == (uint32_t)L));
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t x = __reduce_min_sync(kFull, mn[a]);
        const uint32_t y = __reduce_max_sync(kFull, mx[a]);
        if (lane == 0) {
            red[a][warp] = x;
            red[3 + a][warp] = y;
        }
    }
    if (lane < NL) {
        uint32_t mine = 0;
#pragma unroll
        for (int L = 0; L < NL; ++L)
            if (lane == L) mine = c[L];
        wcnt[warp][lane] = mine;
    }
    __syncthreads();
    // 2. This warp's first slot (from the batch start) per level; the box.
    uint32_t run[NL], cum[8];
    {
        uint32_t acc = 0;
#pragma unroll
        for (int L = 0; L < NL; ++L) {
            const uint32_t x = lane < warps ? wcnt[lane][L] : 0u;
            const uint32_t tot = __reduce_add_sync(kFull, x);
            const uint32_t before = __reduce_add_sync(kFull, lane < warp ? x : 0u);
            run[L] = acc + before;
            acc += tot;
            cum[L] = acc;
        }
#pragma unroll
        for (int L = NL; L < 8; ++L) cum[L] = acc;
    }
    float bmin[3], size[3], bmax[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        bmin[a] = unflip(__reduce_min_sync(kFull, lane < warps ? red[a][lane] : 0xffffffffu));
        bmax[a] = unflip(__reduce_max_sync(kFull, lane < warps ? red[3 + a][lane] : 0u));
        size[a] = fmaxf(bmax[a] - bmin[a], 0.000001f);
    }
    if (threadIdx.x == 0) {
        cr_raster_batch rb;
        rb.state = 1;
        rb.minX = bmin[0];
        rb.minY = bmin[1];
        rb.minZ = bmin[2];
        rb.maxX = bmax[0];
        rb.maxY = bmax[1];
        rb.maxZ = bmax[2];
        rb.numPoints = total;
        rb.firstPoint = slot * ppb;
        rb.fileIndex = 0;
        rb.lodCum01 = cum[0] | (cum[1] << 16);
        rb.lodCum23 = cum[2] | (cum[3] << 16);
        rb.lodCum45 = cum[4] | (cum[5] << 16);
        rb.lodCum67 = cum[6] | (cum[7] << 16);
        rb.padding7 = 0;
        rb.padding8 = 0;
        batches[slot] = rb;
    }
    // 3. Stable bucketing of the warp's segment, each point quantised into
    // its final place.
    const uint32_t *idx = src_out ? final_index(so, si, sg.begin) : nullptr;
    for (uint32_t r0 = s0; r0 < s1; r0 += 32u * kBatchRounds) {
        float4 p[kBatchRounds];
        uint32_t raw[kBatchRounds];
#pragma unroll
        for (int k = 0; k < kBatchRounds; ++k) {
            const uint32_t i = r0 + 32u * k + lane;
            raw[k] = i < s1 ? (uint32_t)blv[i] : 0xffu;
            p[k] = i < s1 ? bsorted[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < kBatchRounds; ++k) {
            const uint32_t i = r0 + 32u * k + lane;
            const bool v = i < s1;
            const uint32_t l = v ? (raw[k] & 7u) : 8u;
            uint32_t dst = 0;
#pragma unroll
            for (int L = 0; L < NL; ++L) {
                const uint32_t b = __ballot_sync(kFull, l == (uint32_t)L);
                if (l == (uint32_t)L) dst = run[L] + __popc(b & lt);
                run[L] += __popc(b);
            }
            if (v && dst < total) {  // always true: the ranks come from the same levels
                const float nx = fminf(fmaxf((p[k].x - bmin[0]) / size[0], 0.0f), 0.99999994f);
                const float ny = fminf(fmaxf((p[k].y - bmin[1]) / size[1], 0.0f), 0.99999994f);
                const float nz = fminf(fmaxf((p[k].z - bmin[2]) / size[2], 0.0f), 0.99999994f);
                // Float(2^30 - 1) rounds to 2^30 in f32.
                const uint32_t qx = (uint32_t)(nx * 1073741824.0f);
                const uint32_t qy = (uint32_t)(ny * 1073741824.0f);
                const uint32_t qz = (uint32_t)(nz * 1073741824.0f);
                const uint64_t j = pool + dst;
                low[j] = ((qx >> 20) & 1023u) | (((qy >> 20) & 1023u) << 10) |
                         (((qz >> 20) & 1023u) << 20);
                med[j] = ((qx >> 10) & 1023u) | (((qy >> 10) & 1023u) << 10) |
                         (((qz >> 10) & 1023u) << 20);
                high[j] = (qx & 1023u) | ((qy & 1023u) << 10) | ((qz & 1023u) << 20);
                colors[j] = __float_as_uint(p[k].w);
                levels[j] = (uint8_t)raw[k];
                if (src_out)
                    src_out[sg.begin + start + dst] =
                        idx ? idx[start + i] : (uint32_t)(start + i);
            }
        }
    }
}

unsigned grid_for(uint64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

template <typename T>
cr_status grow(T **p, uint64_t &cap, uint64_t want_elems) {
    if (*p && cap >= want_elems) return CR_OK;
    if (*p) cudaFree(*p);
    *p = nullptr;
    cudaError_t e = cudaMalloc((void **)p, std::max<uint64_t>(want_elems, 1) * sizeof(T));
    if (e != cudaSuccess) {
        *p = nullptr;
        cap = 0;
        return cri::cuda_fail(e, "cudaMalloc (pack scratch)");
    }
    cap = want_elems;
    return CR_OK;
}

// Keys are sized for 64-bit words so either key width fits.
constexpr uint64_t kPointScratch = 2 * sizeof(float4) + 2 * 8 + 3 * 4 + 1;  // bytes a point
cr_status ensure_points(PackScratch &s, uint64_t n) {
    if (s.cap_points >= n && s.keys[0]) return CR_OK;
    pack_scratch_free(s);
    const uint64_t m = std::max<uint64_t>(n, 1) + 64;
    cudaError_t e;
#define ALLOC(ptr, bytes)                                                   \
    do {                                                                    \
        e = cudaMalloc((void **)&(ptr), (bytes));                           \
        if (e != cudaSuccess) {                                             \
            pack_scratch_free(s);                                           \
            return cri::cuda_fail(e, "cudaMalloc (pack scratch)");          \
        }                                                                   \
    } while (0)
    ALLOC(s.pos, m * sizeof(float4));
    ALLOC(s.keys[0], m * 8);
    ALLOC(s.keys[1], m * 8);
    ALLOC(s.idx[0], m * 4);
    ALLOC(s.idx[1], m * 4);
    ALLOC(s.sorted, m * sizeof(float4));
    ALLOC(s.lv_morton, (m + 15) & ~15ull);
    ALLOC(s.src_idx, m * 4);
#undef ALLOC
    s.cap_points = n;
    return CR_OK;
}

cr_status ensure_segs(PackScratch &s, uint64_t n) {
    if (s.segs && s.cap_segs >= n) return CR_OK;
    uint64_t have[3] = {0, 0, 0};  // grow() keeps a capacity per array; these three go together
    s.cap_segs = 0;
    cr_status st;
    if ((st = grow(&s.segs, have[0], n)) || (st = grow(&s.rsegs, have[1], n)) ||
        (st = grow(&s.bounds, have[2], 8 * n)))
        return st;
    s.cap_segs = n;
    return CR_OK;
}

// Elements of a segment in the scratch arrays: whole 16-byte words of bytes.
uint64_t padded(uint64_t n) { return (n + 15) & ~15ull; }

// Launches kern<true> with the one segment in the parameters, or kern<false>
// with the list.
#define PACK_LAUNCH(nseg, grid, threads, stream, kern1, kernN, ...)      \
    do {                                                                 \
        if ((nseg) == 1u)                                                \
            kern1<<<(grid), (threads), 0, (stream)>>>(__VA_ARGS__);      \
        else                                                             \
            kernN<<<(grid), (threads), 0, (stream)>>>(__VA_ARGS__);      \
        CR_CUDA(cudaGetLastError());                                     \
    } while (0)

// The LOD grids of a segment from its bounds: level `level` has its own
// dense grid.  Returns the cells of all levels in *cells.
cr_status lod_args(PackSeg &sg, const float bmin[3], const float ext[3], int levels, int divs,
                   uint64_t *cells_out) {
    uint64_t total = 0;
    const float longest = std::fmax(ext[0], std::fmax(ext[1], ext[2]));
    const float base_voxel = longest / (float)divs;
    for (int level = 0; level + 1 < levels; ++level) {
        LodArgs &a = sg.lod[level];
        const float voxel = base_voxel * std::pow(0.5f, (float)level);
        a.inv = 1.0f / std::fmax(voxel, 0.000001f);
        uint64_t cells = 1;
        for (int k = 0; k < 3; ++k) {
            a.bmin[k] = bmin[k];
            const float d = std::floor(ext[k] * a.inv);
            if (!(d < 2097151.0f))
                return cri::fail(CR_ERR_CAPACITY, "LOD grid exceeds 2^21 cells per axis");
            a.dims[k] = (uint32_t)d + 1u;
            cells *= a.dims[k];
        }
        if (cells > kLodCellCap)
            return cri::fail(CR_ERR_CAPACITY,
                             "LOD grid of " + std::to_string(cells) + " cells exceeds the cap");
        total += cells;
    }
    *cells_out = total;
    return CR_OK;
}

// Device memory that a wave of several jobs may take anew for each kind of its
// scratch: an eighth of what is free, so that chunks beside a nearly full pool
// are packed one at a time, as in no more memory than the largest of them needs.
cr_status wave_share(uint64_t *bytes) {
    size_t free_b = 0, total_b = 0;
    CR_CUDA(cudaMemGetInfo(&free_b, &total_b));
    *bytes = free_b / 8;
    return CR_OK;
}

// Bytes of a job's host input, staged on the device.
uint64_t staged_bytes(const PackJob &job, int on_device) {
    return on_device ? 0
                     : job.count * ((uint64_t)job.in->positionStrideBytes +
                                    job.in->colorStrideBytes);
}

// Packs jobs [0, njobs) in one run; *done = the jobs packed, fewer than
// njobs when the grids of all would be too large together (at least one), or
// when a job's grid is refused (an error, after packing the jobs before it).
cr_status pack_wave(cr_context *ctx, cr_cloud *cloud, const PackJob *jobs, uint32_t njobs,
                    const cr_pack_params *prm, int on_device, uint32_t *src_idx_host,
                    uint32_t *done) {
    cudaStream_t s = ctx->stream;
    PackScratch &sc = *ctx->pack;
    const bool wide = prm->mortonBits == 21;
    const uint32_t ppb = cloud->cap.pointsPerBatch;
    uint64_t points = 0;
    uint32_t largest = 0;
    for (uint32_t j = 0; j < njobs; ++j) {
        points += padded(jobs[j].count);
        largest = std::max(largest, (uint32_t)jobs[j].count);
    }
    cr_status st = ensure_points(sc, points);
    if (st) return st;
    if ((st = ensure_segs(sc, njobs))) return st;
    std::vector<PackSeg> segs(njobs);
    std::vector<RadixSeg> rsegs(njobs);

    // Stage 0: stage host input (one copy when the colour sits inside the
    // position record).
    std::vector<uint64_t> raw_off(njobs, 0);
    uint64_t raw_bytes = 0;
    auto layout = [](const cr_pack_input *in, uint64_t count, uint64_t &pbytes, uint64_t &cbytes,
                     bool &inside) -> uint64_t {
        const uint64_t csize = in->colorFormat == CR_COLOR_RGBA8 ? 4 : 16;
        const uint8_t *hp = static_cast<const uint8_t *>(in->positions);
        const uint8_t *hc = static_cast<const uint8_t *>(in->colors);
        pbytes = (count - 1) * in->positionStrideBytes + 12;
        cbytes = (count - 1) * in->colorStrideBytes + csize;
        inside = hc >= hp && in->colorStrideBytes == in->positionStrideBytes &&
                 (uint64_t)(hc - hp) + csize <= in->positionStrideBytes;
        return inside ? std::max(pbytes, (uint64_t)(hc - hp) + cbytes)
                      : ((pbytes + 255) & ~255ull) + cbytes;
    };
    if (!on_device) {
        for (uint32_t j = 0; j < njobs; ++j) {
            uint64_t pb, cb;
            bool inside;
            raw_off[j] = raw_bytes;
            raw_bytes += (layout(jobs[j].in, jobs[j].count, pb, cb, inside) + 255) & ~255ull;
        }
        if ((st = grow(reinterpret_cast<uint8_t **>(&sc.raw), sc.cap_raw_bytes, raw_bytes)))
            return st;
    }
    uint64_t begin = 0, blocks = 0, tiles = 0, batches = 0;
    for (uint32_t j = 0; j < njobs; ++j) {
        const cr_pack_input *in = jobs[j].in;
        const uint64_t count = jobs[j].count;
        PackSeg &sg = segs[j];
        sg = PackSeg{};
        sg.begin = begin;
        sg.n = (uint32_t)count;
        sg.block0 = (uint32_t)blocks;
        sg.batch0 = (uint32_t)batches;
        sg.first_slot = jobs[j].first_slot;
        rsegs[j] = RadixSeg{begin, (uint32_t)count, (uint32_t)tiles};
        LoadArgs &la = sg.la;
        la.pos_stride = in->positionStrideBytes;
        la.col_stride = in->colorStrideBytes;
        la.col_format = in->colorFormat;
        if (on_device) {
            la.pos = static_cast<const uint8_t *>(in->positions);
            la.col = static_cast<const uint8_t *>(in->colors);
        } else {
            const uint8_t *hp = static_cast<const uint8_t *>(in->positions);
            const uint8_t *hc = static_cast<const uint8_t *>(in->colors);
            uint64_t pbytes, cbytes;
            bool inside;
            const uint64_t need = layout(in, count, pbytes, cbytes, inside);
            uint8_t *raw = static_cast<uint8_t *>(sc.raw) + raw_off[j];
            la.pos = raw;
            if (inside) {
                CR_CUDA(cudaMemcpyAsync(raw, hp, need, cudaMemcpyHostToDevice, s));
                la.col = raw + (hc - hp);
            } else {
                const uint64_t coff = (pbytes + 255) & ~255ull;
                CR_CUDA(cudaMemcpyAsync(raw, hp, pbytes, cudaMemcpyHostToDevice, s));
                CR_CUDA(cudaMemcpyAsync(raw + coff, hc, cbytes, cudaMemcpyHostToDevice, s));
                la.col = raw + coff;
            }
        }
        // Device-resident 16-byte records {x, y, z, rgba8} already have the
        // layout of the staged positions: read them in place.
        const bool in_place = on_device && in->positionStrideBytes == 16 &&
                              in->colorStrideBytes == 16 && in->colorFormat == CR_COLOR_RGBA8 &&
                              static_cast<const uint8_t *>(in->colors) ==
                                  static_cast<const uint8_t *>(in->positions) + 12 &&
                              ((uintptr_t)in->positions & 15) == 0;
        sg.stage = in_place ? nullptr : sc.pos + begin;
        sg.pos = in_place ? static_cast<const float4 *>(in->positions) : sc.pos + begin;
        begin += padded(count);
        blocks += (count + kPointsPerCta - 1) / kPointsPerCta;
        tiles += radix_tiles((uint32_t)count);
        batches += (count + ppb - 1) / ppb;
    }
    Segs arg;
    arg.list = sc.segs;
    auto upload = [&](uint32_t n) -> cr_status {
        arg.n = n;
        arg.one = segs[0];
        if (n > 1)  // one segment travels in the kernels' parameters
            CR_CUDA(cudaMemcpyAsync(sc.segs, segs.data(), n * sizeof(PackSeg),
                                    cudaMemcpyHostToDevice, s));
        return CR_OK;
    };
    if ((st = upload(njobs))) return st;
    CR_CUDA(cudaMemcpyAsync(sc.rsegs, rsegs.data(), njobs * sizeof(RadixSeg),
                            cudaMemcpyHostToDevice, s));

    // Stage 1: bounds, read back once.
    CR_CUDA(cudaMemsetAsync(sc.bounds, 0xff, (size_t)njobs * 8 * 4, s));
    const unsigned sms = (unsigned)std::max(ctx->sm_count, 1);
    auto rows = [&](uint32_t n) {  // CTAs of a segment in the two-dimensional launches
        return std::max(1u, std::min(grid_for(largest), std::max(sms * 8u / n, 32u)));
    };
    PACK_LAUNCH(njobs, dim3(rows(njobs), njobs), kThreads, s, pack_load_bounds<true>,
                pack_load_bounds<false>, arg, sc.bounds);
    std::vector<uint32_t> bflip((size_t)njobs * 8);
    CR_CUDA(cudaMemcpyAsync(bflip.data(), sc.bounds, bflip.size() * 4, cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaStreamSynchronize(s));
    const int L = std::max(1, std::min(prm->lodLevels, kMaxLevels));
    const int divs = std::max(1, prm->coarseVoxelDivisions);
    const uint32_t max_level = (uint32_t)(L - 1);
    std::vector<uint64_t> cells(njobs, 0);
    uint64_t cell_sum = 0, cell_limit = 0;
    uint32_t nseg = 0;
    cr_status refused = CR_OK;
    for (uint32_t j = 0; j < njobs; ++j) {
        PackSeg &sg = segs[j];
        float bmin[3], bmax[3], ext[3];
        for (int k = 0; k < 3; ++k) {
            bmin[k] = unflip(bflip[8 * j + k]);
            bmax[k] = unflip(~bflip[8 * j + 3 + k]);
            ext[k] = std::fmax(bmax[k] - bmin[k], 0.000001f);
        }
        sg.m.top = wide ? 2097151.0f : 1023.0f;
        for (int k = 0; k < 3; ++k) {
            sg.m.bmin[k] = bmin[k];
            sg.m.scale[k] = sg.m.top / ext[k];
        }
        if ((refused = lod_args(sg, bmin, ext, L, divs, &cells[j]))) break;
        // Grids of several jobs together: in the memory that there is, or in new
        // memory up to the wave's share (asked for only where it can decide: 200
        // nodes in several waves 2350 us a call with a query in each, 2140 without).
        if (j > 0 && cell_sum + cells[j] > std::max(sc.cap_grid, kLodCellCap)) break;
        if (j > 0 && cell_sum + cells[j] > sc.cap_grid) {
            if (cell_limit == 0) {
                uint64_t bytes = 0;
                if ((st = wave_share(&bytes))) return st;
                cell_limit = std::max(sc.cap_grid, bytes / 4);
            }
            if (cell_sum + cells[j] > cell_limit) break;
        }
        cell_sum += cells[j];
        nseg = j + 1;
    }
    *done = nseg;
    if (nseg == 0) return refused;
    if (nseg < njobs) {
        blocks = segs[nseg].block0;
        batches = segs[nseg].batch0;
        tiles = rsegs[nseg].tile0;
    }
    if (!sc.grid || sc.cap_grid < cell_sum) sc.grid_empty = false;
    if ((st = grow(&sc.grid, sc.cap_grid, cell_sum))) return st;
    uint64_t goff = 0;
    for (uint32_t j = 0; j < nseg; ++j)
        for (int level = 0; level + 1 < L; ++level) {
            LodArgs &a = segs[j].lod[level];
            a.grid = sc.grid + goff;
            goff += (uint64_t)a.dims[0] * a.dims[1] * a.dims[2];
        }
    if ((st = upload(nseg))) return st;

    // Stages 2-3: Morton keys and their digits' histograms, stable sort.
    if ((st = radix_begin(sc.radix, nseg, tiles, s))) return st;
    if (wide) {
        using K = unsigned long long;
        const RadixBuffers<K> buf{{static_cast<K *>(sc.keys[0]), static_cast<K *>(sc.keys[1])},
                                  {sc.idx[0], sc.idx[1]}};
        PACK_LAUNCH(nseg, dim3(rows(nseg), nseg), kThreads, s, (pack_morton<K, true>),
                    (pack_morton<K, false>), arg, buf.keys[0], sc.radix.hist);
        st = radix_sort<K>(buf, sc.rsegs, nseg, tiles, segs[0].n, 63, true, sc.radix,
                           ctx->sort_wait_limit, ctx->d_status, s);
    } else {
        using K = uint32_t;
        const RadixBuffers<K> buf{{static_cast<K *>(sc.keys[0]), static_cast<K *>(sc.keys[1])},
                                  {sc.idx[0], sc.idx[1]}};
        PACK_LAUNCH(nseg, dim3(rows(nseg), nseg), kThreads, s, (pack_morton<K, true>),
                    (pack_morton<K, false>), arg, buf.keys[0], sc.radix.hist);
        st = radix_sort<K>(buf, sc.rsegs, nseg, tiles, segs[0].n, 30, false, sc.radix,
                           ctx->sort_wait_limit, ctx->d_status, s);
    }
    if (st) return st;

    // Stages 4-5: gather, LOD levels (each level its own dense grid).
    const Sorted so{{sc.idx[0], sc.idx[1]},
                    {static_cast<const unsigned long long *>(sc.keys[0]),
                     static_cast<const unsigned long long *>(sc.keys[1])},
                    sc.radix.runs,
                    sc.radix.ties,
                    src_idx_host ? 1 : 0};
    // The grids are empty but for a run that did not come to its end.
    if (!sc.grid_empty && cell_sum) CR_CUDA(cudaMemsetAsync(sc.grid, 0xff, sc.cap_grid * 4, s));
    const bool empty_after = sc.grid_empty || cell_sum > 0;
    sc.grid_empty = false;
    PACK_LAUNCH(nseg, (unsigned)blocks, kThreads, s, pack_gather_claim<true>,
                pack_gather_claim<false>, arg, so, sc.sorted, sc.lv_morton, max_level);
    for (uint32_t level = 0; level + 1 < max_level; ++level)
        PACK_LAUNCH(nseg, (unsigned)blocks, kThreads, s, pack_lod_assign<true>,
                    pack_lod_assign<false>, arg, sc.sorted, sc.lv_morton, level, max_level);

    // Stages 6-7: batches, final order, quantisation into the pool; source
    // indices only when asked for.
    uint32_t *src = src_idx_host ? sc.src_idx : nullptr;
    if (L <= 4)
        PACK_LAUNCH(nseg, (unsigned)batches, batch_threads(ppb), s, (pack_batches<4, true>),
                    (pack_batches<4, false>), arg, sc.sorted, sc.lv_morton, max_level, ppb, so,
                    cloud->d_batches, cloud->d_low, cloud->d_med,
                    cloud->d_high, cloud->d_colors, cloud->d_levels, src);
    else
        PACK_LAUNCH(nseg, (unsigned)batches, batch_threads(ppb), s, (pack_batches<8, true>),
                    (pack_batches<8, false>), arg, sc.sorted, sc.lv_morton, max_level, ppb, so,
                    cloud->d_batches, cloud->d_low, cloud->d_med,
                    cloud->d_high, cloud->d_colors, cloud->d_levels, src);
    sc.grid_empty = empty_after;
    if (src)
        CR_CUDA(cudaMemcpyAsync(src_idx_host, src, jobs[0].count * 4, cudaMemcpyDeviceToHost, s));
    return refused;
}

}  // namespace

void pack_scratch_free(PackScratch &s) {
    void *ptrs[] = {s.raw, s.pos, s.keys[0], s.keys[1], s.idx[0], s.idx[1], s.sorted,
                    s.lv_morton, s.grid, s.segs, s.rsegs, s.bounds, s.src_idx};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    radix_scratch_free(s.radix);
    s = PackScratch{};
}

// Packs every job into its slots of the cloud's pool.  Enqueues on the
// context stream; one synchronisation per wave reads the segments' bounds
// back to size the Morton scales and the LOD grids.  src_idx_host (one job
// only): the input index of every packed point.  A wave takes jobs while
// they hold at most kWavePoints points and kWaveStaged bytes of host input
// together, so that a long list of chunks needs no more scratch than one chunk
// of that size, and takes fewer where their scratch would be more than its share
// of the free memory, or is refused.
cr_status pack_run(cr_context *ctx, cr_cloud *cloud, const std::vector<PackJob> &jobs,
                   const cr_pack_params *prm, int on_device, uint32_t *src_idx_host) {
    constexpr uint64_t kWavePoints = 1ull << 24;
    constexpr size_t kWaveJobs = 4096;  // the launches' second grid dimension is bounded
    constexpr uint64_t kWaveStaged = 1ull << 29;
    if (src_idx_host && jobs.size() != 1)
        return cri::fail(CR_ERR_INTERNAL, "pack_run: source indices of one job only");
    size_t first = 0;
    while (first < jobs.size()) {
        size_t last = first + 1;
        uint64_t points = padded(jobs[first].count), staged = staged_bytes(jobs[first], on_device);
        uint64_t share = 0;
        for (; last < jobs.size() && last - first < kWaveJobs; ++last) {
            const uint64_t p = points + padded(jobs[last].count);
            const uint64_t b = staged + staged_bytes(jobs[last], on_device);
            if (p > kWavePoints || b > kWaveStaged) break;
            if (p > ctx->pack->cap_points || b > ctx->pack->cap_raw_bytes) {
                if (share == 0)
                    if (const cr_status st = wave_share(&share)) return st;
                if (p * kPointScratch > share || b > share) break;
            }
            points = p;
            staged = b;
        }
        uint32_t done = 0;
        cr_status st;
        for (;;) {
            st = pack_wave(ctx, cloud, jobs.data() + first, (uint32_t)(last - first), prm, on_device,
                           src_idx_host, &done);
            if (st != CR_ERR_OUT_OF_MEMORY || last - first == 1) break;
            last = first + (last - first) / 2;
        }
        if (st) return st;
        first += done;
    }
    return CR_OK;
}
