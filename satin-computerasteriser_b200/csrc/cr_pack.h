// cr_pack.h — internal interface of the GPU packer.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "cr/cr.h"

// One segment of a sort: keys [begin, begin + n) of the arrays, sorted by
// itself; tile0 is its first tile in the numbering of all segments' tiles.
struct RadixSeg {
    uint64_t begin;
    uint32_t n, tile0;
};
constexpr int kRadixMaxPasses = 8;  // 8-bit digits of a 64-bit key

// The sort's ping-pong buffers: the keys start in keys[0].  A segment whose
// set of passes (RadixScratch::runs) has k members ends in buffer k & 1; with
// k = 0 no values were written, and key i's value is i.
template <typename K>
struct RadixBuffers {
    K *keys[2];
    uint32_t *vals[2];
};

// Grow-only scratch of the radix sort: look-back words (256 per 4096-key
// tile), per segment the histograms and digit bases of up to 8 passes and
// the set of passes to run, one tile ticket counter per pass, and the epoch
// of the last pass (look-back words carry it).
struct RadixScratch {
    unsigned long long *lookback = nullptr;
    uint64_t cap_tiles = 0;
    uint32_t cap_segs = 0;
    uint32_t *hist = nullptr;   // [segment][kRadixMaxPasses][256], filled by the caller
    uint32_t *bases = nullptr;  // the same shape
    uint32_t *runs = nullptr;   // per segment: bit p set = pass p runs
    uint32_t *ties = nullptr;   // per segment: low key bits that no pass sorted
    unsigned long long *sample = nullptr;  // radix_sample's tables and counts
    uint32_t *tiles = nullptr;
    uint32_t epoch = 0;
};
void radix_scratch_free(RadixScratch &r);
// Tiles of n keys.
uint32_t radix_tiles(uint32_t n);
// Makes room for nseg segments of ntiles tiles in all and zeroes the
// histograms; the caller then fills them and calls radix_sort.
cr_status radix_begin(RadixScratch &rs, uint32_t nseg, uint64_t ntiles, cudaStream_t s);
// Stable sort of every segment's keys by their low key_bits bits (the bits
// above them are zero), with the keys' places in the segment as values.
// segs is device memory; n0: the keys of the first.  ties_ok: the passes over
// the lowest digits of a single large segment of 64-bit keys may be left out;
// keys that agree above the segment's tie bits (RadixScratch::ties) are then in
// input order, and the caller orders them.  A tile's wait for those before it
// that gives up after wait_limit polls (0: every tile after a segment's first
// gives up at once) stores kErrSortWait into *status; the segment's keys and
// values may then be anything, and its tie bits are 0.
constexpr uint32_t kSampleMinKeys = 1u << 19;
template <typename K>
cr_status radix_sort(const RadixBuffers<K> &buf, const RadixSeg *segs, uint32_t nseg,
                     uint64_t ntiles, uint32_t n0, int key_bits, bool ties_ok, RadixScratch &rs,
                     uint32_t wait_limit, uint32_t *status, cudaStream_t s);

struct PackSeg;

// Grow-only device scratch of the packer, owned by the context (the
// reference's PackScratch, GPUPacker.swift:453-484).
struct PackScratch {
    uint64_t cap_points = 0;
    uint64_t cap_raw_bytes = 0;
    uint64_t cap_grid = 0;
    uint64_t cap_segs = 0;
    void *raw = nullptr;                    // staged host input
    float4 *pos = nullptr;                  // input x, y, z and RGBA8 bits in w
    void *keys[2] = {nullptr, nullptr};     // Morton keys (u32 or u64), ping-pong
    uint32_t *idx[2] = {nullptr, nullptr};  // sort payload, ping-pong
    float4 *sorted = nullptr;               // positions in Morton order
    uint8_t *lv_morton = nullptr;           // levels in Morton order
    uint32_t *grid = nullptr;               // dense LOD occupancy grids
    bool grid_empty = false;                // every voxel of all cap_grid is empty
    PackSeg *segs = nullptr;                // the segments of a run
    RadixSeg *rsegs = nullptr;              //   and what the sort needs of them
    RadixScratch radix;                     // the sort's look-back words and histograms
    uint32_t *bounds = nullptr;             // per segment: 3 flipped minima, 3 complements of
                                            // flipped maxima
    uint32_t *src_idx = nullptr;            // final order -> input index
};

void pack_scratch_free(PackScratch &s);
