// radix.cu — stable LSD radix sort of (key, index) pairs for the packer.
//
// The reference packer (Pipelines/GPUPacker/Shaders.metal:134-215) sorts
// 30-bit Morton keys with four 8-bit passes, one *thread* per 1024-key tile
// walking the tile serially so histogram and scatter agree on order.  Here
// one kernel per 8-bit digit reads each key and value once and writes them
// once (a single-sweep pass with decoupled look-back).  The arrays hold one
// or more segments (the clouds of one call), each sorted by itself:
//   (caller)          the 256-bin histograms of every digit of every segment,
//                     beside the keys it makes (RadixScratch::hist);
//   radix_bases       per segment: exclusive scans into digit bases, and the
//                     set of digits that its keys do not all share (a pass
//                     over the others would move nothing and is skipped);
//   radix_onesweep    per pass, 4096-key tiles taken in ticket order: a tile
//                     ranks its keys among equal digits in input order (warp
//                     multisplit with ballots, then scans over warps and
//                     digits), publishes its per-digit counts, sums the
//                     counts of its segment's tiles before it per digit
//                     (look-back over their published counts and inclusive
//                     prefixes, a thread per digit), sorts the tile by digit
//                     in shared memory and writes one coalesced run per
//                     digit.  Equal keys keep their input order (stable), as
//                     the CPU's stable sort does.
// Low digits of a large sort (radix_sample).  The keys of a large cloud differ
// mostly in their high digits, so the passes over the lowest digits only order
// the few keys that agree in all others.  A sample of the keys estimates how
// many agree, and when they are few those passes are left out: the segment's
// tie word then says how many low bits were not sorted, and the reader of the
// sorted keys orders each run of keys that agree above them (its cost grows
// with the square of a run's length: the sample bounds their mean and the
// longest).
// Nothing is read back: which of the two buffers a segment's pass reads
// follows from the segment's set of digits (bit p: pass p runs), and so does
// where its sorted keys and indices end up.
// A tile waits only for tiles with smaller tickets, which started before it,
// so the waits end whatever the GPU schedules; each wait is nevertheless
// bounded (wait_limit polls), after which the tile counts the missing
// predecessor as empty and stores kErrSortWait into the status word, which
// the host reports as CR_ERR_TIMEOUT.  The order is then no permutation: places
// of the buffers keep what was there before.  The values' readers bound them,
// and the segment has no ties any more: nobody walks along runs of such keys.
#include <algorithm>
#include <cstring>
#include <vector>

#include "cr_internal.h"
#include "cr_pack.h"

namespace {

constexpr int kThreads = 256;  // one thread per digit in the per-digit phases
constexpr int kWarps = kThreads / 32;
constexpr int kKeysPerLane = 16;
constexpr int kTileKeys = kThreads * kKeysPerLane;  // 4096

// Look-back word of one (tile, digit): epoch (16 bits) | flag (2 bits) |
// count (46 bits).  Flag 1: the tile's own count; flag 2: the inclusive count
// over the tiles up to and including it.
constexpr unsigned long long kFlagAgg = 1ull, kFlagPrefix = 2ull;
__device__ __forceinline__ unsigned long long lookback_word(uint32_t epoch, unsigned long long flag,
                                                            unsigned long long count) {
    return ((unsigned long long)epoch << 48) | (flag << 46) | count;
}
// The look-back words carry their data (the counts) in the word itself, so
// relaxed loads and stores at GPU scope suffice (no other memory is read
// through them).
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ bool lookback_ready(unsigned long long v, uint32_t epoch) {
    return (uint32_t)(v >> 48) == epoch && ((v >> 46) & 3ull) != 0ull;
}
constexpr int kLookbackBatch = 8;  // predecessor words one round loads at once
// Per-warp digit counts and bases (at most kTileKeys) in 16 bits: 55.4 KB of
// shared memory and at most 64 registers let four sort CTAs share an SM.
using WarpCount = uint16_t;
constexpr int kSortBlocksPerSM = 4;

// Inclusive warp scan.
__device__ __forceinline__ uint32_t warp_inclusive(uint32_t x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// How many pairs of kSamples keys, drawn with replacement from all n, agree
// above their low 24 (and 32) bits, and how many samples at most agree with one
// another: a hash table of 39-bit (31-bit) values per choice, each slot a value
// and the samples that had it.  n times the chance that two keys agree is the
// mean length of the run that a key is in; a run of r keys has about
// r * kSamples / n samples.
// found: the pairs of each choice, then the largest counts before a sample.
constexpr uint32_t kSamples = 1u << 16;
constexpr int kSampleSlotBits = 18;
constexpr int kSampleChoices = 2;
__global__ void __launch_bounds__(kThreads)
    radix_sample(const unsigned long long *__restrict__ keys, uint32_t n,
                 unsigned long long *__restrict__ table, unsigned long long *__restrict__ found) {
    constexpr uint32_t kMask = (1u << kSampleSlotBits) - 1u;
    const uint32_t s = blockIdx.x * kThreads + threadIdx.x;
    // A spread of the sample's number: Weyl's sequence by the golden ratio, and
    // the first steps of MurmurHash3's 32-bit finaliser.
    uint32_t h = s * 0x9e3779b9u + 0x7f4a7c15u;
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    const unsigned long long key = keys[((unsigned long long)h * n) >> 32];
#pragma unroll
    for (int v = 0; v < kSampleChoices; ++v) {
        const unsigned long long top = key >> (24 + 8 * v);  // 39 bits at most
        unsigned long long *t = table + ((size_t)v << kSampleSlotBits);
        uint32_t slot = (uint32_t)((top * 0x9e3779b97f4a7c15ull) >> 40);
        uint32_t agree = 0;
        // Lanes with the same value go together, the lowest of them to the table (of
        // points in one place every sample meets in one word: 134 us one by one).
        const uint32_t peers = __match_any_sync(0xffffffffu, top), lead = __ffs(peers) - 1u;
        const uint32_t lane = threadIdx.x & 31, many = __popc(peers);
        if (lane == lead)
            for (int probe = 0; probe < 64; ++probe, ++slot) {
                unsigned long long *w = t + (slot & kMask);
                const unsigned long long old = atomicCAS(w, 0ull, (top << 20) | many);
                if (old == 0ull) break;
                if (old >> 20 != top) continue;
                agree = (uint32_t)(atomicAdd(w, (unsigned long long)many) & 0xfffffull);
                break;
            }
        agree = __shfl_sync(0xffffffffu, agree, lead) + __popc(peers & ((1u << lane) - 1u));
        const uint32_t sum = __reduce_add_sync(0xffffffffu, agree);
        const uint32_t most = __reduce_max_sync(0xffffffffu, agree);
        if ((threadIdx.x & 31) == 0 && sum) {
            atomicAdd(found + v, (unsigned long long)sum);
            atomicMax(found + kSampleChoices + v, (unsigned long long)most);
        }
    }
}

// Low passes to leave out given the sample: those whose bits separate runs of
// at most kMaxMeanRun keys in the mean and, by the samples of one run, of about
// kMaxRun keys (or kMaxRunSamples samples, where one stands for more keys).  By
// the mean alone, 100M points with 24 thousand in one cell were packed in 17.9 ms,
// 10.9 with every digit sorted.
constexpr unsigned long long kMaxMeanRun = 6, kMaxRun = 1024, kMaxRunSamples = 4;
__device__ __forceinline__ uint32_t passes_left_out(const unsigned long long *found, uint32_t n) {
    const unsigned long long longest = max(kMaxRunSamples, kMaxRun * kSamples / n);
    for (int v = kSampleChoices - 1; v >= 0; --v)
        if (2ull * found[v] * n <= kMaxMeanRun * ((unsigned long long)kSamples * kSamples) &&
            found[kSampleChoices + v] < longest)
            return 3u + (uint32_t)v;
    return 0u;
}

// A segment's digit bases, the set of its passes and its tie word: one CTA per
// segment, a thread per digit.  sampled: radix_sample's (null: none was taken).
__global__ void __launch_bounds__(kThreads)
    radix_bases(const uint32_t *__restrict__ hist, const RadixSeg *__restrict__ segs, int passes,
                const unsigned long long *__restrict__ sampled, uint32_t *__restrict__ bases,
                uint32_t *__restrict__ runs, uint32_t *__restrict__ ties) {
    __shared__ uint32_t sums[kRadixMaxPasses][kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t n = segs[blockIdx.x].n;
    const size_t row = (size_t)blockIdx.x * kRadixMaxPasses * 256;
    uint32_t set = 0, incl[kRadixMaxPasses], mine[kRadixMaxPasses];
#pragma unroll
    for (int p = 0; p < kRadixMaxPasses; ++p)
        mine[p] = p < passes ? hist[row + p * 256 + threadIdx.x] : 0u;
#pragma unroll
    for (int p = 0; p < kRadixMaxPasses; ++p) {
        incl[p] = warp_inclusive(mine[p], lane);
        if (lane == 31) sums[p][warp] = incl[p];
        // Every key has this digit: the pass is a copy.
        const bool constant = __syncthreads_or(mine[p] == n);
        if (p < passes && !constant) set |= 1u << p;
    }
#pragma unroll
    for (int p = 0; p < kRadixMaxPasses; ++p) {
        uint32_t base = incl[p] - mine[p];
#pragma unroll
        for (int w = 0; w < kWarps; ++w)
            if (w < warp) base += sums[p][w];
        if (p < passes) bases[row + p * 256 + threadIdx.x] = base;
    }
    if (threadIdx.x == 0) {
        const uint32_t out = sampled ? passes_left_out(sampled, n) : 0u;
        runs[blockIdx.x] = set & ~((1u << out) - 1u);
        ties[blockIdx.x] = 8u * out;
    }
}

template <typename K>
size_t onesweep_smem_bytes() {
    return (size_t)kTileKeys * (sizeof(K) + sizeof(uint32_t)) +
           (size_t)kWarps * 256 * sizeof(WarpCount) + (256 + 32) * sizeof(uint32_t);
}

// Digit of a key: a byte of the 32-bit word that holds it (a digit never
// straddles the words: the shifts are multiples of 8).
struct DigitOf {
    uint32_t word;  // word of the key (0 low, 1 high)
    uint32_t sel;   // byte selector: that byte, then three zero bytes
    __device__ __forceinline__ explicit DigitOf(int shift)
        : word((uint32_t)shift >> 5), sel(0x4440u | (((uint32_t)shift >> 3) & 3u)) {}
    __device__ __forceinline__ uint32_t of_word(uint32_t w) const {
        return __byte_perm(w, 0u, sel);
    }
    // Digit of key i of an array in global memory that the kernel only reads
    // (__ldg, here and where the keys move: a plain load cannot pass the
    // barriers and shared-memory stores between two keys; a pass over 100M
    // keys took 975 us instead of 750 us with them).
    __device__ __forceinline__ uint32_t at(const uint32_t *keys, uint32_t i) const {
        return of_word(__ldg(keys + i));
    }
    __device__ __forceinline__ uint32_t at(const unsigned long long *keys, uint32_t i) const {
        return of_word(__ldg(reinterpret_cast<const uint32_t *>(keys) + (2u * i + word)));
    }
    __device__ __forceinline__ uint32_t of(uint32_t k) const { return of_word(k); }
    __device__ __forceinline__ uint32_t of(unsigned long long k) const {
        return of_word(word ? (uint32_t)(k >> 32) : (uint32_t)k);
    }
};

// Ranks a warp's keys (512, in warp-striped order: key 32 j + lane) among
// equal digits, in input order, against the warp's running digit counts wc.
// rd[j] = rank | digit << 16.  FULL: the tile has all of its keys.
template <typename K, bool FULL>
__device__ __forceinline__ void rank_keys(const K *keys, uint32_t w0, uint32_t tile_n,
                                          const DigitOf &dig, WarpCount *wc, uint32_t lt,
                                          uint32_t (&rd)[kKeysPerLane]) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < kKeysPerLane; ++j) {
        const uint32_t li = w0 + (uint32_t)j * 32u + lane;
        const bool v = FULL || li < tile_n;
        const uint32_t d = v ? dig.at(keys, li) : 0u;
        // Lanes with the same digit: the lanes that agree with this lane's
        // bit, for every bit (eight ballots cost less than
        // __match_any_sync when a warp holds many distinct digits).  A lane
        // differs from this one where its bit of some ballot does.
        uint32_t differ = FULL ? 0u : ~__ballot_sync(0xffffffffu, v);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const bool bit = (d >> b) & 1u;
            const uint32_t m = __ballot_sync(0xffffffffu, bit);
            differ |= m ^ (bit ? 0xffffffffu : 0u);
        }
        const uint32_t lower = ~differ & lt;
        const uint32_t before = wc[d];
        rd[j] = (before + __popc(lower)) | (d << 16);
        __syncwarp();
        if (v && lower == 0u) wc[d] = (WarpCount)(before + __popc(~differ));
        __syncwarp();
    }
}

// Moves a warp's keys and values to their places in the tile sorted by digit.
// vals null: the values are the keys' places in their segment (tile0: the
// tile's).
template <typename K, bool FULL>
__device__ __forceinline__ void move_keys(const K *keys, const uint32_t *vals, uint32_t tile0,
                                          uint32_t w0, uint32_t tile_n, const WarpCount *wc,
                                          const uint32_t (&rd)[kKeysPerLane], K *skey,
                                          uint32_t *sval) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < kKeysPerLane; ++j) {
        const uint32_t li = w0 + (uint32_t)j * 32u + lane;
        if (FULL || li < tile_n) {
            const uint32_t slot = wc[rd[j] >> 16] + (rd[j] & 0xffffu);
            skey[slot] = __ldg(keys + li);
            sval[slot] = vals ? __ldg(vals + li) : tile0 + li;
        }
    }
}

// Writes the sorted tile to global memory: gbase[d] + (slot in the tile).
template <typename K, bool FULL>
__device__ __forceinline__ void write_keys(const K *skey, const uint32_t *sval,
                                           const uint32_t *gbase, const DigitOf &dig,
                                           uint32_t tile_n, uint32_t n, K *keys_out,
                                           uint32_t *vals_out) {
#pragma unroll 8
    for (uint32_t i = threadIdx.x; i < (FULL ? (uint32_t)kTileKeys : tile_n); i += kThreads) {
        const K k = skey[i];
        const uint32_t dst = gbase[dig.of(k)] + i;
        if (dst < n) {  // always true when the counts are consistent
            keys_out[dst] = k;
            vals_out[dst] = sval[i];
        }
    }
}

// One pass: a tile of kTileKeys keys per CTA, in ticket order.
//   1. each warp takes 512 consecutive keys, 16 per lane in warp-striped order
//      (key j*32 + lane), and ranks them among equal digits (peer lanes found
//      by ballots) against running per-warp digit counts, in input order;
//   2. thread d: the tile's count of digit d (published at once); an
//      exclusive scan over the digits, and with it the first slot of every
//      (warp, digit) in a tile sorted by digit;
//   3. keys and values move there in shared memory; then thread d sums the
//      counts of the tiles before it (look-back) and publishes the inclusive
//      prefix;
//   4. threads read the sorted tile in order and write each key to its
//      digit's global offset: keys of one digit are consecutive in shared
//      memory and land at consecutive addresses (coalesced runs).
// Bound by the integer pipe (ballots, selects and address arithmetic; it was
// 83 % busy), so the full tiles have code without bounds (every tile but the
// last), a digit is one byte permute of the word that holds it, offsets are
// 32 bits and one shared word gives a key's place.
// The first pass that a segment runs makes the values (the keys' places in
// the segment); the pass before it wrote none.
template <typename K>
__global__ void __launch_bounds__(kThreads, kSortBlocksPerSM)
    radix_onesweep(RadixBuffers<K> buf, const RadixSeg *__restrict__ segs, uint32_t nseg, int pass,
                   const uint32_t *__restrict__ bases, const uint32_t *__restrict__ runs,
                   unsigned long long *__restrict__ lookback, uint32_t epoch,
                   uint32_t *__restrict__ tile_counter, uint32_t wait_limit,
                   uint32_t *__restrict__ ties, uint32_t *status) {
    extern __shared__ __align__(16) unsigned char smem[];
    K *skey = reinterpret_cast<K *>(smem);
    uint32_t *sval = reinterpret_cast<uint32_t *>(skey + kTileKeys);
    // [kWarps][256]: per-warp digit counts, then the warps' first slots.
    WarpCount *wcnt = reinterpret_cast<WarpCount *>(sval + kTileKeys);
    // Per digit: global place of the tile's run less its first slot in the tile.
    uint32_t *gbase = reinterpret_cast<uint32_t *>(wcnt + kWarps * 256);
    uint32_t *misc = gbase + 256;            // [0] ticket, [1..8] warp sums of the digit scan
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const DigitOf dig(8 * pass);
    if (threadIdx.x == 0) misc[0] = atomicAdd(tile_counter, 1u);
    static_assert(kWarps * 256 * sizeof(WarpCount) == kThreads * sizeof(uint4), "one store each");
    reinterpret_cast<uint4 *>(wcnt)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const uint32_t gtile = misc[0];
    // The segment of the tile, and its tile in the segment.
    uint32_t si = 0;
    for (uint32_t hi = nseg; hi - si > 1u;) {
        const uint32_t mid = (si + hi) >> 1;
        if (segs[mid].tile0 <= gtile)
            si = mid;
        else
            hi = mid;
    }
    const RadixSeg sg = segs[si];
    const uint32_t set = runs[si];
    if (!(set >> pass & 1u)) return;  // every key of the segment has this digit
    const uint32_t done = __popc(set & ((1u << pass) - 1u));  // passes before this one
    const uint32_t n = sg.n, tile = gtile - sg.tile0;
    const uint32_t tile0 = tile * (uint32_t)kTileKeys;  // below n
    const uint32_t tile_n = min(n - tile0, (uint32_t)kTileKeys);
    const bool full = tile_n == (uint32_t)kTileKeys;
    const bool odd = done & 1u;
    const K *keys_in = (odd ? buf.keys[1] : buf.keys[0]) + sg.begin + tile0;
    const uint32_t *vals_in =
        done ? (odd ? buf.vals[1] : buf.vals[0]) + sg.begin + tile0 : nullptr;
    K *keys_out = (odd ? buf.keys[0] : buf.keys[1]) + sg.begin;
    uint32_t *vals_out = (odd ? buf.vals[0] : buf.vals[1]) + sg.begin;
    const uint32_t *digit_base = bases + ((size_t)si * kRadixMaxPasses + pass) * 256;
    const uint32_t w0 = (uint32_t)warp * (32 * kKeysPerLane);
    // 1. Warp-level ranking in input order; a key's rank within its warp
    //    (< 512) and digit are kept packed, the key and value are read again
    //    (from L2) when they move.
    uint32_t rd[kKeysPerLane];
    WarpCount *wc = wcnt + warp * 256;
    if (full)
        rank_keys<K, true>(keys_in, w0, tile_n, dig, wc, lt, rd);
    else
        rank_keys<K, false>(keys_in, w0, tile_n, dig, wc, lt, rd);
    __syncthreads();
    // 2. Digit d = thread: the tile's count and the warps' first slots.
    const uint32_t dd = threadIdx.x;
    uint32_t cw[kWarps], total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        cw[w] = wcnt[w * 256 + dd];
        total += cw[w];
    }
    lookback += (size_t)sg.tile0 * 256;  // the segment's words
    unsigned long long *my = lookback + (size_t)tile * 256 + dd;
    // Publish the tile's count first (tile 0: its prefix), so that the tiles
    // after it can go on while this one sorts its keys.
    st_relaxed64(my, lookback_word(epoch, tile == 0 ? kFlagPrefix : kFlagAgg, total));
    // Exclusive scan of the tile's digit counts (a warp scan per 32 digits,
    // then over the warps).
    const uint32_t incl = warp_inclusive(total, lane);
    if (lane == 31) misc[1 + warp] = incl;
    __syncthreads();
    uint32_t tbase = incl - total;
#pragma unroll
    for (int w = 0; w < kWarps; ++w)
        if (w < warp) tbase += misc[1 + w];
    {
        uint32_t slot = tbase;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            wcnt[w * 256 + dd] = (WarpCount)slot;
            slot += cw[w];
        }
    }
    __syncthreads();
    // 3. The tile sorted by digit.
    if (full)
        move_keys<K, true>(keys_in, vals_in, tile0, w0, tile_n, wc, rd, skey, sval);
    else
        move_keys<K, false>(keys_in, vals_in, tile0, w0, tile_n, wc, rd, skey, sval);
    // The look-back (thread d, digit d) over the tiles before this one, after
    // the tile-local work so that its waits overlap it.
    unsigned long long excl = 0;
    if (tile != 0) {
        // Look-back over the tiles before this one, kLookbackBatch words per
        // round (independent loads), newest first: add counts until a tile's
        // inclusive prefix; a word not yet published is polled (bounded).
        constexpr unsigned long long kCountMask = (1ull << 46) - 1ull;
        bool gave_up = wait_limit == 0u;
        int64_t t = gave_up ? -1 : (int64_t)tile - 1;
        while (t >= 0) {
            const int nb = t + 1 < kLookbackBatch ? (int)(t + 1) : kLookbackBatch;
            unsigned long long v[kLookbackBatch];
#pragma unroll
            for (int k = 0; k < kLookbackBatch; ++k)
                if (k < nb) v[k] = ld_relaxed64(lookback + (size_t)(t - k) * 256 + dd);
            // Add the batch's counts up to the first inclusive prefix (pf)
            // or the first word not yet published (nr).
            int nr = -1;
            bool pf = false;
#pragma unroll
            for (int k = 0; k < kLookbackBatch; ++k) {
                if (k < nb && nr < 0 && !pf) {
                    if (!lookback_ready(v[k], epoch)) {
                        nr = k;
                    } else {
                        excl += v[k] & kCountMask;
                        pf = ((v[k] >> 46) & 3ull) == kFlagPrefix;
                    }
                }
            }
            if (pf) break;
            if (nr < 0) {
                t -= nb;
                continue;
            }
            // Poll the unpublished predecessor, then carry on from the one
            // before it.
            const unsigned long long *w = lookback + (size_t)(t - nr) * 256 + dd;
            uint32_t polls = 0;
            unsigned long long x = ld_relaxed64(w);
            while (!lookback_ready(x, epoch) && ++polls < wait_limit) {
                __nanosleep(32);
                x = ld_relaxed64(w);
            }
            if (!lookback_ready(x, epoch)) {
                gave_up = true;
                break;
            }
            excl += x & kCountMask;
            if (((x >> 46) & 3ull) == kFlagPrefix) break;
            t -= nr + 1;
        }
        if (gave_up) {
            ties[si] = 0u;
            if (status) *(volatile uint32_t *)status = kErrSortWait;
        }
        st_relaxed64(my, lookback_word(epoch, kFlagPrefix, excl + total));
    }
    gbase[dd] = digit_base[dd] + (uint32_t)excl - tbase;
    __syncthreads();  // every digit's place; the sorted tile complete
    // 4. Coalesced runs per digit to the global output.
    if (full)
        write_keys<K, true>(skey, sval, gbase, dig, tile_n, n, keys_out, vals_out);
    else
        write_keys<K, false>(skey, sval, gbase, dig, tile_n, n, keys_out, vals_out);
}

}  // namespace

void radix_scratch_free(RadixScratch &r) {
    void *ptrs[] = {r.lookback, r.hist, r.bases, r.runs, r.ties, r.tiles, r.sample};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    r = RadixScratch{};
}

uint32_t radix_tiles(uint32_t n) {
    return n / (uint32_t)kTileKeys + (n % (uint32_t)kTileKeys != 0u ? 1u : 0u);
}

cr_status radix_begin(RadixScratch &rs, uint32_t nseg, uint64_t ntiles, cudaStream_t s) {
    if (!rs.lookback || rs.cap_tiles < ntiles || rs.cap_segs < nseg) {
        const uint64_t tiles = std::max(ntiles, rs.cap_tiles);
        const uint32_t segs = std::max(nseg, rs.cap_segs);
        radix_scratch_free(rs);
        const size_t rows = (size_t)segs * kRadixMaxPasses * 256;
        CR_CUDA(cudaMalloc((void **)&rs.lookback, tiles * 256 * sizeof(unsigned long long)));
        CR_CUDA(cudaMalloc((void **)&rs.hist, rows * sizeof(uint32_t)));
        CR_CUDA(cudaMalloc((void **)&rs.bases, rows * sizeof(uint32_t)));
        CR_CUDA(cudaMalloc((void **)&rs.runs, segs * sizeof(uint32_t)));
        CR_CUDA(cudaMalloc((void **)&rs.ties, segs * sizeof(uint32_t)));
        CR_CUDA(cudaMalloc((void **)&rs.tiles, kRadixMaxPasses * sizeof(uint32_t)));
        CR_CUDA(cudaMemsetAsync(rs.lookback, 0, tiles * 256 * sizeof(unsigned long long), s));
        rs.cap_tiles = tiles;
        rs.cap_segs = segs;
        rs.epoch = 0;
    }
    CR_CUDA(cudaMemsetAsync(rs.hist, 0, (size_t)nseg * kRadixMaxPasses * 256 * sizeof(uint32_t), s));
    CR_CUDA(cudaMemsetAsync(rs.tiles, 0, kRadixMaxPasses * sizeof(uint32_t), s));
    return CR_OK;
}

template <typename K>
cr_status radix_sort(const RadixBuffers<K> &buf, const RadixSeg *segs, uint32_t nseg,
                     uint64_t ntiles, uint32_t n0, int key_bits, bool ties_ok, RadixScratch &rs,
                     uint32_t wait_limit, uint32_t *status, cudaStream_t s) {
    const int passes = (key_bits + 7) / 8;
    if (nseg == 0 || passes > kRadixMaxPasses || ntiles > rs.cap_tiles || nseg > rs.cap_segs)
        return cri::fail(CR_ERR_INTERNAL, "radix_sort: arguments");
    // A sample is taken of one large segment of 64-bit keys: the passes left
    // out then save more than the sample costs (15 us; at half a million keys
    // two passes take that long).
    const unsigned long long *sampled = nullptr;
    if constexpr (sizeof(K) == 8) {
        if (ties_ok && nseg == 1 && n0 >= kSampleMinKeys) {
            const size_t words = ((size_t)kSampleChoices << kSampleSlotBits) + 2 * kSampleChoices;
            if (!rs.sample) CR_CUDA(cudaMalloc((void **)&rs.sample, words * 8));
            CR_CUDA(cudaMemsetAsync(rs.sample, 0, words * 8, s));
            unsigned long long *found = rs.sample + ((size_t)kSampleChoices << kSampleSlotBits);
            radix_sample<<<kSamples / kThreads, kThreads, 0, s>>>(buf.keys[0], n0, rs.sample, found);
            CR_CUDA(cudaGetLastError());
            sampled = found;
        }
    }
    radix_bases<<<nseg, kThreads, 0, s>>>(rs.hist, segs, passes, sampled, rs.bases, rs.runs, rs.ties);
    CR_CUDA(cudaGetLastError());
    const size_t smem = onesweep_smem_bytes<K>();
    CR_CUDA(cudaFuncSetAttribute(radix_onesweep<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    for (int p = 0; p < passes; ++p) {
        // A fresh epoch per pass, so the look-back words never need clearing;
        // after 65534 epochs the words are cleared once.
        if (++rs.epoch >= 0xffffu) {
            CR_CUDA(cudaMemsetAsync(rs.lookback, 0,
                                    rs.cap_tiles * 256 * sizeof(unsigned long long), s));
            rs.epoch = 1;
        }
        radix_onesweep<K><<<(unsigned)ntiles, kThreads, smem, s>>>(
            buf, segs, nseg, p, rs.bases, rs.runs, rs.lookback, rs.epoch, rs.tiles + p,
            wait_limit, rs.ties, status);
        CR_CUDA(cudaGetLastError());
    }
    return CR_OK;
}

template cr_status radix_sort<uint32_t>(const RadixBuffers<uint32_t> &, const RadixSeg *, uint32_t,
                                        uint64_t, uint32_t, int, bool, RadixScratch &, uint32_t,
                                        uint32_t *, cudaStream_t);
template cr_status radix_sort<unsigned long long>(const RadixBuffers<unsigned long long> &,
                                                  const RadixSeg *, uint32_t, uint64_t, uint32_t,
                                                  int, bool, RadixScratch &, uint32_t, uint32_t *,
                                                  cudaStream_t);
