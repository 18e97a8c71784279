// raster.cu — the per-point passes of the compute rasteriser.
//
//   PASS_DEPTH   depthPassUpdate   (Pipelines/DepthPass/Shaders.metal:21-116)
//   PASS_COLOR   colorPassUpdate   (Pipelines/ColorPass/Shaders.metal:30-219,
//                                   integer R,G,B,count path)
//   PASS_NEAREST nearestDepthUpdate + nearestIndexUpdate
//                (Pipelines/NearestDepth/Shaders.metal:14-91,
//                 Pipelines/NearestIndex/Shaders.metal:14-94) fused into one
//                traversal: the key (depth << 32) | ~pointIndex is combined
//                with a 64-bit max, so the winner is the largest depth and,
//                among equal depths, the lowest point index — the same pixel
//                result as the reference's max pass followed by its
//                min-index pass over the tied points.
//
// Launch shape.  The reference dispatches one 128-thread group per survivor
// of the cull (indirect dispatch).  Here the cull also cuts every survivor's
// point prefix into chunk records of at most `chunkPoints` points carrying
// the per-batch decode values and screen rectangle, and publishes their
// count (the CUDA counterpart of the indirect argument buffer).  A
// persistent grid sized to fill every SM claims the records from a work
// cursor, copying the next record into shared memory (cp.async) while the
// current chunk is processed, so batches of very different sizes spread
// evenly over the SMs.  Each CTA of 256 threads walks a chunk four points
// per thread with 16-byte loads of the level bytes and position / colour
// words; warps skip the projection and the atomics when none of their lanes
// survives the dither or clip tests, and a chunk whose LOD threshold keeps
// every level skips the dither hash.
//
// Screen tiles.  A batch is Morton-compact, so its points land in a small
// screen rectangle (the projection of its AABB's eight corners, widened by
// two pixels, computed by the cull).  When that rectangle has few pixels per
// point, the CTA
// accumulates in shared memory — depth max, or R | count << 20, G and B (a
// chunk of fewer than 4096 points keeps every field below its width), or
// the nearest key — and then flushes one global atomic per touched pixel.  The colour pass
// also stages the rectangle's settled depths in shared memory.  Points that
// round outside the rectangle use global atomics directly, so the tile is a
// cache and never changes a result.  Other batches, large on screen with
// few points per pixel, use one global atomic per point.  Atomics are
// predicated single instructions rather than branches around code.
// Integer max and sum are associative and commutative: the planes are
// bit-identical to a per-point atomic order either way.
#include <algorithm>
#include <type_traits>

#include "cr_device.cuh"
#include "cr_internal.h"
#include "cr_resolve.cuh"

namespace {

constexpr int kThreads = 256;
constexpr uint32_t kFull = 0xffffffffu;

template <int PASS>
struct TileCfg;
template <>
struct TileCfg<PASS_DEPTH> {
    static constexpr int kPx = 8192;
    static constexpr int kBytes = kPx * 4;
};
template <>
struct TileCfg<PASS_COLOR> {
    static constexpr int kPx = 4096;
    static constexpr int kBytes = kPx * 16;  // R|count, G, B accumulators + settled depth
};
template <>
struct TileCfg<PASS_NEAREST> {
    static constexpr int kPx = 4096;
    static constexpr int kBytes = kPx * 8;
};

template <>
struct TileCfg<PASS_DEPTH_FRAG> {
    static constexpr int kPx = 4096;
    static constexpr int kBytes = kPx * 4;
};
// The kernels that draw footprints of more than a pixel only, and so have no
// screen tiles: other kernels draw single pixels in the nearest pass (FP false),
// the one-view colour pass (from fragments), the batched views' depth pass (with
// fragments) and the FP32 passes.
template <int PASS, bool MV, bool FP>
__host__ __device__ constexpr bool footprints_only() {
    return (PASS == PASS_NEAREST && FP) || (PASS == PASS_COLOR && !MV) ||
           (PASS == PASS_DEPTH && MV) || PASS == PASS_COLOR_F32 || PASS == PASS_GRAD;
}
template <int PASS, bool MV>
constexpr int tile_bytes() {
    if constexpr (footprints_only<PASS, MV, true>())
        return 0;
    else
        return TileCfg<PASS>::kBytes;
}

__host__ __device__ constexpr bool is_depth(int p) { return p == PASS_DEPTH || p == PASS_DEPTH_FRAG; }
__host__ __device__ constexpr bool is_color(int p) { return p == PASS_COLOR; }

// Two floats in one 64-bit register pair.  Products and sums are fused
// multiply-adds with an addend of -0 or a factor of 1, each rounded once, and
// the two constants come from the kernel's parameters: as literals they are
// folded away and the products and sums contracted, which rounds otherwise.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void split2(F2 a, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
struct F2Consts {
    F2 one, minus_zero;
    __device__ __forceinline__ F2 mul(F2 a, F2 b) const { return fma2(a, b, minus_zero); }
    __device__ __forceinline__ F2 add(F2 a, F2 b) const { return fma2(a, one, b); }
};

struct RasterArgs {
    const ChunkRec *chunks;
    const cr_raster_file *files;
    InlineFiles ifiles;  // the one-view file table, when small (else ifiles.n = 0)
    uint32_t *counters;
    const uint32_t *low, *med, *high, *colors;
    const uint8_t *levels;
    RasterTargets t;
    RasterUniforms u;
    float keep_scale;  // 1 - depthTolerance
    F2Consts two;      // 1 and -0, twice each
    int radius_zero;   // every footprint is a single pixel
    int use_tiles;
    uint32_t round_shift;  // of the fragment passes' rounds (warp_span)
    uint32_t *frag_xy;     // pixel x | row << 16
    uint2 *frag_zc;     // NDC z bits, RGBA8: two stores per fragment
    uint32_t *frag_count;
    // Differentiable colours: learnable colours, dL/dpixel, gradient (3 floats each).
    const float *fcolors;
    const float *dldimg;
    float *fgrad;
    // Batched views (MV kernels): per-view frames, culls and file tables.
    const ViewDesc *views;
    uint32_t nviews;
    uint32_t nfiles;        // files per view; view v's table starts at files + v * nfiles
    uint32_t chunk_stride;  // view v's chunk records start at chunks + v * chunk_stride
    // Batched views with fragments: chunk record -> offset in its view's
    // fragment span; the arena's capacity; set by the depth pass when the
    // views' spans do not fit (the colour pass then decodes the points).
    const uint32_t *chunk_poff;
    unsigned long long frag_cap;
    uint32_t *frag_overflow;
};

// The frame and camera of the view whose chunk a CTA is drawing (MV kernels).
struct ViewState {
    int width, height;
    uint32_t *depth;
    uint4 *accum;
    unsigned long long *nearest;
    float view[16], proj[16];
};
__shared__ ViewState s_view;

// Frame and camera of the point being drawn: the kernel's own (one view) or
// the current chunk's view (batched views).
template <bool MV>
__device__ __forceinline__ int view_w(const RasterArgs &a) { return MV ? s_view.width : a.u.width; }
template <bool MV>
__device__ __forceinline__ int view_h(const RasterArgs &a) { return MV ? s_view.height : a.u.height; }
template <bool MV>
__device__ __forceinline__ uint32_t *view_depth(const RasterArgs &a) {
    return MV ? s_view.depth : a.t.depth;
}
template <bool MV>
__device__ __forceinline__ uint4 *view_accum(const RasterArgs &a) {
    return MV ? s_view.accum : a.t.accum;
}
template <bool MV>
__device__ __forceinline__ unsigned long long *view_nearest(const RasterArgs &a) {
    return MV ? s_view.nearest : a.t.nearest;
}
template <bool MV>
__device__ __forceinline__ const float *view_view(const RasterArgs &a) {
    return MV ? s_view.view : a.u.view;
}
template <bool MV>
__device__ __forceinline__ const float *view_proj(const RasterArgs &a) {
    return MV ? s_view.proj : a.u.proj;
}

// The current view's size and planes in registers: read once per chunk, not
// per point (loads from shared memory could not be hoisted past the
// shared-memory atomics); for one view, the kernel's own parameters.
template <bool MV>
struct ViewRegsT;
template <>
struct ViewRegsT<true> {
    int W, H;
    uint32_t *depth;
    uint4 *accum;
    unsigned long long *nearest;
};
template <>
struct ViewRegsT<false> {  // reads the kernel parameters where used
    const RasterArgs &a;
    __device__ __forceinline__ ViewRegsT(const RasterArgs &args) : a(args) {}
};
template <bool MV>
__device__ __forceinline__ int vw(const ViewRegsT<MV> &r);
template <>
__device__ __forceinline__ int vw<true>(const ViewRegsT<true> &r) { return r.W; }
template <>
__device__ __forceinline__ int vw<false>(const ViewRegsT<false> &r) { return r.a.u.width; }
template <bool MV>
__device__ __forceinline__ int vh(const ViewRegsT<MV> &r);
template <>
__device__ __forceinline__ int vh<true>(const ViewRegsT<true> &r) { return r.H; }
template <>
__device__ __forceinline__ int vh<false>(const ViewRegsT<false> &r) { return r.a.u.height; }
template <bool MV>
__device__ __forceinline__ uint32_t *vdepth(const ViewRegsT<MV> &r);
template <>
__device__ __forceinline__ uint32_t *vdepth<true>(const ViewRegsT<true> &r) { return r.depth; }
template <>
__device__ __forceinline__ uint32_t *vdepth<false>(const ViewRegsT<false> &r) { return r.a.t.depth; }
template <bool MV>
__device__ __forceinline__ uint4 *vaccum(const ViewRegsT<MV> &r);
template <>
__device__ __forceinline__ uint4 *vaccum<true>(const ViewRegsT<true> &r) { return r.accum; }
template <>
__device__ __forceinline__ uint4 *vaccum<false>(const ViewRegsT<false> &r) { return r.a.t.accum; }
template <bool MV>
__device__ __forceinline__ unsigned long long *vnearest(const ViewRegsT<MV> &r);
template <>
__device__ __forceinline__ unsigned long long *vnearest<true>(const ViewRegsT<true> &r) {
    return r.nearest;
}
template <>
__device__ __forceinline__ unsigned long long *vnearest<false>(const ViewRegsT<false> &r) {
    return r.a.t.nearest;
}
__device__ __forceinline__ ViewRegsT<true> view_regs_mv() {
    return ViewRegsT<true>{s_view.width, s_view.height, s_view.depth, s_view.accum,
                           s_view.nearest};
}

struct BatchShared {
    float T[16];      // file.transform
    F2 T2[16];        // its entries twice (two points at a time)
    float world[16];  // file.world (footprint only)
    uint32_t file;    // file cached in T / world
};

struct PointOut {
    bool ok;
    int ix, iy;  // pixel after the y flip
    uint32_t depth;
    float nz;
    uint32_t color;
    uint32_t pointIndex;
    float px, py, pz;
};

// Dither keep-test of one point (DepthPass/Shaders.metal:174-179).
__device__ __forceinline__ bool keep_point(const RasterArgs &a, const ChunkRec &c,
                                           uint32_t pointIndex, uint32_t lvl) {
    const float pointLevel = (float)(lvl & 7u);
    const float dither = a.u.lodDither ? crd::hash_unit(pointIndex) : 0.5f;
    return !(dither >= (c.thr - pointLevel) + 0.5f);
}

// Split-precision decode: the coarse (low), medium and fine (high) 10-bit
// chunks for level >= 2 (10 bits), level 1 (20 bits) or level 0 (30 bits).  A
// word the chunk's level does not use was never loaded and is zero; the level
// is the same for the whole chunk, so the branch is uniform and each level
// does only its own shifts.
__device__ __forceinline__ void decode_words(const ChunkRec &c, uint32_t lo, uint32_t me,
                                             uint32_t hi, float &fx, float &fy, float &fz) {
    uint32_t x, y, z;
    if (c.level >= 2) {
        x = lo & 1023u;
        y = (lo >> 10) & 1023u;
        z = (lo >> 20) & 1023u;
    } else if (c.level == 1) {
        x = ((lo & 1023u) << 10) | (me & 1023u);
        y = (((lo >> 10) & 1023u) << 10) | ((me >> 10) & 1023u);
        z = (((lo >> 20) & 1023u) << 10) | ((me >> 20) & 1023u);
    } else {
        const uint32_t sl = c.level == 0 ? 20u : 0u, sm = c.level == 0 ? 10u : 0u;
        x = ((lo & 1023u) << sl) | ((me & 1023u) << sm) | (hi & 1023u);
        y = (((lo >> 10) & 1023u) << sl) | (((me >> 10) & 1023u) << sm) | ((hi >> 10) & 1023u);
        z = (((lo >> 20) & 1023u) << sl) | (((me >> 20) & 1023u) << sm) | ((hi >> 20) & 1023u);
    }
    fx = (float)x;
    fy = (float)y;
    fz = (float)z;
}

// Clip tests and pixel of a projected point (ColorPass/Shaders.metal:70-104,
// NearestDepth/Shaders.metal:68-85).
template <int PASS, bool MV>
__device__ __forceinline__ void place_point(const RasterArgs &a, const ViewRegsT<MV> &vr,
                                            const ChunkRec &c, const crd::f4 &clip, PointOut &o) {
    bool ok = o.ok;
    if (clip.w <= 0.0f) ok = false;
    const float nx = clip.x / clip.w, ny = clip.y / clip.w, nz = clip.z / clip.w;
    // |x| > 1 is x < -1 || x > 1 for every float (false for NaN either way).
    if (fabsf(nx) > 1.0f || fabsf(ny) > 1.0f || nz > 1.0f) ok = false;
    if (PASS == PASS_NEAREST ? (nz <= 0.0f) : (nz < 0.0f)) ok = false;
    const int W = vw<MV>(vr), H = vh<MV>(vr);
    o.ix = (int)((nx * 0.5f + 0.5f) * (float)W);
    const int iy = (int)((ny * 0.5f + 0.5f) * (float)H);
    if ((uint32_t)o.ix >= (uint32_t)W || (uint32_t)iy >= (uint32_t)H) ok = false;
    o.iy = H - 1 - iy;
    // depth_to_uint without its clamps: the saturating conversion already
    // maps z * 2^32 to 0 for z <= 0 or NaN and to 0xFFFFFFFF for z >= 1.
    o.depth = __float2uint_rz(nz * 4294967296.0f);
    o.nz = nz;
    o.ok = ok;
    if (PASS == PASS_COLOR || PASS == PASS_DEPTH_FRAG) {  // ColorPass/Shaders.metal:95-100
        if (a.u.colorizeChunks)
            o.color = c.batchIndex * 1234567u;
        else if (a.u.colorizeOverdraw)
            o.color = 0x00010101u;
    }
}

// decodePoint + projection + clip + pixel (DepthPass/Shaders.metal:188-211).
template <int PASS, bool MV>
__device__ __forceinline__ void project_point(const RasterArgs &a, const ViewRegsT<MV> &vr, const float *T,
                                              const ChunkRec &c, uint32_t lo, uint32_t me,
                                              uint32_t hi, PointOut &o) {
    float x, y, z;
    decode_words(c, lo, me, hi, x, y, z);
    o.px = x * c.qx + c.minX;
    o.py = y * c.qy + c.minY;
    o.pz = z * c.qz + c.minZ;
    place_point<PASS, MV>(a, vr, c, crd::mulp(T, o.px, o.py, o.pz), o);
}

// A transform's entries, each twice.
struct Twice {
    const float *T;
    __device__ __forceinline__ F2 operator[](int i) const { return f2(T[i], T[i]); }
};

// project_point of two points.  T2: the transform with every entry twice.  The
// decode's and the transform's 60 products and sums are 30 instructions, of
// which the passes, bound by instruction issue, have one in seven fewer: 100M
// points at 1080p 335 -> 328 us a frame, 64 views 8.45 -> 8.24 ms.
template <int PASS, bool MV, class M>
__device__ __forceinline__ void project_pair(const RasterArgs &a, const ViewRegsT<MV> &vr,
                                             const M T2, const ChunkRec &c, const uint32_t *lo,
                                             const uint32_t *me, const uint32_t *hi, PointOut &o0,
                                             PointOut &o1) {
    float x0, y0, z0, x1, y1, z1;
    decode_words(c, lo[0], me[0], hi[0], x0, y0, z0);
    decode_words(c, lo[1], me[1], hi[1], x1, y1, z1);
    const F2Consts &k = a.two;
    const F2 x = k.add(k.mul(f2(x0, x1), f2(c.qx, c.qx)), f2(c.minX, c.minX));
    const F2 y = k.add(k.mul(f2(y0, y1), f2(c.qy, c.qy)), f2(c.minY, c.minY));
    const F2 z = k.add(k.mul(f2(z0, z1), f2(c.qz, c.qz)), f2(c.minZ, c.minZ));
    auto row = [&](int r, float &v0, float &v1) {
        split2(k.add(k.add(k.add(k.mul(T2[r], x), k.mul(T2[4 + r], y)), k.mul(T2[8 + r], z)),
                     T2[12 + r]),
               v0, v1);
    };
    crd::f4 p0, p1;
    row(0, p0.x, p1.x);
    row(1, p0.y, p1.y);
    row(2, p0.z, p1.z);
    row(3, p0.w, p1.w);
    place_point<PASS, MV>(a, vr, c, p0, o0);
    place_point<PASS, MV>(a, vr, c, p1, o1);
}

__device__ __forceinline__ unsigned long long nearest_key(uint32_t depth, uint32_t index) {
    return ((unsigned long long)depth << 32) | (unsigned long long)(~index);
}


// Reductions into the frame planes (global memory).  Written as red.global
// on explicitly global addresses: the batched-view passes take the plane
// pointers from shared memory, where the compiler cannot tell their
// address space, and would otherwise emit generic atomics that wait for a
// returned value.
__device__ __forceinline__ void red_add_u32(uint32_t *p, uint32_t v) {
    asm volatile("red.global.add.u32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(v)
                 : "memory");
}
__device__ __forceinline__ void red_add_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("red.global.add.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "l"(v)
                 : "memory");
}
__device__ __forceinline__ void red_max_u32(uint32_t *p, uint32_t v) {
    asm volatile("red.global.max.u32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(v)
                 : "memory");
}
__device__ __forceinline__ void red_max_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("red.global.max.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "l"(v)
                 : "memory");
}

__device__ __forceinline__ void red_add_f32x3(float4 *p, float r, float g, float b) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(
                     __cvta_generic_to_global(p)),
                 "f"(r), "f"(g), "f"(b), "f"(0.0f)
                 : "memory");
}

// Differentiable colours, one visible (point, pixel): the forward adds the
// point's FP32 colour and one sample; the adjoint adds dL/dpixel / count to
// the point's gradient (g, in registers, written once per point).
__device__ __forceinline__ void color_f32_sample(const RasterArgs &a, uint32_t pix,
                                                 uint32_t pointIndex) {
    const float *c = a.fcolors + 3 * (size_t)pointIndex;
    red_add_f32x3(a.t.fsum + pix, c[0], c[1], c[2]);
    red_add_u32(a.t.fcount + pix, 1u);
}
__device__ __forceinline__ void grad_sample(const RasterArgs &a, uint32_t pix, float g[3]) {
    const float n = (float)a.t.fcount[pix];
    const float *d = a.dldimg + 3 * (size_t)pix;
    g[0] = g[0] + d[0] / n;
    g[1] = g[1] + d[1] / n;
    g[2] = g[2] + d[2] / n;
}
__device__ __forceinline__ void grad_store(const RasterArgs &a, uint32_t pointIndex,
                                           const float g[3]) {
    float *o = a.fgrad + 3 * (size_t)pointIndex;
    o[0] = o[0] + g[0];
    o[1] = o[1] + g[1];
    o[2] = o[2] + g[2];
}

// Adds one sample group to a pixel's R, G, B and count.  Packed: the uint4
// as two 64-bit words, R | G << 32 and B | count << 32 — half the global
// atomics.  A lower field that passes 2^32 would carry into its neighbour;
// that needs more than kPackedMaxCount samples in the pixel, which the
// resolve detects (the frame is then re-run unpacked).  Unpacked: one
// 32-bit add per field.
template <bool MV>
__device__ __forceinline__ void color_global(const RasterArgs &a, const ViewRegsT<MV> &vr, uint32_t pix, uint32_t r,
                                             uint32_t g, uint32_t b, uint32_t n) {
    if (a.t.packed) {
        unsigned long long *w = reinterpret_cast<unsigned long long *>(&vaccum<MV>(vr)[pix]);
        red_add_u64(w, (unsigned long long)r | ((unsigned long long)g << 32));
        red_add_u64(w + 1, (unsigned long long)b | ((unsigned long long)n << 32));
    } else {
        unsigned int *acc = reinterpret_cast<unsigned int *>(&vaccum<MV>(vr)[pix]);
        red_add_u32(acc + 0, r);
        red_add_u32(acc + 1, g);
        red_add_u32(acc + 2, b);
        red_add_u32(acc + 3, n);
    }
}

// Direct path, radius 0: one global atomic per point (batches large on
// screen, where points rarely share a pixel).
template <int PASS, bool MV>
__device__ __forceinline__ void emit_direct(const RasterArgs &a, const ViewRegsT<MV> &vr, PointOut &o) {
    const uint32_t pix = (uint32_t)(o.iy * vw<MV>(vr) + o.ix);
    if (is_depth(PASS)) {
        if (o.ok) red_max_u32(&vdepth<MV>(vr)[pix], o.depth);
    } else if (is_color(PASS)) {
        const uint32_t closest = o.ok ? vdepth<MV>(vr)[pix] : 0u;
        const bool vis = closest != 0u && o.nz >= crd::uint_to_depth(closest) * a.keep_scale;
        if (vis)
            color_global<MV>(a, vr, pix, o.color & 0xffu, (o.color >> 8) & 0xffu, (o.color >> 16) & 0xffu,
                         1u);
    } else {
        if (o.ok) red_max_u64(&vnearest<MV>(vr)[pix], nearest_key(o.depth, o.pointIndex));
    }
}

// Tile path, radius 0: shared-memory accumulation, global atomics for points
// that round outside the rectangle.  Colour tiles hold R | count << 20, G and
// B per pixel in 32-bit words (exact while a chunk has at most 4095 points).
template <int PASS, bool MV>
__device__ __forceinline__ void emit_tile(const RasterArgs &a, const ViewRegsT<MV> &vr, const ChunkRec &c,
                                          unsigned char *smem, PointOut &o) {
    const int lx = o.ix - c.x0, ly = o.iy - c.y0;
    const bool inside = (unsigned)lx < (unsigned)c.tw && (unsigned)ly < (unsigned)c.th;
    const bool in_tile = o.ok && inside, outside = o.ok && !inside;
    const uint32_t pix = (uint32_t)(o.iy * vw<MV>(vr) + o.ix);
    const int l = inside ? ly * c.tw + lx : 0;
    if (is_depth(PASS)) {
        if (in_tile) atomicMax(reinterpret_cast<uint32_t *>(smem) + l, o.depth);
        if (outside) red_max_u32(&vdepth<MV>(vr)[pix], o.depth);
    } else if (is_color(PASS)) {
        constexpr int kPx = TileCfg<PASS_COLOR>::kPx;
        uint32_t *acc = reinterpret_cast<uint32_t *>(smem);
        const uint32_t *sdep = acc + 3 * kPx;
        uint32_t closest = sdep[l];
        if (outside) closest = vdepth<MV>(vr)[pix];
        const bool vis = o.ok && closest != 0u &&
                         o.nz >= crd::uint_to_depth(closest) * a.keep_scale;
        const uint32_t r = o.color & 0xffu, g = (o.color >> 8) & 0xffu,
                       b = (o.color >> 16) & 0xffu;
        if (vis && inside) {
            atomicAdd(acc + l, r | (1u << 20));
            atomicAdd(acc + kPx + l, g);
            atomicAdd(acc + 2 * kPx + l, b);
        }
        if (vis && !inside) color_global<MV>(a, vr, pix, r, g, b, 1u);
    } else {
        const unsigned long long k = nearest_key(o.depth, o.pointIndex);
        if (in_tile) atomicMax(reinterpret_cast<unsigned long long *>(smem) + l, k);
        if (outside) red_max_u64(&vnearest<MV>(vr)[pix], k);
    }
}

// General footprint (radius from pointFootprintRadius), global atomics.
template <int PASS, bool MV>
__device__ __forceinline__ void emit_footprint(const RasterArgs &a, const ViewRegsT<MV> &vr, const BatchShared &sb,
                                               const PointOut &o) {
    if (!o.ok) return;
    const crd::PointSize ps{a.u.pointSizeMode, a.u.minimumPointSize, a.u.maximumPointSize,
                            a.u.pointSizeScale};
    const int rad =
        crd::footprint_radius(o.px, o.py, o.pz, sb.world, view_view<MV>(a), view_proj<MV>(a), vh<MV>(vr), ps);
    const int W = vw<MV>(vr), H = vh<MV>(vr);
    float g[3] = {0.0f, 0.0f, 0.0f};  // PASS_GRAD
    for (int oy = -rad; oy <= rad; ++oy) {
        for (int ox = -rad; ox <= rad; ++ox) {
            if (!crd::inside_footprint(ox, oy, rad)) continue;
            const int tx = o.ix + ox, ty = o.iy + oy;
            if (tx < 0 || tx >= W || ty < 0 || ty >= H) continue;
            const uint32_t pix = (uint32_t)(ty * W + tx);
            if (is_depth(PASS)) {
                red_max_u32(&vdepth<MV>(vr)[pix], o.depth);
            } else if (is_color(PASS) || PASS == PASS_COLOR_F32 || PASS == PASS_GRAD) {
                const uint32_t closest = vdepth<MV>(vr)[pix];
                if (closest == 0u) continue;
                if (!(o.nz >= crd::uint_to_depth(closest) * a.keep_scale)) continue;
                if (PASS == PASS_COLOR_F32)
                    color_f32_sample(a, pix, o.pointIndex);
                else if (PASS == PASS_GRAD)
                    grad_sample(a, pix, g);
                else
                    color_global<MV>(a, vr, pix, o.color & 0xffu, (o.color >> 8) & 0xffu,
                                     (o.color >> 16) & 0xffu, 1u);
            } else {
                red_max_u64(&vnearest<MV>(vr)[pix], nearest_key(o.depth, o.pointIndex));
            }
        }
    }
    if (PASS == PASS_GRAD) grad_store(a, o.pointIndex, g);
}

// A chunk's points are split over the CTA's warps in contiguous pieces of
// whole rounds (warp_span points a warp, the same split in every
// pass): each warp packs the fragments of its piece from the piece's own
// start, counting them in a register, and leaves its count beside the other
// warps' (kFragWarps per chunk record); the colour pass walks each piece with
// the warp of the same number.  One count per chunk instead took a
// shared-memory atomic and a shuffle per point (per two points in the
// one-view kernel, at the price of eight registers).  100M points at 1080p: the
// frame 358 -> 353 us; a 1M-point lattice at 720p 45.6 -> 41.0; 64 views of 50M
// points 9.30 -> 9.12 ms.
constexpr uint32_t kFragWarps = kThreads / 32;
static_assert(kFragWarps == kFragCounts, "the count arrays have a word per warp");
// A round is 128 points, four to a lane, or 32 where pointsPerBatch is no
// multiple of four: most batches then start unaligned and are read a point to a
// lane (2M points in batches of 257 at 1080p: 71 us with pieces of 128, 58 so).
// round_shift: its logarithm, the same for all of a cloud's passes.
__device__ __forceinline__ uint32_t warp_span(uint32_t round_shift, uint32_t count) {
    static_assert(kFragWarps == 8, "a round for every warp is eight rounds");
    return (((count - 1u) >> (round_shift + 3)) + 1u) << round_shift;
}

// Appends the warp's kept points at fragment `at`, lanes placed by ballot
// rank; returns how many were kept.
__device__ __forceinline__ uint32_t emit_fragment(const RasterArgs &a, uint32_t at,
                                                  const PointOut &o) {
    const uint32_t ballot = __ballot_sync(kFull, o.ok);
    if (o.ok) {
        const uint32_t i = at + __popc(ballot & ((1u << (threadIdx.x & 31)) - 1u));
        a.frag_xy[i] = (uint32_t)o.ix | ((uint32_t)o.iy << 16);
        a.frag_zc[i] = make_uint2(__float_as_uint(o.nz), o.color);
    }
    return __popc(ballot);
}

// One point; every lane of the warp calls this (warp-uniform early outs).
// frag_at: the depth pass's next fragment, advanced by the points it kept.
template <int PASS, bool MV, bool FP>
__device__ __forceinline__ void do_point(const RasterArgs &a, const ViewRegsT<MV> &vr, const BatchShared &sb,
                                         unsigned char *smem, const ChunkRec &c, bool tiled,
                                         bool valid, uint32_t local, uint32_t lvl, uint32_t lo,
                                         uint32_t me, uint32_t hi, uint32_t color,
                                         uint32_t &frag_at, bool emit, bool all_keep) {
    PointOut o;
    o.pointIndex = c.first + local;
    o.color = color;
    o.ok = valid;
    if (!all_keep) o.ok = o.ok && keep_point(a, c, o.pointIndex, lvl);
    // The depth passes keep nearly every point, so a warp vote to skip the
    // projection or the emission would cost more than it saves (the
    // emission is correct for a warp with no kept point).
    if (!is_depth(PASS) && !__any_sync(kFull, o.ok)) return;
    project_point<PASS, MV>(a, vr, sb.T, c, lo, me, hi, o);
    if (!is_depth(PASS) && !__any_sync(kFull, o.ok)) return;
    if constexpr (footprints_only<PASS, MV, FP>()) {
        emit_footprint<PASS, MV>(a, vr, sb, o);
    } else {
        if (FP && !a.radius_zero)
            emit_footprint<PASS, MV>(a, vr, sb, o);
        else if (tiled)
            emit_tile<PASS, MV>(a, vr, c, smem, o);
        else
            emit_direct<PASS, MV>(a, vr, o);
    }
    if (PASS == PASS_DEPTH_FRAG && emit) frag_at += emit_fragment(a, frag_at, o);
}

template <int PASS, bool MV>
__device__ __forceinline__ void tile_init(const RasterArgs &a, const ChunkRec &c,
                                          unsigned char *smem) {
    const int n = c.tw * c.th;
    for (int l = threadIdx.x; l < n; l += kThreads) {
        if (is_depth(PASS)) {
            reinterpret_cast<uint32_t *>(smem)[l] = 0u;
        } else if (is_color(PASS)) {
            constexpr int kPx = TileCfg<PASS_COLOR>::kPx;
            uint32_t *acc = reinterpret_cast<uint32_t *>(smem);
            acc[l] = 0u;
            acc[kPx + l] = 0u;
            acc[2 * kPx + l] = 0u;
            const int gx = c.x0 + l % c.tw, gy = c.y0 + l / c.tw;
            acc[3 * kPx + l] = view_depth<MV>(a)[gy * view_w<MV>(a) + gx];
        } else {
            reinterpret_cast<unsigned long long *>(smem)[l] = 0ull;
        }
    }
}

template <int PASS, bool MV>
__device__ __forceinline__ void tile_flush(const RasterArgs &a, const ViewRegsT<MV> &vr, const ChunkRec &c,
                                           const unsigned char *smem) {
    const int n = c.tw * c.th;
    for (int l = threadIdx.x; l < n; l += kThreads) {
        const uint32_t pix = (uint32_t)((c.y0 + l / c.tw) * vw<MV>(vr) + c.x0 + l % c.tw);
        if (is_depth(PASS)) {
            const uint32_t v = reinterpret_cast<const uint32_t *>(smem)[l];
            if (v) red_max_u32(&vdepth<MV>(vr)[pix], v);
        } else if (is_color(PASS)) {
            constexpr int kPx = TileCfg<PASS_COLOR>::kPx;
            const uint32_t *acc = reinterpret_cast<const uint32_t *>(smem);
            const uint32_t rc = acc[l];
            const uint32_t cnt = rc >> 20;
            if (cnt) color_global<MV>(a, vr, pix, rc & 0xfffffu, acc[kPx + l], acc[2 * kPx + l], cnt);
        } else {
            const unsigned long long k = reinterpret_cast<const unsigned long long *>(smem)[l];
            if (k) red_max_u64(&vnearest<MV>(vr)[pix], k);
        }
    }
}

// 16-byte asynchronous global -> shared copy (cp.async), for the chunk record.
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gmem_src) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem_src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem_dst, const void *gmem_src) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem_src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// Largest view v with begin[v] <= k (views without chunks share their
// begin with the next view, so the view found holds chunk k).
__device__ __forceinline__ uint32_t find_view(const uint32_t *begin, uint32_t nviews, uint32_t k) {
    uint32_t lo = 0, hi = nviews;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (begin[mid] <= k)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// Persistent pass over the chunk records: the record of the CTA's next chunk
// is copied into shared memory with cp.async while the current chunk is
// processed.  One view: the CTAs claim chunks from the cloud's work cursor
// (dynamic schedule; a chunk's work varies with its batch's LOD prefix), and
// the last CTA to finish resets the cursor for the next launch.  Batched views (MV): the chunks of
// all views form one index space, view after view; each CTA scans the
// per-view chunk counts once, finds a chunk's view by binary search and
// switches frame, camera and file table when the view changes.
// FP: footprints may be larger than a pixel.  Without them (fragments are of
// single pixels; the nearest pass when its points are) the generic footprint
// code stays out, and two points are projected at a time.
template <int PASS, bool MV, bool FP>
__device__ __forceinline__ void raster_body(const RasterArgs &a) {
    constexpr bool kFrag = PASS == PASS_DEPTH_FRAG;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ BatchShared sb;
    __shared__ __align__(16) ChunkRec rec[2];
    __shared__ __align__(16) uint32_t rec_poff[2][4];  // offset in the view's fragment span
    __shared__ uint32_t s_vbegin[MV ? kMaxViews + 1 : 1];
    __shared__ unsigned long long s_pbegin[MV && kFrag ? kMaxViews + 1 : 1];
    __shared__ uint32_t s_wsum[kThreads / 32];
    crd::grid_wait();
    crd::launch_dependents();
    if (a.t.redo && *a.t.redo == 0u) return;
    uint32_t nchunks;
    bool emit = true;  // fragments fit the arena (batched views)
    if (MV) {
        // Exclusive prefixes over the views (at most kMaxViews) of their chunk
        // counts and, with fragments, of their fragment spans.
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const uint32_t* vc = a.counters + threadIdx.x * CNT_COUNT;
        uint32_t x = threadIdx.x < a.nviews ? vc[CNT_CHUNKS] : 0u;
        unsigned long long y = (kFrag && threadIdx.x < a.nviews) ? vc[CNT_POINTS] : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t xs = __shfl_up_sync(kFull, x, o);
            const unsigned long long ys = __shfl_up_sync(kFull, y, o);
            if (lane >= o) {
                x += xs;
                y += ys;
            }
        }
        if (lane == 31) s_wsum[warp] = x;
        if (kFrag && lane == 31) s_pbegin[warp] = y;
        __syncthreads();
        for (int w = 0; w < warp; ++w) {
            x += s_wsum[w];
            if (kFrag) y += s_pbegin[w];
        }
        __syncthreads();
        s_vbegin[threadIdx.x + 1] = x;
        if (kFrag) s_pbegin[threadIdx.x + 1] = y;
        if (threadIdx.x == 0) {
            s_vbegin[0] = 0u;
            if (kFrag) s_pbegin[0] = 0ull;
        }
        __syncthreads();
        nchunks = s_vbegin[a.nviews];
        if (kFrag) {
            emit = s_pbegin[a.nviews] <= a.frag_cap;
            if (PASS == PASS_DEPTH_FRAG && blockIdx.x == 0 && threadIdx.x == 0)
                *a.frag_overflow = emit ? 0u : 1u;
        }
    } else {
        nchunks = a.counters[CNT_CHUNKS];
    }
    // Chunks are claimed from a work cursor in the launch's counters (the
    // cull zeroes it; the last CTA to finish resets it for the next launch):
    // a dynamic schedule, since a chunk's work varies with its batch's LOD
    // prefix and its view.  Thread 0 claims the next chunk, finds its view
    // and record and prefetches the record while the CTA draws the current
    // one.
    __shared__ uint32_t s_k[2], s_kview[2], s_kslot[2];  // per record buffer
    auto finish = [&]() {
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(a.counters + CNT_DONE, 1u) == gridDim.x - 1u) {
                a.counters[CNT_WORK_DEPTH] = 0u;
                a.counters[CNT_DONE] = 0u;
            }
        }
    };
    // View of chunk kk and the index of its record (also its fragment-count slot).
    auto locate = [&](uint32_t kk, uint32_t &view) -> uint32_t {
        if (!MV) {
            view = 0u;
            return kk;
        }
        view = find_view(s_vbegin, a.nviews, kk);
        return view * a.chunk_stride + (kk - s_vbegin[view]);
    };
    // Thread 0: claim a chunk into record buffer b and start its copy.
    auto claim = [&](int b) {
        const uint32_t kk = atomicAdd(a.counters + CNT_WORK_DEPTH, 1u);
        s_k[b] = kk;
        if (kk >= nchunks) return;
        uint32_t view;
        const uint32_t slot = locate(kk, view);
        s_kview[b] = view;
        s_kslot[b] = slot;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            cp_async16(reinterpret_cast<uint4 *>(&rec[b]) + q,
                       reinterpret_cast<const uint4 *>(a.chunks + slot) + q);
        if (MV && kFrag) cp_async4(&rec_poff[b][0], a.chunk_poff + slot);
    };
    if (threadIdx.x == 0) {
        claim(0);
        sb.file = 0xffffffffu;
    }
    cp_async_commit();
    uint32_t loaded_view = 0xffffffffu;
    for (int buf = 0;; buf ^= 1) {
        cp_async_wait_all();
        __syncthreads();  // rec[buf] complete; the previous chunk is fully done
        if (s_k[buf] >= nchunks) break;
        const uint32_t cur_view = s_kview[buf], cur_slot = s_kslot[buf];
        // Batched views read the record where it is: sixteen registers fewer, and
        // a fifth CTA per SM (depth_views_kernel).
        std::conditional_t<MV, const ChunkRec &, const ChunkRec> c = rec[buf];
        const uint32_t fslot = cur_slot;
        // First fragment of the chunk: pool index space (one view), or the
        // view's fragment span in the arena (batched views).
        const uint32_t fbase =
            MV ? (kFrag ? (uint32_t)(s_pbegin[cur_view] + rec_poff[buf][0]) : 0u) : c.first;
        if (threadIdx.x == 0) claim(buf ^ 1);
        cp_async_commit();
        const uint32_t file_id = MV ? cur_view * a.nfiles + c.file : c.file;
        const bool new_file = file_id != sb.file;
        bool tiled = false;
        if constexpr (!footprints_only<PASS, MV, FP>())
            tiled = a.use_tiles && a.radius_zero && c.tw > 0 &&
                    c.tw * c.th <= TileCfg<PASS>::kPx && c.tw * c.th <= (int)c.count &&
                    (!is_color(PASS) || c.count < 4096u);
        if (new_file || tiled) {
            __syncthreads();  // everyone has read sb.file (and the view state)
            if (new_file) {
                // The kernels take RasterArgs as a __grid_constant__
                // parameter, so the inline table is read in place.
                const cr_raster_file *file = &(a.ifiles.n ? a.ifiles.f : a.files)[file_id];
                if (threadIdx.x < 16)
                {
                    const float t = file->transform[threadIdx.x];
                    sb.T[threadIdx.x] = t;
                    sb.T2[threadIdx.x] = f2(t, t);
                }
                else if (threadIdx.x < 32)
                    sb.world[threadIdx.x - 16] = file->world[threadIdx.x - 16];
                if (threadIdx.x == 0) sb.file = file_id;
            }
            if (MV && cur_view != loaded_view) {  // a new view always brings a new file id
                const ViewDesc &vd = a.views[cur_view];
                if (threadIdx.x >= 32 && threadIdx.x < 48)
                    s_view.view[threadIdx.x - 32] = vd.view[threadIdx.x - 32];
                else if (threadIdx.x >= 48 && threadIdx.x < 64)
                    s_view.proj[threadIdx.x - 48] = vd.proj[threadIdx.x - 48];
                else if (threadIdx.x == 64) {
                    s_view.width = vd.width;
                    s_view.height = vd.height;
                    s_view.depth = vd.depth;
                    s_view.accum = vd.accum;
                    s_view.nearest = vd.nearest;
                }
                loaded_view = cur_view;
                if (tiled) __syncthreads();  // the tile's set-up reads the view state
            }
            if constexpr (!footprints_only<PASS, MV, FP>())
                if (tiled) tile_init<PASS, MV>(a, c, smem);
            __syncthreads();
        }
        // The view's size and planes: registers (batched views, read once
        // per chunk) or the kernel's parameters (one view).
        const ViewRegsT<MV> vr = [&] {
            if constexpr (MV)
                return view_regs_mv();
            else
                return ViewRegsT<false>(a);
        }();
        const bool need_med = c.level <= 1, need_high = c.level == 0;
        constexpr bool kNeedColor = PASS == PASS_COLOR || PASS == PASS_DEPTH_FRAG;
        // Every point of the chunk passes the dither test when even its
        // highest level (7) does with the largest dither (hash_unit reaches
        // 1.0f; 0.5f without dither): (thr - L) + 0.5f only grows as L falls.
        const bool all_keep = (a.u.lodDither ? 1.0f : 0.5f) < (c.thr - 7.0f) + 0.5f;
        // The warp's piece of the chunk and its fragments' place.
        const uint32_t span = warp_span(a.round_shift, c.count), piece = (threadIdx.x >> 5) * span;
        // Passes without fragments take rounds of the whole CTA in turn.
        constexpr bool kPieces = PASS == PASS_DEPTH_FRAG;
        const uint32_t end = kPieces ? min(piece + span, c.count) : c.count;
        const uint32_t frag0 = fbase + piece;
        uint32_t frag_at = frag0;
        // The nearest pass of single pixels takes records of no more points than
        // threads a point to a thread: four in turn are the longer chain (2M points
        // in batches of 16 at 1080p 188 us, 94 so; of 64 87 and 51).
        const bool spread = !kPieces && !FP && c.count <= kThreads;
        if ((c.first & 3u) == 0u && !spread) {
            // Four points per thread, 16-byte loads.
            const uint32_t nquads = (c.count + 3u) >> 2;
            for (uint32_t p0 = kPieces ? piece : 0u; kPieces ? p0 < end : p0 < nquads;
                 p0 += kPieces ? 128u : kThreads) {
                const uint32_t l0 = kPieces ? p0 + 4u * (threadIdx.x & 31) : 4u * (p0 + threadIdx.x);
                const bool qv = kPieces ? l0 < end : p0 + threadIdx.x < nquads;
                const uint32_t base = c.first + l0;
                uint32_t lv4 = 0;
                uint4 lo4 = make_uint4(0, 0, 0, 0), me4 = lo4, hi4 = lo4, co4 = lo4;
                if (qv) {
                    lv4 = __ldg(reinterpret_cast<const uint32_t *>(a.levels + base));
                    lo4 = __ldg(reinterpret_cast<const uint4 *>(a.low + base));
                    if (need_med) me4 = __ldg(reinterpret_cast<const uint4 *>(a.med + base));
                    if (need_high) hi4 = __ldg(reinterpret_cast<const uint4 *>(a.high + base));
                    if (kNeedColor)
                        co4 = __ldg(reinterpret_cast<const uint4 *>(a.colors + base));
                }
                const uint32_t lvs[4] = {lv4 & 0xffu, (lv4 >> 8) & 0xffu, (lv4 >> 16) & 0xffu,
                                         lv4 >> 24};
                const uint32_t los[4] = {lo4.x, lo4.y, lo4.z, lo4.w};
                const uint32_t mes[4] = {me4.x, me4.y, me4.z, me4.w};
                const uint32_t his[4] = {hi4.x, hi4.y, hi4.z, hi4.w};
                const uint32_t cos[4] = {co4.x, co4.y, co4.z, co4.w};
                if constexpr (!FP) {
#pragma unroll
                    for (int j = 0; j < 4; j += 2) {
                        PointOut o[2];
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            o[q].pointIndex = c.first + l0 + j + q;
                            o[q].color = cos[j + q];
                            o[q].ok = l0 + j + q < end;
                            if (!all_keep)
                                o[q].ok = o[q].ok && keep_point(a, c, o[q].pointIndex, lvs[j + q]);
                        }
                        project_pair<PASS, MV, const F2 *>(a, vr, sb.T2, c, los + j, mes + j,
                                                           his + j, o[0], o[1]);
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            if (tiled)
                                emit_tile<PASS, MV>(a, vr, c, smem, o[q]);
                            else
                                emit_direct<PASS, MV>(a, vr, o[q]);
                            if (PASS == PASS_DEPTH_FRAG && emit)
                                frag_at += emit_fragment(a, frag_at, o[q]);
                        }
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        do_point<PASS, MV, FP>(a, vr, sb, smem, c, tiled, l0 + j < end, l0 + j, lvs[j],
                                           los[j], mes[j], his[j], cos[j], frag_at, emit,
                                           all_keep);
                }
            }
        } else {
            // Unaligned start (pointsPerBatch not a multiple of 4), or few points: one
            // point per thread.
            for (uint32_t p0 = kPieces ? piece : (threadIdx.x & ~31u); p0 < end;
                 p0 += kPieces ? 32u : kThreads) {
                const uint32_t local = p0 + (threadIdx.x & 31);
                const bool v = local < end;
                const uint32_t i = c.first + (v ? local : 0u);
                const uint32_t lv = v ? a.levels[i] : 0u;
                const uint32_t lo = v ? a.low[i] : 0u;
                const uint32_t me = (v && need_med) ? a.med[i] : 0u;
                const uint32_t hi = (v && need_high) ? a.high[i] : 0u;
                const uint32_t co = (v && kNeedColor) ? a.colors[i] : 0u;
                do_point<PASS, MV, FP>(a, vr, sb, smem, c, tiled, v, local, lv, lo, me, hi, co,
                                   frag_at, emit, all_keep);
            }
        }
        if (PASS == PASS_DEPTH_FRAG && (threadIdx.x & 31) == 0)
            a.frag_count[fslot * kFragWarps + (threadIdx.x >> 5)] = frag_at - frag0;
        if constexpr (!footprints_only<PASS, MV, FP>())
            if (tiled) {
                __syncthreads();
                tile_flush<PASS, MV>(a, vr, c, smem);
            }
    }
    cp_async_wait_all();
    finish();
}

// Colour pass over the depth pass's fragments for one view, one chunk per CTA
// (claimed from the work cursor).  A chunk's points are one compact region of
// a Morton-ordered batch: its fragments hit few distinct pixels, but rarely
// in a row (over a 1080p frame of 100M points, 10.7M visible fragments,
// 1.9M distinct pixels per chunk).  Each visible fragment is summed into a
// shared-memory table with one slot per pixel of a small window (R, G, B,
// count as 32-bit sums: a chunk holds at most 65,536 points, so none
// overflows; 64-bit shared atomics were slower), and the table is flushed
// with one global add pair (or four 32-bit adds) per distinct pixel.  A
// fragment whose slot another pixel has taken is added to the frame directly:
// probing further costs more than that add (100M-point 1080p frame: 364 us
// with 16 probes, 355 with 2, 352 with none; a 1M-point lattice at 720p, whose
// chunks have more pixels than slots, 54 against 48 us; 2048 slots 377,
// 512 slots 351 us but 120 instead of 118 us for 20M sparse points).
constexpr int kHashBits = 10;
constexpr uint32_t kHashSlots = 1u << kHashBits;
constexpr uint32_t kHashEmpty = 0xffffffffu;

// Slot of pixel (x, y): x + 37 y over the table.  Distinct pixels of any
// 37 × 27 window take distinct slots, and the 32 lanes of a warp, whose
// fragments lie in one small patch of the screen, mostly fall in distinct
// shared-memory banks (x + 5 y mod 32).
__device__ __forceinline__ uint32_t hash_slot(uint32_t xy) {
    return ((xy & 0xffffu) + 37u * (xy >> 16)) & (kHashSlots - 1u);
}

template <bool MV>
__device__ __forceinline__ void hash_add(uint32_t *hkey, uint32_t *hsum, const RasterArgs &a,
                                         const ViewRegsT<MV> &vr, uint32_t pix, uint32_t xy,
                                         uint32_t col) {
    const uint32_t r = col & 0xffu, g = (col >> 8) & 0xffu, b = (col >> 16) & 0xffu;
    const uint32_t h = hash_slot(xy);
    uint32_t cur = hkey[h];
    if (cur == kHashEmpty) cur = atomicCAS(hkey + h, kHashEmpty, pix);
    if (cur == kHashEmpty || cur == pix) {
        atomicAdd(hsum + h, r);
        atomicAdd(hsum + kHashSlots + h, g);
        atomicAdd(hsum + 2 * kHashSlots + h, b);
        atomicAdd(hsum + 3 * kHashSlots + h, 1u);
    } else {
        color_global<MV>(a, vr, pix, r, g, b, 1u);
    }
}

// Clears the table (at kernel start).
__device__ __forceinline__ void hash_clear(uint32_t *hkey, uint32_t *hsum) {
    for (uint32_t i = threadIdx.x; i < kHashSlots; i += kThreads) {
        hkey[i] = kHashEmpty;
        hsum[i] = hsum[kHashSlots + i] = hsum[2 * kHashSlots + i] = hsum[3 * kHashSlots + i] = 0u;
    }
}

// Streaming loads of two fragments' words (zero where there are none).
__device__ __forceinline__ uint2 load2(const uint32_t *p, bool in) {
    return in ? __ldcs(reinterpret_cast<const uint2 *>(p)) : make_uint2(0u, 0u);
}
__device__ __forceinline__ uint4 load4(const uint2 *p, bool in) {
    return in ? __ldcs(reinterpret_cast<const uint4 *>(p)) : make_uint4(0u, 0u, 0u, 0u);
}

// The colour pass over the fragments of chunk record `slot`, whose range
// starts at base, against the frame of W columns whose depth plane is `depth`:
// sums into the table.  Each warp walks its piece of the range.
template <bool MV>
__device__ __forceinline__ void hash_frags(const RasterArgs &a, const ViewRegsT<MV> &vr,
                                           uint32_t *hkey, uint32_t *hsum, size_t slot,
                                           uint32_t base, int W, const uint32_t *depth) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t n = __ldg(a.frag_count + slot * kFragWarps + warp);
    base += warp * warp_span(a.round_shift, __ldg(&a.chunks[slot].count));
    if ((base & 3u) == 0u) {
        // Two neighbouring fragments per lane and half round: a piece's last
        // round then fills whole half warps before it leaves lanes idle.
        for (uint32_t f0 = 2u * lane; f0 - 2u * lane < n; f0 += 128u) {
            const uint32_t f1 = f0 + 64u;
            const uint2 x0 = load2(a.frag_xy + base + f0, f0 < n);
            const uint2 x1 = load2(a.frag_xy + base + f1, f1 < n);
            const uint4 z0 = load4(a.frag_zc + base + f0, f0 < n);
            const uint4 z1 = load4(a.frag_zc + base + f1, f1 < n);
            const uint32_t fs[4] = {f0, f0 + 1u, f1, f1 + 1u};
            const uint32_t xs[4] = {x0.x, x0.y, x1.x, x1.y}, cs[4] = {z0.y, z0.w, z1.y, z1.w};
            const float zs[4] = {__uint_as_float(z0.x), __uint_as_float(z0.z),
                                 __uint_as_float(z1.x), __uint_as_float(z1.z)};
            uint32_t pix[4], cl[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                pix[q] = (xs[q] >> 16) * (uint32_t)W + (xs[q] & 0xffffu);
                cl[q] = fs[q] < n ? __ldg(depth + pix[q]) : 0u;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (cl[q] != 0u && zs[q] >= crd::uint_to_depth(cl[q]) * a.keep_scale)
                    hash_add<MV>(hkey, hsum, a, vr, pix[q], xs[q], cs[q]);
        }
    } else {
        for (uint32_t f = lane; f < n; f += 32u) {
            const uint32_t xy = a.frag_xy[base + f];
            const uint32_t pix = (xy >> 16) * (uint32_t)W + (xy & 0xffffu);
            const uint32_t cl = __ldg(depth + pix);
            const uint2 zc = a.frag_zc[base + f];
            if (cl != 0u && __uint_as_float(zc.x) >= crd::uint_to_depth(cl) * a.keep_scale)
                hash_add<MV>(hkey, hsum, a, vr, pix, xy, zc.y);
        }
    }
}

// Flushes the table (one global add pair per distinct pixel) and clears it.
// With a cursor, thread 0 also claims the next chunk into *next, so the
// claim's round trip overlaps the flush.  Called after a barrier that
// completes the sums (and after every thread has read the current claim).
template <bool MV>
__device__ __forceinline__ void hash_flush(const RasterArgs &a, const ViewRegsT<MV> &vr,
                                           uint32_t *hkey, uint32_t *hsum,
                                           uint32_t *cursor = nullptr, uint32_t *next = nullptr) {
    uint32_t claimed = 0u;
    if (cursor && threadIdx.x == 0) claimed = atomicAdd(cursor, 1u);
    for (uint32_t i = threadIdx.x; i < kHashSlots; i += kThreads) {
        const uint32_t pix = hkey[i];
        if (pix == kHashEmpty) continue;
        color_global<MV>(a, vr, pix, hsum[i], hsum[kHashSlots + i], hsum[2 * kHashSlots + i],
                         hsum[3 * kHashSlots + i]);
        hkey[i] = kHashEmpty;
        hsum[i] = hsum[kHashSlots + i] = hsum[2 * kHashSlots + i] = hsum[3 * kHashSlots + i] = 0u;
    }
    if (cursor && threadIdx.x == 0) *next = claimed;
}

// The colour pass over chunk k of one view.  Every thread of the CTA calls
// this; the caller's barrier before the next chunk orders the clearing
// before its first add.
__device__ __forceinline__ void hash_chunk(const RasterArgs &a, const ViewRegsT<false> &vr,
                                           uint32_t *hkey, uint32_t *hsum, uint32_t k,
                                           uint32_t *cursor = nullptr, uint32_t *next = nullptr) {
    hash_frags<false>(a, vr, hkey, hsum, k, __ldg(&a.chunks[k].first), a.u.width, a.t.depth);
    __syncthreads();  // the chunk's sums are complete (and k has been read by all)
    hash_flush<false>(a, vr, hkey, hsum, cursor, next);
}

// 1024 slots (about three times a chunk's typical distinct visible pixels)
// and at most 40 registers: six CTAs share an SM.
__global__ void __launch_bounds__(kThreads, 6) color_hash_kernel(const __grid_constant__ RasterArgs a) {
    crd::grid_wait();
    crd::launch_dependents();
    if (a.t.redo && *a.t.redo == 0u) return;
    __shared__ uint32_t hkey[kHashSlots];
    __shared__ uint32_t hsum[4 * kHashSlots];
    __shared__ uint32_t s_k;
    const uint32_t nchunks = a.counters[CNT_CHUNKS];
    const ViewRegsT<false> vr(a);
    hash_clear(hkey, hsum);
    uint32_t *cursor = a.counters + CNT_WORK_DEPTH;
    if (threadIdx.x == 0) s_k = atomicAdd(cursor, 1u);
    for (;;) {
        __syncthreads();  // s_k and the cleared table
        const uint32_t k = s_k;
        if (k >= nchunks) break;
        hash_chunk(a, vr, hkey, hsum, k, cursor, &s_k);  // claims the next chunk into s_k
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(a.counters + CNT_DONE, 1u) == gridDim.x - 1u) {
            a.counters[CNT_WORK_DEPTH] = 0u;
            a.counters[CNT_DONE] = 0u;
        }
    }
}

// The colour pass of a group of batched views over their fragments: the
// one-view hash kernel with each chunk's view found by binary search over
// the per-view chunk prefix (as the point passes do), accumulating into that
// view's planes.  It returns at once when the group's fragments overflowed
// the arena; color_views_kernel then decodes the points instead.
__global__ void __launch_bounds__(kThreads, 6)
    color_hash_views_kernel(const __grid_constant__ RasterArgs a) {
    crd::grid_wait();
    if (*a.frag_overflow) return;
    __shared__ uint32_t hkey[kHashSlots];
    __shared__ uint32_t hsum[4 * kHashSlots];
    __shared__ uint32_t s_vbegin[kMaxViews + 1];
    __shared__ unsigned long long s_pbegin[kMaxViews + 1];
    __shared__ uint32_t s_wsum[kThreads / 32];
    __shared__ unsigned long long s_psum[kThreads / 32];
    __shared__ uint32_t s_k;
    // Exclusive prefixes over the views (at most kMaxViews = kThreads) of
    // their chunk counts and fragment spans.
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const uint32_t *vc = a.counters + threadIdx.x * CNT_COUNT;
        uint32_t x = threadIdx.x < a.nviews ? vc[CNT_CHUNKS] : 0u;
        unsigned long long y = threadIdx.x < a.nviews ? vc[CNT_POINTS] : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t xs = __shfl_up_sync(kFull, x, o);
            const unsigned long long ys = __shfl_up_sync(kFull, y, o);
            if (lane >= o) {
                x += xs;
                y += ys;
            }
        }
        if (lane == 31) {
            s_wsum[warp] = x;
            s_psum[warp] = y;
        }
        __syncthreads();
        for (int w = 0; w < warp; ++w) {
            x += s_wsum[w];
            y += s_psum[w];
        }
        s_vbegin[threadIdx.x + 1] = x;
        s_pbegin[threadIdx.x + 1] = y;
        if (threadIdx.x == 0) {
            s_vbegin[0] = 0u;
            s_pbegin[0] = 0ull;
        }
    }
    hash_clear(hkey, hsum);
    uint32_t *cursor = a.counters + CNT_WORK_DEPTH;
    if (threadIdx.x == 0) s_k = atomicAdd(cursor, 1u);
    __syncthreads();  // prefixes, table and first claim
    const uint32_t nchunks = s_vbegin[a.nviews];
    for (;;) {
        const uint32_t k = s_k;
        if (k >= nchunks) break;
        const uint32_t view = find_view(s_vbegin, a.nviews, k);
        const uint32_t slot = view * a.chunk_stride + (k - s_vbegin[view]);
        const ViewDesc &vd = a.views[view];
        const ViewRegsT<true> vr{vd.width, vd.height, vd.depth, vd.accum, vd.nearest};
        hash_frags<true>(a, vr, hkey, hsum, slot,
                         (uint32_t)(s_pbegin[view] + __ldg(a.chunk_poff + slot)), vd.width,
                         vd.depth);
        __syncthreads();  // the chunk's sums are complete (and k has been read by all)
        hash_flush<true>(a, vr, hkey, hsum, cursor, &s_k);
        __syncthreads();  // the next claim and the cleared table
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(a.counters + CNT_DONE, 1u) == gridDim.x - 1u) {
            a.counters[CNT_WORK_DEPTH] = 0u;
            a.counters[CNT_DONE] = 0u;
        }
    }
}

// ---------------------------------------------------------------------------
// Footprints of more than a pixel (world- or screen-sized splats), one view.
// A step is 1,024 consecutive points of a chunk record, four to a thread.
// Their splats overlap one another many times over a compact patch of the
// screen, so a step finds the rectangle that its splats really cover (the
// record's rectangle is the whole batch's), sums the patch in shared memory
// and sends each touched pixel to the frame once.  The depth pass leaves each
// kept point as a fragment, its radius in the colour's alpha byte (which no
// sum uses), and the colour pass starts from those instead of decoding,
// projecting and sizing the points again.  A step whose rectangle is larger
// than the tile goes to the frame pixel by pixel.
// 20M points with 0.5 m splats at 1080p: the frame 433 -> 280 us (one global
// atomic (depth), and one depth read and two global adds (colour) per splat
// pixel, with a second decode, took 108 and 292 us; these passes 72 and 119).
// Bound by the scattered global adds of the steps that do not fit a tile:
// without tiles 305 us; tiles of 4,096 pixels (three CTAs an SM) the same as
// of 2,048, of 6,144 or steps of 512 or 2,048 points slower; larger
// rectangles cut into bands of the tile's size 338 us, since their splats
// overlap too little to pay for clearing and flushing the bands.
// ---------------------------------------------------------------------------
constexpr int kSplatEach = 4;  // points per thread and step
constexpr uint32_t kSplatPoints = kSplatEach * kThreads;
constexpr int kSplatPx = 2048;  // 16 KB of depths; 64 KB of sums and thresholds

// Rectangle of a step's splats, clamped to the frame; tiled: it fits the tile.
struct SplatBox {
    int x0, y0, w, h;
    bool any, tiled;
};
struct SplatShared {
    int lo[2], hi[2];
    uint32_t frags, next;
};

// Rows and columns of the splat of radius r at (x, y) inside a W x H frame.
struct SplatSpan {
    int x0, x1, y0, y1;
};
__device__ __forceinline__ SplatSpan splat_span(int x, int y, int r, int W, int H) {
    return SplatSpan{max(x - r, 0), min(x + r, W - 1), max(y - r, 0), min(y + r, H - 1)};
}
// insidePointFootprint over whole numbers: ox^2 + oy^2 <= (r + 1/2)^2.
__device__ __forceinline__ bool splat_inside(int ox, int oy, int r) {
    return ox * ox + oy * oy <= r * r + r;
}

// Adds a thread's splats to the step's rectangle; every thread calls it, and a
// barrier follows before splat_box.
__device__ __forceinline__ void splat_widen(SplatShared &ss, const SplatSpan &s) {
    const int x0 = __reduce_min_sync(kFull, s.x0), y0 = __reduce_min_sync(kFull, s.y0);
    const int x1 = __reduce_max_sync(kFull, s.x1), y1 = __reduce_max_sync(kFull, s.y1);
    if ((threadIdx.x & 31) == 0 && x0 <= x1) {
        atomicMin(&ss.lo[0], x0);
        atomicMin(&ss.lo[1], y0);
        atomicMax(&ss.hi[0], x1);
        atomicMax(&ss.hi[1], y1);
    }
}
__device__ __forceinline__ SplatBox splat_box(const SplatShared &ss, int use_tiles) {
    SplatBox b;
    b.x0 = ss.lo[0];
    b.y0 = ss.lo[1];
    b.w = ss.hi[0] - b.x0 + 1;
    b.h = ss.hi[1] - b.y0 + 1;
    b.any = b.w > 0;
    b.tiled = use_tiles && b.any && (long long)b.w * b.h <= kSplatPx;
    return b;
}
constexpr int kFar = 1 << 30;
__device__ __forceinline__ void splat_reset(SplatShared &ss) {  // one thread
    ss.lo[0] = ss.lo[1] = kFar;
    ss.hi[0] = ss.hi[1] = -1;
    ss.frags = 0u;
}
// The depth a splat must reach to be seen in a pixel whose depth word is
// `closest` (none reaches an untouched pixel's).
__device__ __forceinline__ float splat_threshold(uint32_t closest, float keep_scale) {
    return closest != 0u ? crd::uint_to_depth(closest) * keep_scale : __int_as_float(0x7f800000);
}
// A fragment's splat added to the frame pixel by pixel.
__device__ __forceinline__ void splat_to_frame(const RasterArgs &a, const ViewRegsT<false> &vr,
                                               uint32_t xy, uint2 zc) {
    const int W = a.u.width, x = (int)(xy & 0xffffu), y = (int)(xy >> 16), r = (int)(zc.y >> 24);
    const SplatSpan s = splat_span(x, y, r, W, a.u.height);
    for (int ty = s.y0; ty <= s.y1; ++ty)
        for (int tx = s.x0; tx <= s.x1; ++tx) {
            if (!splat_inside(tx - x, ty - y, r)) continue;
            const uint32_t pix = (uint32_t)(ty * W + tx);
            if (__uint_as_float(zc.x) >= splat_threshold(__ldg(a.t.depth + pix), a.keep_scale))
                color_global<false>(a, vr, pix, zc.y & 0xffu, (zc.y >> 8) & 0xffu,
                                    (zc.y >> 16) & 0xffu, 1u);
        }
}
// Steps per chunk record, from the size that the cull gave its records.  The
// records' steps are no more than two and a half times the records at the
// smallest size, of which the fragment counts have room for kFragCounts.
__device__ __forceinline__ uint32_t splat_steps(const uint32_t *counters) {
    return (counters[CNT_CHUNK_POINTS] + kSplatPoints - 1) / kSplatPoints;
}
// Steps are claimed from the cloud's work cursor, as the point passes claim
// their records; the last CTA resets it.
__device__ __forceinline__ void splat_finish(const RasterArgs &a) {
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(a.counters + CNT_DONE, 1u) == gridDim.x - 1u) {
            a.counters[CNT_WORK_DEPTH] = 0u;
            a.counters[CNT_DONE] = 0u;
        }
    }
}

__global__ void __launch_bounds__(kThreads, 4)
    splat_depth(const __grid_constant__ RasterArgs a) {
    __shared__ uint32_t tile[kSplatPx];
    __shared__ SplatShared ss;
    __shared__ __align__(16) float sfile[kInlineFiles][32];  // transform, world
    for (uint32_t t = threadIdx.x; t < 32u * a.ifiles.n; t += kThreads) {
        const cr_raster_file &f = a.ifiles.f[t >> 5];
        sfile[t >> 5][t & 31u] = (t & 16u) ? f.world[t & 15u] : f.transform[t & 15u];
    }
    crd::grid_wait();
    crd::launch_dependents();
    const ViewRegsT<false> vr(a);
    const int W = a.u.width, H = a.u.height;
    const crd::PointSize ps{a.u.pointSizeMode, a.u.minimumPointSize, a.u.maximumPointSize,
                            a.u.pointSizeScale};
    const int lane = threadIdx.x & 31;
    const uint32_t steps = splat_steps(a.counters), total = a.counters[CNT_CHUNKS] * steps;
    uint32_t *cursor = a.counters + CNT_WORK_DEPTH;
    if (threadIdx.x == 0) {
        ss.next = atomicAdd(cursor, 1u);
        splat_reset(ss);
    }
    for (;;) {
        __syncthreads();  // the claim; the last step is done with the tile
        const uint32_t v = ss.next;
        if (v >= total) break;
        const uint32_t k = v / steps, l0 = (v - k * steps) * kSplatPoints;
        ChunkRec c;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            reinterpret_cast<uint4 *>(&c)[q] = __ldg(reinterpret_cast<const uint4 *>(a.chunks + k) + q);
        const bool need_med = c.level <= 1, need_high = c.level == 0;
        uint32_t lv[kSplatEach], lo[kSplatEach], me[kSplatEach], hi[kSplatEach], co[kSplatEach];
#pragma unroll
        for (int j = 0; j < kSplatEach; ++j) {
            const uint32_t l = l0 + j * kThreads + threadIdx.x, i = c.first + l;
            const bool in = l < c.count;
            lv[j] = in ? __ldg(a.levels + i) : 0u;
            lo[j] = in ? __ldg(a.low + i) : 0u;
            me[j] = in && need_med ? __ldg(a.med + i) : 0u;
            hi[j] = in && need_high ? __ldg(a.high + i) : 0u;
            co[j] = in ? __ldg(a.colors + i) : 0u;
        }
        const float *T = a.ifiles.n ? sfile[c.file] : a.files[c.file].transform;
        const float *world = a.ifiles.n ? sfile[c.file] + 16 : a.files[c.file].world;
        const bool all_keep = (a.u.lodDither ? 1.0f : 0.5f) < (c.thr - 7.0f) + 0.5f;
        uint32_t xy[kSplatEach], depth[kSplatEach];
        int rad[kSplatEach];
        SplatSpan mine{kFar, -1, kFar, -1};
#pragma unroll
        for (int j = 0; j < kSplatEach; ++j) {
            const uint32_t l = l0 + j * kThreads + threadIdx.x;
            PointOut o;
            o.pointIndex = c.first + l;
            o.color = co[j];
            o.ok = l < c.count;
            if (!all_keep) o.ok = o.ok && keep_point(a, c, o.pointIndex, lv[j]);
            project_point<PASS_DEPTH_FRAG, false>(a, vr, T, c, lo[j], me[j], hi[j], o);
            rad[j] = -1;
            xy[j] = depth[j] = 0u;
            if (o.ok) {
                rad[j] = crd::footprint_radius(o.px, o.py, o.pz, world, a.u.view, a.u.proj, H, ps);
                xy[j] = (uint32_t)o.ix | ((uint32_t)o.iy << 16);
                depth[j] = o.depth;
                const SplatSpan s = splat_span(o.ix, o.iy, rad[j], W, H);
                mine.x0 = min(mine.x0, s.x0);
                mine.x1 = max(mine.x1, s.x1);
                mine.y0 = min(mine.y0, s.y0);
                mine.y1 = max(mine.y1, s.y1);
            }
            const uint32_t kept = __ballot_sync(kFull, o.ok);
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&ss.frags, __popc(kept));
            at = __shfl_sync(kFull, at, 0);
            if (o.ok) {
                const uint32_t i = c.first + l0 + at + __popc(kept & ((1u << lane) - 1u));
                a.frag_xy[i] = xy[j];
                a.frag_zc[i] = make_uint2(__float_as_uint(o.nz),
                                          (o.color & 0xffffffu) | ((uint32_t)rad[j] << 24));
            }
        }
        splat_widen(ss, mine);
        __syncthreads();
        const SplatBox box = splat_box(ss, a.use_tiles);
        if (box.tiled) {
            for (int l = threadIdx.x; l < box.w * box.h; l += kThreads) tile[l] = 0u;
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < kSplatEach; ++j) {
            if (rad[j] < 0) continue;
            const int x = (int)(xy[j] & 0xffffu), y = (int)(xy[j] >> 16);
            const SplatSpan s = splat_span(x, y, rad[j], W, H);
            for (int ty = s.y0; ty <= s.y1; ++ty)
                for (int tx = s.x0; tx <= s.x1; ++tx) {
                    if (!splat_inside(tx - x, ty - y, rad[j])) continue;
                    if (box.tiled) {
                        const int l = (ty - box.y0) * box.w + tx - box.x0;
                        if (tile[l] < depth[j]) atomicMax(tile + l, depth[j]);
                    } else {
                        red_max_u32(a.t.depth + (size_t)ty * W + tx, depth[j]);
                    }
                }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            a.frag_count[v] = ss.frags;
            ss.next = atomicAdd(cursor, 1u);
            splat_reset(ss);
        }
        if (box.tiled)
            for (int l = threadIdx.x; l < box.w * box.h; l += kThreads)
                if (tile[l])
                    red_max_u32(a.t.depth + (size_t)(box.y0 + l / box.w) * W + box.x0 + l % box.w,
                                tile[l]);
    }
    splat_finish(a);
}

// Dynamic shared memory: R | count << 20, G, B sums (a step's 1,024 points
// keep every field below its width) and the pixels' visibility thresholds.
constexpr int kSplatColorBytes = kSplatPx * 16;
__global__ void __launch_bounds__(kThreads, 5)
    splat_color(const __grid_constant__ RasterArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t *acc = reinterpret_cast<uint32_t *>(smem);
    float *thr = reinterpret_cast<float *>(acc + 3 * kSplatPx);
    __shared__ SplatShared ss;
    crd::grid_wait();
    crd::launch_dependents();
    const ViewRegsT<false> vr(a);
    const int W = a.u.width, H = a.u.height;
    const uint32_t steps = splat_steps(a.counters), total = a.counters[CNT_CHUNKS] * steps;
    uint32_t *cursor = a.counters + CNT_WORK_DEPTH;
    if (threadIdx.x == 0) {
        ss.next = atomicAdd(cursor, 1u);
        splat_reset(ss);
    }
    for (;;) {
        __syncthreads();  // the claim; the last step is done with the tile
        const uint32_t v = ss.next;
        if (v >= total) break;
        const uint32_t k = v / steps;
        const uint32_t n = __ldg(a.frag_count + v);
        const uint32_t base = __ldg(&a.chunks[k].first) + (v - k * steps) * kSplatPoints;
        uint32_t xy[kSplatEach], col[kSplatEach];
        float z[kSplatEach];
#pragma unroll
        for (int j = 0; j < kSplatEach; ++j) {
            const uint32_t f = j * kThreads + threadIdx.x;
            xy[j] = f < n ? __ldcs(a.frag_xy + base + f) : 0u;
            const uint2 q = f < n ? __ldcs(a.frag_zc + base + f) : make_uint2(0u, 0u);
            z[j] = __uint_as_float(q.x);
            col[j] = q.y;
        }
        SplatSpan mine{kFar, -1, kFar, -1};
#pragma unroll
        for (int j = 0; j < kSplatEach; ++j)
            if (j * kThreads + threadIdx.x < n) {
                const SplatSpan s = splat_span((int)(xy[j] & 0xffffu), (int)(xy[j] >> 16),
                                               (int)(col[j] >> 24), W, H);
                mine.x0 = min(mine.x0, s.x0);
                mine.x1 = max(mine.x1, s.x1);
                mine.y0 = min(mine.y0, s.y0);
                mine.y1 = max(mine.y1, s.y1);
            }
        splat_widen(ss, mine);
        __syncthreads();
        const SplatBox box = splat_box(ss, a.use_tiles);
        if (box.tiled) {
            for (int l = threadIdx.x; l < box.w * box.h; l += kThreads) {
                acc[l] = acc[kSplatPx + l] = acc[2 * kSplatPx + l] = 0u;
                thr[l] = splat_threshold(
                    __ldg(a.t.depth + (size_t)(box.y0 + l / box.w) * W + box.x0 + l % box.w),
                    a.keep_scale);
            }
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < kSplatEach; ++j) {
            if (j * kThreads + threadIdx.x >= n) continue;
            if (!box.tiled) {
                splat_to_frame(a, vr, xy[j], make_uint2(__float_as_uint(z[j]), col[j]));
                continue;
            }
            const int x = (int)(xy[j] & 0xffffu), y = (int)(xy[j] >> 16), r = (int)(col[j] >> 24);
            const SplatSpan s = splat_span(x, y, r, W, H);
            for (int ty = s.y0; ty <= s.y1; ++ty)
                for (int tx = s.x0; tx <= s.x1; ++tx) {
                    if (!splat_inside(tx - x, ty - y, r)) continue;
                    const int l = (ty - box.y0) * box.w + tx - box.x0;
                    if (z[j] >= thr[l]) {
                        atomicAdd(acc + l, (col[j] & 0xffu) | (1u << 20));
                        atomicAdd(acc + kSplatPx + l, (col[j] >> 8) & 0xffu);
                        atomicAdd(acc + 2 * kSplatPx + l, (col[j] >> 16) & 0xffu);
                    }
                }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            ss.next = atomicAdd(cursor, 1u);
            splat_reset(ss);
        }
        if (box.tiled)
            for (int l = threadIdx.x; l < box.w * box.h; l += kThreads) {
                const uint32_t rc = acc[l];
                if (rc >> 20)
                    color_global<false>(
                        a, vr, (uint32_t)((box.y0 + l / box.w) * W + box.x0 + l % box.w),
                        rc & 0xfffffu, acc[kSplatPx + l], acc[2 * kSplatPx + l], rc >> 20);
            }
    }
    splat_finish(a);
}

// Exact re-run of a frame whose packed colour adds may have carried (the
// resolve set the redo word).  One CTA, launched every frame, that returns
// at once unless the word is set; then, in order, it zeroes the
// accumulators, runs the colour pass of every cloud over its fragments with
// one 32-bit add per field, and resolves every pixel.  A single CTA orders
// the three steps with block barriers, so they take one launch instead of
// three; the re-run is rare and its speed does not matter.
struct RedoCloud {
    const ChunkRec *chunks;
    const uint32_t *counters, *frag_count, *frag_xy;
    const uint2 *frag_zc;
    uint32_t round_shift;
};
constexpr uint32_t kRedoMaxClouds = 32;
struct RedoArgs {
    RasterArgs a;  // frame targets (unpacked adds) and uniforms; per-cloud fields from clouds[]
    RedoCloud clouds[kRedoMaxClouds];
    uint32_t nclouds;
    const uint32_t *redo;
    uint32_t *rgba;
    float *depthf;
    uint32_t npix;
    ResolveUniforms ru;
    int splats;  // the fragments are the splat passes'
};

__global__ void __launch_bounds__(kThreads) hqs_redo_kernel(RedoArgs r) {
    crd::grid_wait();
    crd::launch_dependents();
    if (*r.redo == 0u) return;
    __shared__ uint32_t hkey[kHashSlots];
    __shared__ uint32_t hsum[4 * kHashSlots];
    for (uint32_t p = threadIdx.x; p < r.npix; p += kThreads) r.a.t.accum[p] = make_uint4(0, 0, 0, 0);
    hash_clear(hkey, hsum);
    __syncthreads();  // accumulators and table zeroed
    for (uint32_t ci = 0; ci < r.nclouds; ++ci) {
        RasterArgs a = r.a;
        a.chunks = r.clouds[ci].chunks;
        a.frag_count = const_cast<uint32_t *>(r.clouds[ci].frag_count);
        a.frag_xy = const_cast<uint32_t *>(r.clouds[ci].frag_xy);
        a.frag_zc = const_cast<uint2 *>(r.clouds[ci].frag_zc);
        a.round_shift = r.clouds[ci].round_shift;
        const ViewRegsT<false> vr(a);
        const uint32_t nchunks = r.clouds[ci].counters[CNT_CHUNKS];
        if (r.splats) {
            const uint32_t steps = splat_steps(r.clouds[ci].counters), total = nchunks * steps;
            for (uint32_t v = 0; v < total; ++v) {
                const uint32_t k = v / steps;
                const uint32_t base = a.chunks[k].first + (v - k * steps) * kSplatPoints;
                for (uint32_t f = threadIdx.x; f < a.frag_count[v]; f += kThreads)
                    splat_to_frame(a, vr, a.frag_xy[base + f], a.frag_zc[base + f]);
            }
            continue;
        }
        for (uint32_t k = 0; k < nchunks; ++k) {
            hash_chunk(a, vr, hkey, hsum, k);
            __syncthreads();  // the table is clear again
        }
    }
    __threadfence();
    __syncthreads();  // every add of the block has reached L2
    for (uint32_t p = threadIdx.x; p < r.npix; p += kThreads) {
        const uint4 acc = __ldcg(r.a.t.accum + p);
        crd::resolve_pixel(acc, acc.w ? r.a.t.depth[p] : 0u, r.ru, r.rgba[p], r.depthf[p]);
    }
}

// The nearest pass of larger footprints asks for four CTAs per SM: left to the
// compiler it had 48 registers, some spilled, and 5M points of 4 m splats at
// 1080p took 1268 us, 1052 so (1028 at three, but 20M points of 0.5 m splats 161
// instead of 147).
template <int PASS, bool MV>
__global__ void __launch_bounds__(kThreads, PASS == PASS_NEAREST ? 4 : 1) raster_kernel(const __grid_constant__ RasterArgs a) {
    raster_body<PASS, MV, true>(a);
}

// The nearest pass of single-pixel points, at five CTAs per SM (48 registers, a
// few spilled): 100M points at 1080p 207 us with the generic footprint code,
// 195 so, 204 at four; 206 at five with one point at a time.
__global__ void __launch_bounds__(kThreads, 5)
    nearest_kernel(const __grid_constant__ RasterArgs a) {
    raster_body<PASS_NEAREST, false, false>(a);
}

// The differentiable passes of one view with single-pixel footprints (depth
// plane, FP32 colour sums, adjoint): 512 points of a chunk record to a step,
// two to a thread, as many steps to a record as the size that the cull gave
// its records takes; the grid strides over all of them.  A training view holds a million points or so, of which the
// four-points-a-thread passes make two rounds in the few hundred chunks that
// there are: half of the SMs' warps had no work, and each waited for its
// chain of loads (record, words, depth, colour) alone.  Steps spread the work
// over every warp slot, and a thread's two points wait together.  10M points,
// 512 x 512, 16 views: the step 1.80 ms with the four-point passes, 1.17 with a
// point a thread (six CTAs an SM; 1.14 with eight), 1.12 with two (1.14 with
// five CTAs), 1.19 with four; 1.10 with the two in the same instructions.
constexpr int kStepEach = 2;  // points per thread and step
static_assert(kStepEach % 2 == 0, "points are projected in pairs");
constexpr int kStepPoints = kStepEach * kThreads;
template <int PASS>
__global__ void __launch_bounds__(kThreads, 6)
    point_pass(const __grid_constant__ RasterArgs a) {
    // The inline files' transforms; a larger table is read where it is.
    __shared__ __align__(16) float sT[kInlineFiles][16];
    for (uint32_t t = threadIdx.x; t < 16u * a.ifiles.n; t += kThreads)
        sT[t >> 4][t & 15u] = a.ifiles.f[t >> 4].transform[t & 15u];
    crd::grid_wait();
    crd::launch_dependents();
    __syncthreads();
    const ViewRegsT<false> vr(a);
    const int W = a.u.width;
    const uint32_t steps = (a.counters[CNT_CHUNK_POINTS] + kStepPoints - 1) / kStepPoints;
    const uint32_t total = a.counters[CNT_CHUNKS] * steps;
    for (uint32_t v = blockIdx.x; v < total; v += gridDim.x) {
        const uint32_t k = v / steps, local0 = (v - k * steps) * kStepPoints + threadIdx.x;
        ChunkRec c;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            reinterpret_cast<uint4 *>(&c)[q] = __ldg(reinterpret_cast<const uint4 *>(a.chunks + k) + q);
        if (local0 >= c.count) continue;
        const float *T = a.ifiles.n ? sT[c.file] : a.files[c.file].transform;
        const bool all_keep = (a.u.lodDither ? 1.0f : 0.5f) < (c.thr - 7.0f) + 0.5f;
        uint32_t lo[kStepEach], me[kStepEach], hi[kStepEach], lv[kStepEach];
#pragma unroll
        for (int j = 0; j < kStepEach; ++j) {
            const uint32_t i = c.first + local0 + j * kThreads;
            const bool in = local0 + j * kThreads < c.count;
            lo[j] = in ? __ldg(a.low + i) : 0u;
            me[j] = in && c.level <= 1 ? __ldg(a.med + i) : 0u;
            hi[j] = in && c.level == 0 ? __ldg(a.high + i) : 0u;
            lv[j] = in && !all_keep ? __ldg(a.levels + i) : 0u;
        }
        PointOut o[kStepEach];
        uint32_t pix[kStepEach], closest[kStepEach];
#pragma unroll
        for (int j = 0; j < kStepEach; ++j) {
            o[j].pointIndex = c.first + local0 + j * kThreads;
            o[j].color = 0u;
            o[j].ok = local0 + j * kThreads < c.count;
            if (!all_keep) o[j].ok = o[j].ok && keep_point(a, c, o[j].pointIndex, lv[j]);
            if (j & 1)
                project_pair<PASS, false>(a, vr, Twice{T}, c, lo + j - 1, me + j - 1, hi + j - 1,
                                          o[j - 1], o[j]);
        }
#pragma unroll
        for (int j = 0; j < kStepEach; ++j) {
            pix[j] = (uint32_t)(o[j].iy * W + o[j].ix);
            if (PASS == PASS_DEPTH) {
                if (o[j].ok) red_max_u32(a.t.depth + pix[j], o[j].depth);
            } else {
                closest[j] = o[j].ok ? __ldg(a.t.depth + pix[j]) : 0u;
            }
        }
        if constexpr (PASS != PASS_DEPTH) {
#pragma unroll
            for (int j = 0; j < kStepEach; ++j) {
                if (closest[j] == 0u ||
                    !(o[j].nz >= crd::uint_to_depth(closest[j]) * a.keep_scale))
                    continue;
                if (PASS == PASS_COLOR_F32) {
                    color_f32_sample(a, pix[j], o[j].pointIndex);
                } else {
                    float g[3] = {0.0f, 0.0f, 0.0f};
                    grad_sample(a, pix[j], g);
                    grad_store(a, o[j].pointIndex, g);
                }
            }
        }
    }
}

// The one-view depth passes fit 64 registers without spilling, so four CTAs
// (and their screen tiles, 16 KB with fragments and 32 without) share an SM.
template <int PASS>
__global__ void __launch_bounds__(kThreads, 4) depth_kernel(const __grid_constant__ RasterArgs a) {
    raster_body<PASS, false, PASS != PASS_DEPTH_FRAG>(a);
}

// The batched-view depth passes at five CTAs per SM (48 registers, a dozen
// spilled): 64 views of 50M points 8.83 ms, 9.05 ms at four, 9.13 ms with the
// chunk record in registers (9.41 ms at five).  With footprints 16 views of 20M
// points 2.86 ms, 2.88 at four.
template <int PASS>
__global__ void __launch_bounds__(kThreads, 5)
    depth_views_kernel(const __grid_constant__ RasterArgs a) {
    raster_body<PASS, true, PASS != PASS_DEPTH_FRAG>(a);
}

// The batched views' colour pass that decodes the points holds a 64 KB screen
// tile, so at most three CTAs share an SM whatever their registers; saying so
// lets the compiler use up to 85 registers per thread instead of spilling.
template <bool MV>
__global__ void __launch_bounds__(kThreads, 3) raster_kernel_color(const __grid_constant__ RasterArgs a) {
    raster_body<PASS_COLOR, MV, true>(a);
}

// Colour pass of batched views whose fragments overflowed the arena: the
// decode-and-project pass (color_hash_views_kernel draws the others).
__global__ void __launch_bounds__(kThreads, 3) color_views_kernel(const __grid_constant__ RasterArgs a) {
    if (*a.frag_overflow) raster_body<PASS_COLOR, true, true>(a);
}

// The kernel a pass launches.
template <int PASS, bool MV>
constexpr auto kernel_for() {
    if constexpr (PASS == PASS_COLOR)
        return raster_kernel_color<MV>;
    else if constexpr (!MV && is_depth(PASS))
        return depth_kernel<PASS>;
    else if constexpr (MV && is_depth(PASS))
        return depth_views_kernel<PASS>;
    else
        return raster_kernel<PASS, MV>;
}

template <typename Kernel>
int resident_blocks(Kernel k, int smem) {
    int n = 0;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kThreads, smem) != cudaSuccess) n = 1;
    return n < 1 ? 1 : n;
}

template <int PASS, bool MV>
int blocks_per_sm_for() {
    int n = 0;
    constexpr auto k = kernel_for<PASS, MV>();
    constexpr int kBytes = tile_bytes<PASS, MV>();
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kThreads, kBytes) != cudaSuccess)
        n = 1;
    return n < 1 ? 1 : n;
}

int color_views_blocks_per_sm() {
    int n = 0;
    constexpr int kBytes = TileCfg<PASS_COLOR>::kBytes;
    cudaFuncSetAttribute(color_views_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, color_views_kernel, kThreads, kBytes) !=
        cudaSuccess)
        n = 1;
    return n < 1 ? 1 : n;
}

template <bool MV>
int raster_blocks_per_sm(int pass) {
    switch (pass) {
    case PASS_DEPTH: return blocks_per_sm_for<PASS_DEPTH, MV>();
    case PASS_COLOR: return blocks_per_sm_for<PASS_COLOR, MV>();
    case PASS_DEPTH_FRAG: return blocks_per_sm_for<PASS_DEPTH_FRAG, MV>();
    case PASS_COLOR_FRAG:
        if (MV) return color_views_blocks_per_sm();
        {
            int n = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, color_hash_kernel, kThreads, 0) !=
                cudaSuccess)
                n = 1;
            return n < 1 ? 1 : n;
        }
    default:
        if constexpr (MV)
            return 1;  // batched views draw HQS only
        else
            return blocks_per_sm_for<PASS_NEAREST, false>();
    }
}

RasterArgs make_args(cr_cloud *cloud, const RasterUniforms &u, const RasterTargets &t) {
    RasterArgs a;
    a.chunks = cloud->d_chunks;
    a.files = cloud->d_files;
    a.ifiles = inline_files(cloud);
    a.counters = cloud->d_counters;
    a.low = cloud->d_low;
    a.med = cloud->d_med;
    a.high = cloud->d_high;
    a.colors = cloud->d_colors;
    a.levels = cloud->d_levels;
    a.t = t;
    a.u = u;
    a.keep_scale = 1.0f - u.depthTolerance;
    a.two = F2Consts{F2{0x3f8000003f800000ull}, F2{0x8000000080000000ull}};
    // pointFootprintRadius clamps the size to [lo, hi] with lo >= 1; when the
    // upper bound is 1 every radius is 0 whatever the distance.
    a.radius_zero = fmaxf(u.minimumPointSize, u.maximumPointSize) <= 1.0f ? 1 : 0;
    a.use_tiles = cloud->ctx->use_tiles ? 1 : 0;
    a.round_shift = cloud->cap.pointsPerBatch % 4u == 0u ? 7u : 5u;
    a.frag_xy = cloud->d_frag_xy;
    a.frag_zc = cloud->d_frag_zc;
    a.frag_count = cloud->d_frag_count;
    a.views = nullptr;
    a.nviews = 0;
    a.nfiles = 0;
    a.chunk_stride = 0;
    a.chunk_poff = nullptr;
    a.frag_cap = 0;
    a.frag_overflow = nullptr;
    a.fcolors = nullptr;
    a.dldimg = nullptr;
    a.fgrad = nullptr;
    return a;
}

// One-view passes start while the previous kernel drains (programmatic
// dependent launch); batched views, captured in a graph, launch plainly.
template <int PASS, bool MV>
void launch_pass(const RasterArgs &a, int grid, cudaStream_t s) {
    if constexpr (MV)
        kernel_for<PASS, MV>()<<<grid, kThreads, (tile_bytes<PASS, MV>()), s>>>(a);
    else
        launch_programmatic(kernel_for<PASS, MV>(), dim3(grid), dim3(kThreads),
                            (size_t)tile_bytes<PASS, MV>(), s, a);
}

}  // namespace

cr_status launch_raster(cr_cloud *cloud, RasterPass pass, const RasterUniforms &u,
                        const RasterTargets &t, cudaStream_t s) {
    const RasterArgs a = make_args(cloud, u, t);
    cr_context *ctx = cloud->ctx;
    if (ctx->blocks_per_sm[pass] == 0) ctx->blocks_per_sm[pass] = raster_blocks_per_sm<false>(pass);
    const int grid = ctx->sm_count * ctx->blocks_per_sm[pass];
    switch (pass) {
    case PASS_DEPTH: launch_pass<PASS_DEPTH, false>(a, grid, s); break;
    case PASS_COLOR: launch_pass<PASS_COLOR, false>(a, grid, s); break;
    case PASS_DEPTH_FRAG: launch_pass<PASS_DEPTH_FRAG, false>(a, grid, s); break;
    case PASS_COLOR_FRAG:
        CR_CUDA(launch_programmatic(color_hash_kernel, dim3(grid), dim3(kThreads), 0, s, a));
        break;
    default:
        if (a.radius_zero) {
            constexpr int kBytes = TileCfg<PASS_NEAREST>::kBytes;
            if (ctx->blocks_per_sm_nearest == 0)
                ctx->blocks_per_sm_nearest = resident_blocks(nearest_kernel, kBytes);
            CR_CUDA(launch_programmatic(nearest_kernel,
                                        dim3(ctx->sm_count * ctx->blocks_per_sm_nearest),
                                        dim3(kThreads), (size_t)kBytes, s, a));
        } else {
            launch_pass<PASS_NEAREST, false>(a, grid, s);
        }
        break;
    }
    CR_CUDA(cudaGetLastError());
    return CR_OK;
}

cr_status launch_splats(cr_cloud *cloud, bool color, const RasterUniforms &u,
                        const RasterTargets &t, cudaStream_t s) {
    const RasterArgs a = make_args(cloud, u, t);
    if (!a.ifiles.n) {
        const cr_status st = ensure_device_files(cloud);
        if (st) return st;
    }
    cr_context *ctx = cloud->ctx;
    if (color) {
        if (ctx->blocks_per_sm_splat[1] == 0)
            ctx->blocks_per_sm_splat[1] = resident_blocks(splat_color, kSplatColorBytes);
        CR_CUDA(launch_programmatic(splat_color, dim3(ctx->sm_count * ctx->blocks_per_sm_splat[1]),
                                    dim3(kThreads), (size_t)kSplatColorBytes, s, a));
    } else {
        if (ctx->blocks_per_sm_splat[0] == 0)
            ctx->blocks_per_sm_splat[0] = resident_blocks(splat_depth, 0);
        CR_CUDA(launch_programmatic(splat_depth, dim3(ctx->sm_count * ctx->blocks_per_sm_splat[0]),
                                    dim3(kThreads), 0, s, a));
    }
    return CR_OK;
}

cr_status launch_hqs_redo(cr_frame *f, cr_cloud *const *clouds, uint32_t nclouds,
                          bool splats, const RasterUniforms &u, const RasterTargets &t,
                          const ResolveUniforms &ru, cudaStream_t s) {
    if (nclouds > kRedoMaxClouds || t.packed || !t.redo)
        return cri::fail(CR_ERR_INTERNAL, "launch_hqs_redo: arguments");
    if (nclouds == 0) return CR_OK;  // no sample: the resolve cannot have asked for a re-run
    RedoArgs r;
    r.a = make_args(clouds[0], u, t);
    for (uint32_t i = 0; i < nclouds; ++i) {
        r.clouds[i] = RedoCloud{clouds[i]->d_chunks,   clouds[i]->d_counters, clouds[i]->d_frag_count,
                                clouds[i]->d_frag_xy, clouds[i]->d_frag_zc,
                                make_args(clouds[i], u, t).round_shift};
    }
    r.splats = splats ? 1 : 0;
    r.nclouds = nclouds;
    r.redo = t.redo;
    r.rgba = f->d_rgba[0];
    r.depthf = f->d_depthf;
    r.npix = (uint32_t)f->width * (uint32_t)f->height;
    r.ru = ru;
    CR_CUDA(launch_programmatic(hqs_redo_kernel, dim3(1), dim3(kThreads), 0, s, r));
    CR_CUDA(cudaGetLastError());
    return CR_OK;
}

uint32_t hqs_redo_max_clouds() { return kRedoMaxClouds; }

// A step to a CTA while there are CTAs.
template <int PASS>
cudaError_t launch_point_pass(const RasterArgs &a, cr_context *ctx, cudaStream_t s) {
    int &blocks = ctx->blocks_per_sm_point[PASS];
    if (blocks == 0) blocks = resident_blocks(point_pass<PASS>, 0);
    return launch_programmatic(point_pass<PASS>, dim3(ctx->sm_count * blocks), dim3(kThreads), 0, s,
                               a);
}

// Many points to a pixel meet in their atomics: past this many resident points a
// pixel the depth plane is drawn by depth_kernel, whose screen tiles send a pixel
// to the frame once a record.  Terrains, four views: 100M points at 256 x 256
// 3.88 ms with point_pass and 2.11 so, 20M at 512 x 512 (76 a pixel) 749 and 649
// us, 5M at 256 x 256 (76) 274 and 254; below, 10M at 512 x 512 (38) 426 and 405
// but 16 views of square patches 1094 and 1139, 5M at 512 x 512 (19) 263 and 274,
// 2M at 640 x 512 (6) 172 and 188.
constexpr uint64_t kDensePoints = 64;

cr_status launch_raster_f32(cr_cloud *cloud, RasterPass pass, const RasterUniforms &u,
                            const RasterTargets &t, const float *colors, const float *dldimg,
                            float *grad, cudaStream_t s) {
    if (pass != PASS_DEPTH && pass != PASS_COLOR_F32 && pass != PASS_GRAD)
        return cri::fail(CR_ERR_INTERNAL, "launch_raster_f32: pass");
    RasterArgs a = make_args(cloud, u, t);
    if (!a.ifiles.n) {
        const cr_status st = ensure_device_files(cloud);
        if (st) return st;
    }
    a.fcolors = colors;
    a.dldimg = dldimg;
    a.fgrad = grad;
    cr_context *ctx = cloud->ctx;
    const bool dense = (uint64_t)cloud->resident * cloud->cap.pointsPerBatch >
                       kDensePoints * (uint64_t)u.width * (uint64_t)u.height;
    if (a.radius_zero && !(dense && pass == PASS_DEPTH)) {
        CR_CUDA(pass == PASS_DEPTH       ? launch_point_pass<PASS_DEPTH>(a, ctx, s)
                : pass == PASS_COLOR_F32 ? launch_point_pass<PASS_COLOR_F32>(a, ctx, s)
                                         : launch_point_pass<PASS_GRAD>(a, ctx, s));
        return CR_OK;
    }
    if (pass == PASS_DEPTH) return launch_raster(cloud, pass, u, t, s);
    if (ctx->blocks_per_sm[pass] == 0)
        ctx->blocks_per_sm[pass] = pass == PASS_COLOR_F32
                                       ? blocks_per_sm_for<PASS_COLOR_F32, false>()
                                       : blocks_per_sm_for<PASS_GRAD, false>();
    const int grid = ctx->sm_count * ctx->blocks_per_sm[pass];
    if (pass == PASS_COLOR_F32)
        launch_pass<PASS_COLOR_F32, false>(a, grid, s);
    else
        launch_pass<PASS_GRAD, false>(a, grid, s);
    CR_CUDA(cudaGetLastError());
    return CR_OK;
}

void raster_prepare_views(cr_context *ctx) {
    for (int p : {PASS_DEPTH, PASS_COLOR, PASS_DEPTH_FRAG, PASS_COLOR_FRAG})
        if (ctx->blocks_per_sm_views[p] == 0) ctx->blocks_per_sm_views[p] = raster_blocks_per_sm<true>(p);
    if (ctx->blocks_per_sm_hash_views == 0) {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, color_hash_views_kernel, kThreads, 0) !=
            cudaSuccess)
            n = 1;
        ctx->blocks_per_sm_hash_views = n < 1 ? 1 : n;
    }
}

cr_status launch_raster_views(cr_cloud *cloud, RasterPass pass, const RasterUniforms &u,
                              const RasterTargets &t, const ViewDesc *views, uint32_t nviews,
                              const cr_raster_file *files, uint32_t nfiles,
                              const ChunkRec *chunks, uint32_t chunk_stride,
                              uint32_t *counters, const ViewsFragments *frags, cudaStream_t s) {
    const bool frag_pass = pass == PASS_DEPTH_FRAG || pass == PASS_COLOR_FRAG;
    if (nviews == 0 || nviews > kMaxViews || (frag_pass && !frags) || pass == PASS_NEAREST)
        return cri::fail(CR_ERR_INTERNAL, "batched views: bad pass arguments");
    RasterArgs a = make_args(cloud, u, t);
    a.chunks = chunks;
    a.files = files;
    a.ifiles.n = 0;  // the views' own tables
    a.counters = counters;
    a.views = views;
    a.nviews = nviews;
    a.nfiles = nfiles;
    a.chunk_stride = chunk_stride;
    if (frags) {
        a.frag_xy = frags->xy;
        a.frag_zc = frags->zc;
        a.frag_count = frags->count;
        a.chunk_poff = frags->poff;
        a.frag_cap = frags->cap;
        a.frag_overflow = frags->overflow;
    }
    cr_context *ctx = cloud->ctx;
    if (ctx->blocks_per_sm_views[pass] == 0)
        ctx->blocks_per_sm_views[pass] = raster_blocks_per_sm<true>(pass);
    const int grid = ctx->sm_count * ctx->blocks_per_sm_views[pass];
    switch (pass) {
    case PASS_DEPTH: launch_pass<PASS_DEPTH, true>(a, grid, s); break;
    case PASS_COLOR: launch_pass<PASS_COLOR, true>(a, grid, s); break;
    case PASS_DEPTH_FRAG: launch_pass<PASS_DEPTH_FRAG, true>(a, grid, s); break;
    default: {  // PASS_COLOR_FRAG: fragments, or decode when they overflowed
        if (ctx->blocks_per_sm_hash_views == 0) raster_prepare_views(ctx);
        color_hash_views_kernel<<<ctx->sm_count * ctx->blocks_per_sm_hash_views, kThreads, 0, s>>>(
            a);
        color_views_kernel<<<grid, kThreads, TileCfg<PASS_COLOR>::kBytes, s>>>(a);
        break;
    }
    }
    CR_CUDA(cudaGetLastError());
    return CR_OK;
}
