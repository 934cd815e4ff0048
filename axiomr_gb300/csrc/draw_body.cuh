// Device-side steps of one draw, shared by the per-draw kernels (kernels.cu) and the
// batched persistent kernel (batch.cu): per-vertex transform and shading, per-face clip /
// cull / setup / small-triangle raster, the large-triangle tile raster, and the shading of
// one pixel's winning fragment. The kernels differ only in how work is handed out.
#pragma once
#include <cuda_runtime.h>

#include "raster.cuh"
#include "shade.cuh"

namespace axr {
namespace {

constexpr uint32_t kNoTile = 0xFFFFFFFFu;

// Tag bit of an unclipped triangle that left a shading record (clipped triangles use bits
// 0-3 for 8 + their clip index; an unclipped one has them free). Both shading paths give
// the same bits; the record saves re-deriving the setup, which pays off when the
// triangle's box holds at least kRecMinPixels pixels.
constexpr uint32_t kRecTag = 1u;
constexpr int kRecMinPixels = 16;

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }

// A tile that holds at least one depth key is flagged for the key scan (a plain store:
// every writer stores the same value).
__device__ __forceinline__ void mark_tile(const DevTarget& t, uint32_t tile) { t.tile_flag[tile] = 1u; }

__device__ __forceinline__ uint32_t tile_of(const DevTarget& t, int px, int py) {
    return (uint32_t)(py >> 4) * (uint32_t)t.tiles_x + (uint32_t)(px >> 4);
}

// Visibility write of one covered pixel (no return value used: compiles to a reduction).
// Returns whether a key was written.
__device__ __forceinline__ bool write_key_at(unsigned long long* key, float z, uint32_t tag) {
    if (!(z < __int_as_float(0x7f800000))) return false;  // +inf and NaN never pass early-Z
    atomicMin(key, make_key(z, tag));
    return true;
}

__device__ __forceinline__ bool write_key(const DevTarget& t, int px, int py, float z, uint32_t tag) {
    return write_key_at(&t.key[(uint32_t)py * (uint32_t)t.width + (uint32_t)px], z, tag);
}

struct GeomStats {
    uint32_t tris, frags, large, tested;
};

// Rasterise a small triangle's pixel box in this thread; returns whether any key was
// written. Walks the box the way the reference's tile raster does: per 16-pixel tile
// column and row, the row start (a*(sx+0.5) + b*(py+0.5)) + c and its 8-pixel step are
// computed once, then each pixel adds a*lane (eval_pixel gives the same bits per pixel).
__device__ __forceinline__ bool raster_box(const DevTarget& t, const Edges& e, uint32_t tag, GeomStats& st) {
    bool wrote = false;
    for (int tx = e.x_lo >> 4; tx <= (e.x_hi - 1) >> 4; ++tx) {
        const int sx = max(tx * kTile, e.x_lo);
        const int ex = min((tx + 1) * kTile, e.x_hi);
        const float fsx = fadd((float)sx, 0.5f);
        float as[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) as[k] = fmul(e.a[k], fsx);
        for (int py = e.y_lo; py < e.y_hi; ++py) {
            const float fpy = fadd((float)py, 0.5f);
            float r0[3], r8[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                r0[k] = fadd(fadd(as[k], fmul(e.b[k], fpy)), e.c[k]);
                r8[k] = fadd(r0[k], fmul(e.a[k], 8.0f));
            }
            st.tested += (uint32_t)(ex - sx);
            for (int px = sx; px < ex; ++px) {
                const int i = px - sx;
                const float lane = (float)(i & 7);
                float cov[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) cov[k] = fadd(i >= 8 ? r8[k] : r0[k], fmul(e.a[k], lane));
                if (cov[0] >= 0.f && cov[1] >= 0.f && cov[2] >= 0.f) {
                    ++st.frags;
                    const float al = fmul(cov[0], e.inv_area), be = fmul(cov[1], e.inv_area),
                                ga = fmul(cov[2], e.inv_area);
                    const float z = fadd(fadd(fmul(e.z[0], al), fmul(e.z[1], be)), fmul(e.z[2], ga));
                    wrote |= write_key(t, px, py, z, tag);
                }
            }
        }
    }
    return wrote;
}

// The same out of line, for the rare paths.
__device__ __noinline__ bool raster_box_call(const DevTarget& t, const Edges& e, uint32_t tag, GeomStats& st) {
    return raster_box(t, e, tag, st);
}

__device__ __forceinline__ uint32_t tiles_of(const Edges& e, uint32_t& ntx) {
    int tx0 = e.x_lo >> 4, tx1 = (e.x_hi - 1) >> 4;
    int ty0 = e.y_lo >> 4, ty1 = (e.y_hi - 1) >> 4;
    ntx = (uint32_t)(tx1 - tx0 + 1);
    return ntx * (uint32_t)(ty1 - ty0 + 1);
}

__device__ void mark_box(const DevTarget& t, const Edges& e) {
    for (int ty = e.y_lo >> 4; ty <= (e.y_hi - 1) >> 4; ++ty)
        for (int tx = e.x_lo >> 4; tx <= (e.x_hi - 1) >> 4; ++tx)
            mark_tile(t, (uint32_t)ty * (uint32_t)t.tiles_x + (uint32_t)tx);
}

__device__ __forceinline__ void store_large(LargeTri* dst, const Edges& e, uint32_t tag) {
    float4* d = reinterpret_cast<float4*>(dst);
    d[0] = make_float4(e.a[0], e.b[0], e.c[0], e.a[1]);
    d[1] = make_float4(e.b[1], e.c[1], e.a[2], e.b[2]);
    d[2] = make_float4(e.c[2], e.inv_area, e.z[0], e.z[1]);
    uint32_t xs = (uint32_t)e.x_lo | ((uint32_t)e.x_hi << 16);
    uint32_t ys = (uint32_t)e.y_lo | ((uint32_t)e.y_hi << 16);
    d[3] = make_float4(e.z[2], __uint_as_float(tag), __uint_as_float(xs), __uint_as_float(ys));
}

__device__ __forceinline__ void load_large(const LargeTri* src, Edges& e, uint32_t& tag) {
    const float4* s = reinterpret_cast<const float4*>(src);
    float4 v0 = s[0], v1 = s[1], v2 = s[2], v3 = s[3];
    e.a[0] = v0.x; e.b[0] = v0.y; e.c[0] = v0.z; e.a[1] = v0.w;
    e.b[1] = v1.x; e.c[1] = v1.y; e.a[2] = v1.z; e.b[2] = v1.w;
    e.c[2] = v2.x; e.inv_area = v2.y; e.z[0] = v2.z; e.z[1] = v2.w;
    e.z[2] = v3.x;
    tag = __float_as_uint(v3.y);
    uint32_t xs = __float_as_uint(v3.z), ys = __float_as_uint(v3.w);
    e.x_lo = (int)(xs & 0xFFFFu); e.x_hi = (int)(xs >> 16);
    e.y_lo = (int)(ys & 0xFFFFu); e.y_hi = (int)(ys >> 16);
}

// Raster record (kRasterRec float4, see device_types.h): edges, 1/area, depths, pixel range
// and one extra word (material or tag).
__device__ __forceinline__ void store_raster(float4* r, const Edges& e, uint32_t word) {
    r[0] = make_float4(e.a[0], e.b[0], e.c[0], e.a[1]);
    r[1] = make_float4(e.b[1], e.c[1], e.a[2], e.b[2]);
    r[2] = make_float4(e.c[2], e.inv_area, e.z[0], e.z[1]);
    const uint32_t xs = (uint32_t)e.x_lo | ((uint32_t)e.x_hi << 16);
    const uint32_t ys = (uint32_t)e.y_lo | ((uint32_t)e.y_hi << 16);
    r[3] = make_float4(e.z[2], __uint_as_float(xs), __uint_as_float(ys), __uint_as_float(word));
}

__device__ __forceinline__ uint32_t unpack_raster(const float4 r0, const float4 r1, const float4 r2, const float4 r3,
                                                  Edges& e) {
    e.a[0] = r0.x; e.b[0] = r0.y; e.c[0] = r0.z; e.a[1] = r0.w;
    e.b[1] = r1.x; e.c[1] = r1.y; e.a[2] = r1.z; e.b[2] = r1.w;
    e.c[2] = r2.x; e.inv_area = r2.y; e.z[0] = r2.z; e.z[1] = r2.w;
    e.z[2] = r3.x;
    const uint32_t xs = __float_as_uint(r3.y), ys = __float_as_uint(r3.z);
    e.x_lo = (int)(xs & 0xFFFFu); e.x_hi = (int)(xs >> 16);
    e.y_lo = (int)(ys & 0xFFFFu); e.y_hi = (int)(ys >> 16);
    return __float_as_uint(r3.w);
}

__device__ __forceinline__ void store_record(const DrawParams& p, uint32_t ordinal, const Edges& e, uint32_t material,
                                             const uint3& f) {
    float4* r = p.scratch.rec + (size_t)kRecFloat4 * ordinal;
    store_raster(r, e, material);
    r[4] = make_float4(__uint_as_float(f.x), __uint_as_float(f.y), __uint_as_float(f.z), 0.0f);
}

// kCoherent: the record was written earlier in the same launch (plain loads).
template <bool kCoherent>
__device__ __forceinline__ uint32_t load_record(const DrawParams& p, uint32_t ordinal, Edges& e, uint3& f) {
    const float4* r = p.scratch.rec + (size_t)kRecFloat4 * ordinal;
    const float4 r0 = ld_cached<kCoherent>(r), r1 = ld_cached<kCoherent>(r + 1), r2 = ld_cached<kCoherent>(r + 2);
    const float4 r3 = ld_cached<kCoherent>(r + 3), r4 = ld_cached<kCoherent>(r + 4);
    const uint32_t material = unpack_raster(r0, r1, r2, r3, e);
    f = make_uint3(__float_as_uint(r4.x), __float_as_uint(r4.y), __float_as_uint(r4.z));
    return material;
}

// A box that goes to the large-triangle pass: its setup record and one item per 16x16 tile
// (or, with the lists full, its pixels in this thread). Unclipped triangles leave their
// shading record at the caller.
__device__ __forceinline__ void emit_large(const DrawParams& p, const Edges& e, uint32_t tag, GeomStats& st) {
    DevCounters* c = p.scratch.counters;
    uint32_t ntx;
    const uint32_t nt = tiles_of(e, ntx);
    const uint32_t slot = atomicAdd(&c->large_count, 1u);
    const uint32_t base = atomicAdd(&c->item_count, nt);
    const uint32_t icap = p.scratch.item_cap;
    if (slot < p.scratch.large_cap && base + nt <= icap && base + nt > base) {
        store_large(&p.scratch.large[slot], e, tag);
        if (p.scratch.large_draw) p.scratch.large_draw[slot] = p.draw;
        for (uint32_t k = 0; k < nt; ++k) p.scratch.items[base + k] = LargeItem{slot, k};
        ++st.large;
    } else {
        // lists full: mark the reserved items empty and rasterise the triangle here
        for (uint32_t k = base; k < icap && k - base < nt; ++k) p.scratch.items[k] = LargeItem{kNoItem, 0u};
        GeomStats here = {0, 0, 0, 0};
        const Edges copy = e;  // for the call: e itself stays in registers
        if (raster_box_call(p.target, copy, tag, here)) mark_box(p.target, copy);
        st.frags += here.frags;
        st.tested += here.tested;
    }
}

// IShader::vertex of vertex i plus its screen position, NDC depth and clip-plane masks
// (the per-vertex part of the reference's Triangle ctor, src/tiled_pipeline.cpp:53-72).
template <int S>
__device__ __forceinline__ void vertex_one(const DrawParams& p, uint32_t i) {
    constexpr int A = ShaderAttrs<S>::mask;
    CVFull v = load_vertex<A>(p.mesh, i);
    f4 clip = mat4_mul(p.u.mvp, v.pos.x, v.pos.y, v.pos.z, 1.0f);
    f3 sc = screen_vertex(clip, (float)p.target.width, (float)p.target.height);
    p.scratch.vscreen[i] = make_float4(sc.x, sc.y, sc.z, __uint_as_float(plane_masks(clip)));
    pack_vsout<S>(vertex_shader<S>(p.u, v), &p.scratch.vattr[(size_t)VAttr<S>::n * i]);
}

// A face whose vertices straddle the clip volume: the clipper's output triangles, each culled,
// set up and, with its clip index in the tag, rasterised here (boxes of at most
// kClippedThreadPixels: such faces are few and far between) or sent to the large-triangle pass.
constexpr int kClippedThreadPixels = 8;

__device__ __noinline__ void geometry_clipped(const DrawParams& p, uint32_t o, GeomStats& st) {
    const uint3 f = load_face(p.mesh, face_of(p.mesh, o).face);
    CVClip a[kMaxClipVerts], b[kMaxClipVerts];
    a[0].clip = load_clip(p.mesh, p.u.mvp, f.x);
    a[1].clip = load_clip(p.mesh, p.u.mvp, f.y);
    a[2].clip = load_clip(p.mesh, p.u.mvp, f.z);
    CVClip* out;
    const int n = clip_triangle<0>(a, b, &out);
    for (int j = 0; 3 * j + 2 < n; ++j) {
        Screen s;
        screen_setup(out[3 * j].clip, out[3 * j + 1].clip, out[3 * j + 2].clip, p.target.width, p.target.height, s);
        if (is_backface(s)) continue;
        ++st.tris;
        Edges e;
        if (!edge_setup(s, p.target.width, p.target.height, e)) continue;
        const uint32_t tag = (o << 4) | 8u | (uint32_t)j;
        if ((e.x_hi - e.x_lo) * (e.y_hi - e.y_lo) > min(p.small_max_pixels, kClippedThreadPixels))
            emit_large(p, e, tag, st);
        else if (raster_box_call(p.target, e, tag, st))
            mark_box(p.target, e);
    }
}

// Warp-wide end of the geometry step: one mark per distinct single tile in the warp, and
// the statistics. All 32 lanes must call it.
__device__ __forceinline__ void geometry_warp_tail(const DevTarget& t, DevCounters* c, bool stats, const GeomStats& st,
                                                   uint32_t single_tile) {
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, single_tile);
    if (single_tile != kNoTile && (threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1)) mark_tile(t, single_tile);
    if (stats) {
        const unsigned full = 0xFFFFFFFFu;
        uint32_t tr = __reduce_add_sync(full, st.tris), fr = __reduce_add_sync(full, st.frags);
        uint32_t l = __reduce_add_sync(full, st.large), te = __reduce_add_sync(full, st.tested);
        if ((threadIdx.x & 31) == 0) {
            if (tr) atomicAdd(&c->stat_triangles, (unsigned long long)tr);
            if (fr) atomicAdd(&c->stat_fragments, (unsigned long long)fr);
            if (l) atomicAdd(&c->stat_large, (unsigned long long)l);
            if (te) atomicAdd(&c->stat_tested, (unsigned long long)te);
        }
    }
}

// ---- the face phase: setup by face, raster by pixel
//
// Each thread sets up a face and rasterises a box of at most kThreadPixels pixels itself. The
// pixels of larger boxes (up to p.small_max_pixels) are numbered one box after another over
// a group of threads, a warp or the CTA, and the group's threads share these (triangle, pixel)
// pairs evenly. Boxes differ by two orders of magnitude within a warp and about half of a
// closed mesh's faces are culled, so a thread per triangle left 8 to 18 of 32 lanes at work
// (ncu: 8.4 on a 4k-triangle sphere, 8.6 on 200k small triangles, 12.3 on the mixed batch)
// behind the warp's largest box. Bound: issue and the gathers' latency. Frames, before and
// after: 4k-triangle sphere at 512x512 60 to 31 us, 2M-triangle terrain at 1920x1080 109 to
// 103, 200k triangles at 3840x2160 133 to 127, 30 mixed draws in a batch 220 to 192; all pixels
// by pairs instead (no box in its own thread) left the terrain, most of whose boxes hold 2 to 6
// pixels, at 129.
constexpr int kWarpPairs = 8192;  // pairs that the 32 faces of a warp may share: 32 boxes of 256
                                  // pixels; boxes past them go to the large-triangle pass
constexpr int kThreadPixels = 6;  // boxes a thread rasterises itself (at most 8)

template <int kThreads>
struct FaceSmem {
    float4 job[kThreads][5];                         // store_job, 80 bytes: no bank conflicts
    __align__(16) uint32_t start[kThreads / 32 * kWarpPairs / 32]; // bit k: pair k is the first of its box
    uint16_t owner[kThreads / 32 * kWarpPairs / 32]; // the box that holds pair 32 w
    uint32_t warp_sum[kThreads / 32];
};

// Small non-negative integers as floats without the conversion unit (2^23 + v has v in its
// low mantissa bits): v, and v + 1/2 (2^23 - 1/2 is a float), both exact.
__device__ __forceinline__ float small_float(int v) { return __int_as_float(0x4B000000 | v) - 8388608.0f; }
__device__ __forceinline__ float small_centre(int v) { return __int_as_float(0x4B000000 | v) - 8388607.5f; }

__device__ __forceinline__ void store_job(float4* j, const Edges& e, uint32_t tag, uint32_t first) {
    const uint32_t w = (uint32_t)(e.x_hi - e.x_lo);
    j[0] = make_float4(e.a[0], e.b[0], e.c[0], e.a[1]);
    j[1] = make_float4(e.b[1], e.c[1], e.a[2], e.b[2]);
    j[2] = make_float4(e.c[2], e.inv_area, e.z[0], e.z[1]);
    j[3] = make_float4(e.z[2], __uint_as_float((uint32_t)e.x_lo | ((uint32_t)e.y_lo << 16)), __uint_as_float(tag),
                       __uint_as_float(first | (w << 16)));
}

// A box of at most 8 pixels in this thread (the 8-pixel step of eval_pixel never comes up);
// returns whether a key was written.
__device__ __forceinline__ bool raster_tiny(const DevTarget& t, const Edges& e, uint32_t tag, uint32_t npx, GeomStats& st) {
    bool wrote = false;
    int px = e.x_lo, py = e.y_lo;
    st.tested += npx;
    for (uint32_t q = 0; q < npx; ++q) {
        const int sx = max(px & ~(kTile - 1), e.x_lo);
        const float fsx = small_centre(sx), fpy = small_centre(py), lane = small_float(px - sx);
        float cov[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
            cov[k] = fadd(fadd(fadd(fmul(e.a[k], fsx), fmul(e.b[k], fpy)), e.c[k]), fmul(e.a[k], lane));
        if (cov[0] >= 0.f && cov[1] >= 0.f && cov[2] >= 0.f) {
            ++st.frags;
            const float al = fmul(cov[0], e.inv_area), be = fmul(cov[1], e.inv_area), ga = fmul(cov[2], e.inv_area);
            wrote |= write_key(t, px, py, fadd(fadd(fmul(e.z[0], al), fmul(e.z[1], be)), fmul(e.z[2], ga)), tag);
        }
        if (++px == e.x_hi) {
            px = e.x_lo;
            ++py;
        }
    }
    return wrote;
}

// Pair k: coverage and depth of one pixel of the box `j`, in eval_pixel's operations. first
// (below 65536) and w (at most 8192) share a word; the row is the floor of (q + 1/2) / w, q < 8192
// pixels into the box: an approximate reciprocal leaves it off by less than q / w * 2^-22, and no
// exact value is nearer than 1 / (2 w) to an integer, so the truncation is the quotient.
__device__ __forceinline__ void raster_pair(const DevTarget& t, const float4* j, uint32_t k, GeomStats& st) {
    const float4 v0 = j[0], v1 = j[1], v2 = j[2], v3 = j[3];
    const uint32_t xy = __float_as_uint(v3.y), fw = __float_as_uint(v3.w);
    const uint32_t w = fw >> 16, q = k - (fw & 0xFFFFu);
    const uint32_t row = (uint32_t)__float2int_rz(small_centre((int)q) * crcp(small_float((int)w)));
    const int x_lo = (int)(xy & 0xFFFFu);
    const int px = x_lo + (int)(q - row * w), py = (int)((xy >> 16) + row);
    const int sx = max(px & ~(kTile - 1), x_lo), i = px - sx;
    const float fsx = small_centre(sx), fpy = small_centre(py), lane = small_float(i & 7);
    const float a[3] = {v0.x, v0.w, v1.z}, b[3] = {v0.y, v1.x, v1.w}, c[3] = {v0.z, v1.y, v2.x};
    float cov[3];
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        float r = fadd(fadd(fmul(a[n], fsx), fmul(b[n], fpy)), c[n]);
        if (i >= 8) r = fadd(r, fmul(a[n], 8.0f));
        cov[n] = fadd(r, fmul(a[n], lane));
    }
    if (cov[0] >= 0.f && cov[1] >= 0.f && cov[2] >= 0.f) {
        ++st.frags;
        const float al = fmul(cov[0], v2.y), be = fmul(cov[1], v2.y), ga = fmul(cov[2], v2.y);
        write_key(t, px, py, fadd(fadd(fmul(v2.z, al), fmul(v2.w, be)), fmul(v3.x, ga)), __float_as_uint(v3.z));
    }
}

// Checks, vertex-cache gathers, clip classification, cull and setup of the face at draw-order
// position o. One inside the clip volume that faces the camera and has a pixel box is returned
// (true) with its depth-key tag, its shading record stored; `cut`: it straddles the volume (for
// geometry_clipped). kCoherent: the vertex cache was written earlier in the same launch (plain loads).
template <bool kCoherent>
__device__ __forceinline__ bool face_setup(const DrawParams& p, uint32_t o, GeomStats& st, Edges& e, uint32_t& tag,
                                           bool& cut) {
    if (o > kMaxOrdinal) {
        atomicOr(&p.scratch.counters->error, kErrOrdinal);
        return false;
    }
    const FaceRef fr = face_of(p.mesh, o);
    const uint3 f = load_face(p.mesh, fr.face);
    const uint32_t nv = p.mesh.num_vertices;
    if (f.x >= nv || f.y >= nv || f.z >= nv) {
        atomicOr(&p.scratch.counters->error, kErrIndex);
        return false;
    }
    const float4* vs = p.scratch.vscreen;
    const float4 g0 = ld_cached<kCoherent>(&vs[f.x]), g1 = ld_cached<kCoherent>(&vs[f.y]),
                 g2 = ld_cached<kCoherent>(&vs[f.z]);
    const int cls = classify_masks(__float_as_uint(g0.w), __float_as_uint(g1.w), __float_as_uint(g2.w));
    cut = cls < 0;
    if (cls != 3) return false;
    Screen s;
    s.x[0] = g0.x; s.y[0] = g0.y; s.z[0] = g0.z;
    s.x[1] = g1.x; s.y[1] = g1.y; s.z[1] = g1.z;
    s.x[2] = g2.x; s.y[2] = g2.y; s.z[2] = g2.z;
    if (is_backface(s)) return false;
    ++st.tris;
    screen_bbox(s);
    if (!edge_setup(s, p.target.width, p.target.height, e)) return false;
    tag = o << 4;
    if ((e.x_hi - e.x_lo) * (e.y_hi - e.y_lo) >= kRecMinPixels) {
        tag |= kRecTag;
        store_record(p, o, e, fr.material, f);
    }
    return true;
}

// The faces of a CTA, thread t's at draw-order position o (valid: it has one); a group is a
// warp (kWarp) or the CTA. Faces that straddle the clip volume go to scratch.cut (kCutList) or
// through the clipper here. The tiles of a shared box are flagged whether or not a pixel of it turns
// out covered (a flagged tile without keys costs the tile pass its key reads).
template <bool kCoherent, bool kCutList, int kThreads, bool kWarp>
__device__ __forceinline__ void face_group(const DrawParams& p, uint32_t o, bool valid, DevCounters* c, bool stats,
                                           FaceSmem<kThreads>& sm) {
    constexpr int kGroupWarps = kWarp ? 1 : kThreads / 32;
    constexpr uint32_t kCap = kGroupWarps * kWarpPairs;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gw = kWarp ? 0 : warp, gt = kWarp ? lane : tid;  // this warp and thread in the group
    const uint32_t table = kWarp ? (uint32_t)warp * (kWarpPairs / 32) : 0u;
    float4(*job)[5] = sm.job + (kWarp ? 32 * warp : 0);
    uint32_t* start = sm.start + table;
    uint16_t* owner = sm.owner + table;
    GeomStats st = {0, 0, 0, 0};
    uint32_t single_tile = kNoTile, tag = 0;
    Edges e;
    bool cut = false;
    bool has = valid && face_setup<kCoherent>(p, o, st, e, tag, cut);
    const uint32_t npx = has ? (uint32_t)(e.x_hi - e.x_lo) * (uint32_t)(e.y_hi - e.y_lo) : 0u;
    bool large = npx > (uint32_t)max(p.small_max_pixels, kThreadPixels);
    has = has && !large;
    if (has && npx <= (uint32_t)kThreadPixels) {
        has = false;
        if (raster_tiny(p.target, e, tag, npx, st)) {
            uint32_t ntx;
            if (tiles_of(e, ntx) == 1u) single_tile = tile_of(p.target, e.x_lo, e.y_lo);
            else mark_box(p.target, e);
        }
    }
    if (!kWarp || __any_sync(0xFFFFFFFFu, has)) {
        for (int k = gt; k < (int)kCap / 128; k += 32 * kGroupWarps)
            reinterpret_cast<uint4*>(start)[k] = make_uint4(0u, 0u, 0u, 0u);
        // (boxes, pairs) before this thread's: boxes above bit 22, pairs below. A warp takes the
        // boxes that its share of the tables holds, in face order.
        const uint32_t mine = has ? (1u << 22) | min(npx, (uint32_t)kWarpPairs + 1u) : 0u;
        uint32_t incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += v;
        }
        const unsigned past = __ballot_sync(0xFFFFFFFFu, (incl & 0x3FFFFFu) > (uint32_t)kWarpPairs);
        uint32_t before = incl - mine;
        uint32_t total = __shfl_sync(0xFFFFFFFFu, past ? before : incl, past ? __ffs(past) - 1 : 31);
        if (past >> lane & 1u) {
            large = large || has;
            has = false;
        }
        if (!kWarp) {
            if (lane == 31) sm.warp_sum[warp] = total;
            __syncthreads();
            total = 0;
#pragma unroll
            for (int w = 0; w < kGroupWarps; ++w) {
                const uint32_t v = sm.warp_sum[w];
                if (w < warp) before += v;
                total += v;
            }
        } else {
            __syncwarp();  // the zeroed table
        }
        const uint32_t pairs = total & 0x3FFFFFu;
        if (has) {
            const uint32_t at = before & 0x3FFFFFu, rank = before >> 22;
            store_job(job[rank], e, tag, at);
            atomicOr(&start[at >> 5], 1u << (at & 31u));
            for (uint32_t w = (at + 31u) >> 5; (w << 5) < at + npx; ++w) owner[w] = (uint16_t)rank;
            uint32_t ntx;
            if (tiles_of(e, ntx) == 1u) single_tile = tile_of(p.target, e.x_lo, e.y_lo);
            else mark_box(p.target, e);
        }
        if (kWarp) __syncwarp();
        else __syncthreads();
#pragma unroll 2
        for (uint32_t w = (uint32_t)gw; (w << 5) < pairs; w += kGroupWarps) {
            const uint32_t k = (w << 5) + (uint32_t)lane;
            const uint32_t rank = owner[w] + (uint32_t)__popc(start[w] & ~1u & ((2u << lane) - 1u));
            if (k < pairs) {
                ++st.tested;
                raster_pair(p.target, job[rank], k, st);
            }
        }
    }
    if (large) emit_large(p, e, tag, st);
    if (kCutList) {  // to the clip kernel
        const unsigned m = __ballot_sync(0xFFFFFFFFu, cut);
        if (m) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&c->cut_count, (uint32_t)__popc(m));
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
            if (cut) p.scratch.cut[at + (uint32_t)__popc(m & ((1u << lane) - 1u))] = o;
        }
    } else if (cut) {  // last: the clipper is a long chain, and the group would wait for it
        GeomStats clipped = {0, 0, 0, 0};  // its own: no pointer to st leaves this function
        geometry_clipped(p, o, clipped);
        st.tris += clipped.tris;
        st.frags += clipped.frags;
        st.large += clipped.large;
        st.tested += clipped.tested;
    }
    geometry_warp_tail(p.target, c, stats, st, single_tile);
}

// The CTA's faces from draw-order position `first`, one to each of its first threads. Pairs are
// shared by the CTA, or (kSolo, the per-draw path, with a face for every thread) by each warp: one draw of
// many faces, mostly tiny boxes, does without the two barriers (2M-triangle terrain 102 against
// 133 us a frame), while a batch's draws of all densities gain more from the CTA's balance
// (512 mixed draws, boxes up to 128 pixels: 5.77 against 5.84 ms with their PNG files).
template <bool kCoherent, bool kSolo, int kThreads>
__device__ __forceinline__ void face_cta(const DrawParams& p, uint32_t first, uint32_t faces_of_cta, DevCounters* c,
                                         bool stats, FaceSmem<kThreads>& sm) {
    const uint32_t o = first + threadIdx.x;
    const bool valid = threadIdx.x < faces_of_cta && o < p.mesh.num_drawn;
    if (kSolo && faces_of_cta == (uint32_t)kThreads)
        face_group<kCoherent, kSolo, kThreads, true>(p, o, valid, c, stats, sm);
    else
        face_group<kCoherent, kSolo, kThreads, false>(p, o, valid, c, stats, sm);
}

// Whether no pixel of 16x16 tile (tx, ty) inside the triangle's box can test covered.
// Each edge function is linear, so over the tile's pixel centres it peaks at a corner of
// their rectangle. eval_pixel's float evaluation of an edge at a centre is within a few
// units of 2^-24 * M of its exact value, M = |a|(|x|+16) + |b||y| + |c| bounding the
// magnitudes of its terms, and the corner values here are within 3 such units; if the
// corner maximum of some edge is below -64 * 2^-24 * M, every evaluated value of that edge
// in the tile is negative, so the tile holds no covered pixel and is skipped.
__device__ __forceinline__ bool tile_outside(const Edges& e, int tx, int ty) {
    const float x0 = (float)max(tx * kTile, e.x_lo) + 0.5f, x1 = (float)min(tx * kTile + kTile, e.x_hi) - 0.5f;
    const float y0 = (float)max(ty * kTile, e.y_lo) + 0.5f, y1 = (float)min(ty * kTile + kTile, e.y_hi) - 0.5f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float a = e.a[k], b = e.b[k], c = e.c[k];
        const float ex = a >= 0.f ? a * x1 : a * x0;  // the larger of a*x0, a*x1
        const float ey = b >= 0.f ? b * y1 : b * y0;
        const float emax = (ex + ey) + c;
        const float m = fabsf(a) * (fabsf(x1) + 16.0f) + fabsf(b) * fabsf(y1) + fabsf(c);
        if (emax < -64.0f * 5.9604645e-8f * m) return true;
    }
    return false;
}

// One large-triangle work item: the warp evaluates the 256 pixels of tile `item_tile` of
// the triangle's tile box, 8 per lane, and flags the tile if a key was written. Bound: issue. A
// lane's rows inside the box are a mask found once and what its column decides (row start, step and
// lane terms of eval_pixel) is computed once; with both per pixel: 1365x767 close-up 93.8 us a
// frame, 91.0 now; 512 draws with their PNG files 4.39 and 4.35 ms. Two rows in packed
// f32x2 arithmetic is not open: ptxas contracts a packed product and sum into one rounding, also
// under --fmad=false.
__device__ __forceinline__ void large_tile(const DevTarget& t, const Edges& e, uint32_t tag, uint32_t item_tile,
                                           uint32_t& frags, uint32_t& tested) {
    const int lane = threadIdx.x & 31;
    uint32_t ntx;
    tiles_of(e, ntx);
    const int tx = (e.x_lo >> 4) + (int)(item_tile % ntx);
    const int ty = (e.y_lo >> 4) + (int)(item_tile / ntx);
    if (tile_outside(e, tx, ty)) return;
    // the lane's pixels: column px, rows base + 2 r; those inside the box are bits of `rows`
    const int px = tx * kTile + (lane & 15), base = ty * kTile + (lane >> 4);
    uint32_t rows = 0u;
    if (px >= e.x_lo && px < e.x_hi)
        rows = ((1u << min((e.y_hi - base + 1) >> 1, 8)) - 1u) & (0xFFu << (max(e.y_lo - base + 1, 0) >> 1));
    tested += (uint32_t)__popc(rows);
    // eval_pixel, less what the rows share
    const int sx = max(tx * kTile, e.x_lo), i = px - sx;
    const float fsx = small_centre(sx), fl = (float)(i & 7), fpy = small_centre(base);
    const bool step = i >= 8;
    float s[3], l[3], t8[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s[k] = fmul(e.a[k], fsx);
        l[k] = fmul(e.a[k], fl);
        t8[k] = fmul(e.a[k], 8.0f);
    }
    unsigned long long* key = t.key + (uint32_t)base * (uint32_t)t.width + (uint32_t)px;
    bool wrote = false;
#pragma unroll
    for (int r = 0; r < 8; ++r, key += 2 * t.width) {
        if (!(rows >> r & 1u)) continue;
        const float y = fadd(fpy, (float)(2 * r));
        float cov[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            cov[k] = fadd(fadd(s[k], fmul(e.b[k], y)), e.c[k]);
            if (step) cov[k] = fadd(cov[k], t8[k]);
            cov[k] = fadd(cov[k], l[k]);
        }
        if (cov[0] >= 0.f && cov[1] >= 0.f && cov[2] >= 0.f) {
            ++frags;
            const float al = fmul(cov[0], e.inv_area), be = fmul(cov[1], e.inv_area), ga = fmul(cov[2], e.inv_area);
            wrote |= write_key_at(key, fadd(fadd(fmul(e.z[0], al), fmul(e.z[1], be)), fmul(e.z[2], ga)), tag);
        }
    }
    if (__any_sync(0xFFFFFFFFu, wrote) && lane == 0) mark_tile(t, (uint32_t)ty * (uint32_t)t.tiles_x + (uint32_t)tx);
}

// Winner inputs of an unclipped tag without a record: screen positions from the vertex
// cache and the cached vertex-shader outputs.
template <int S, bool kCoherent = false>
__device__ __forceinline__ uint32_t winner_inputs(const DrawParams& p, uint32_t tag, Screen& s, VSOut* vo) {
    const FaceRef fr = face_of(p.mesh, tag >> 4);
    const uint3 f = load_face(p.mesh, fr.face);
    const uint32_t vi[3] = {f.x, f.y, f.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 g = ld_cached<kCoherent>(&p.scratch.vscreen[vi[k]]);
        s.x[k] = g.x;
        s.y[k] = g.y;
        s.z[k] = g.z;
        vo[k] = unpack_vsout<S, kCoherent>(&p.scratch.vattr[(size_t)VAttr<S>::n * vi[k]]);
    }
    screen_bbox(s);
    return fr.material;
}

// Winner inputs of an unclipped tag: its shading record and the cached vertex-shader
// outputs of its three vertices. Returns the material.
template <int S, bool kCoherent = false>
__device__ __forceinline__ uint32_t record_inputs(const DrawParams& p, uint32_t tag, Edges& e, VSOut* vo) {
    uint3 f;
    const uint32_t material = load_record<kCoherent>(p, tag >> 4, e, f);
    const uint32_t vi[3] = {f.x, f.y, f.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) vo[k] = unpack_vsout<S, kCoherent>(&p.scratch.vattr[(size_t)VAttr<S>::n * vi[k]]);
    return material;
}

// Winner inputs of a clipped tag: the clipper re-run on the face's raw vertex attributes
// (the geometry stage's clip, now carrying attributes; src/pipeline.cpp:243-272), output
// triangle j of the tag. Returns false if the tag names no output triangle.
template <int S>
__device__ bool clipped_inputs(const DrawParams& p, uint32_t tag, Screen& s, VSOut* vo, uint32_t& material) {
    constexpr int A = ShaderAttrs<S>::mask;
    const FaceRef fr = face_of(p.mesh, tag >> 4);
    const uint3 f = load_face(p.mesh, fr.face);
    CVFull a[kMaxClipVerts], b[kMaxClipVerts];
    a[0] = load_vertex<A>(p.mesh, f.x);
    a[1] = load_vertex<A>(p.mesh, f.y);
    a[2] = load_vertex<A>(p.mesh, f.z);
#pragma unroll
    for (int k = 0; k < 3; ++k) a[k].clip = mat4_mul(p.u.mvp, a[k].pos.x, a[k].pos.y, a[k].pos.z, 1.0f);
    CVFull* out;
    const int cnt = clip_triangle<A>(a, b, &out);
    const int j = (int)(tag & 7u);
    if (3 * j + 2 >= cnt) return false;  // cannot happen: the tag came from this clip
    screen_setup(out[3 * j].clip, out[3 * j + 1].clip, out[3 * j + 2].clip, p.target.width, p.target.height, s);
    for (int k = 0; k < 3; ++k) vo[k] = vertex_shader<S>(p.u, out[3 * j + k]);
    material = fr.material;
    return true;
}

// The clip pass of a listed face: geometry_clipped with the attributes carried along, and each
// output triangle's setup and vertex-shader outputs stored for the tile pass, which would
// otherwise re-run the clipper for every pixel it wins (a chain of 10 us that a CTA waits for).
template <int S>
__device__ void clip_listed(const DrawParams& p, uint32_t o, GeomStats& st) {
    constexpr int A = ShaderAttrs<S>::mask;
    constexpr uint32_t kStride = 4 + 3 * VAttr<S>::n;
    static_assert(kStride <= (uint32_t)kClipRecFloat4, "clipped-triangle record size");
    const FaceRef fr = face_of(p.mesh, o);
    const uint3 f = load_face(p.mesh, fr.face);
    CVFull a[kMaxClipVerts], b[kMaxClipVerts];
    a[0] = load_vertex<A>(p.mesh, f.x);
    a[1] = load_vertex<A>(p.mesh, f.y);
    a[2] = load_vertex<A>(p.mesh, f.z);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 q = __ldg(&p.mesh.pos[k == 0 ? f.x : k == 1 ? f.y : f.z]);
        a[k].clip = mat4_mul(p.u.mvp, q.x, q.y, q.z, 1.0f);
    }
    CVFull* out;
    const int n = clip_triangle<A>(a, b, &out);
    const uint32_t nt = (uint32_t)n / 3u;
    uint32_t base = nt ? atomicAdd(&p.scratch.counters->crec_count, nt) : 0u;
    if (base + nt > p.scratch.crec_cap) base = kNoClipRec;
    p.scratch.rec[(size_t)kRecFloat4 * o] = make_float4(__uint_as_float(base), 0.f, 0.f, 0.f);
    for (uint32_t j = 0; j < nt; ++j) {
        const CVFull* v = out + 3 * j;
        Screen s;
        screen_setup(v[0].clip, v[1].clip, v[2].clip, p.target.width, p.target.height, s);
        if (is_backface(s)) continue;
        ++st.tris;
        Edges e;
        if (!edge_setup(s, p.target.width, p.target.height, e)) continue;
        if (base != kNoClipRec) {
            float4* r = p.scratch.crec + (size_t)kStride * (base + j);
            store_raster(r, e, fr.material);
            for (int k = 0; k < 3; ++k) pack_vsout<S>(vertex_shader<S>(p.u, v[k]), r + 4 + VAttr<S>::n * k);
        }
        const uint32_t tag = (o << 4) | 8u | j;
        if ((e.x_hi - e.x_lo) * (e.y_hi - e.y_lo) > min(p.small_max_pixels, kClippedThreadPixels))
            emit_large(p, e, tag, st);
        else if (raster_box_call(p.target, e, tag, st))
            mark_box(p.target, e);
    }
}

// Fragment of the winner at (px, py): exact barycentrics and depth, the merge test against
// `old_depth` (tile depth < framebuffer depth, strict; src/tiled_pipeline.cpp:1171-1174)
// and the shader. Returns whether the fragment is written.
template <int S>
__device__ __forceinline__ bool shade_pixel(const DrawParams& p, int px, int py, uint32_t material, Screen& s,
                                            const VSOut* vo, float old_depth, uint32_t& bgra, float& z) {
    Edges e;
    if (!edge_setup(s, p.target.width, p.target.height, e)) return false;
    const PixelEval r = eval_pixel(e, px, py);
    if (!(r.z < old_depth)) return false;
    const f4 col = fragment_shader<S>(p.u, p.mesh.materials[material], mk3(r.alpha, r.beta, r.gamma), vo);
    bgra = pack_bgra(col);
    z = r.z;
    return true;
}

}  // namespace
}  // namespace axr

namespace axr {
namespace {

// Fragment of the unclipped winner `tag` at (px, py): the setup from its shading record
// when it has one, else re-derived from the face; then exact barycentrics and depth, the
// strict merge test against `old_depth` and the shader. Returns whether it is written.
// Fragment at (px, py) of a triangle given its setup, vertex-shader outputs and material:
// exact barycentrics and depth, the strict merge test against `old_depth` and the shader.
template <int S>
__device__ __forceinline__ bool shade_from(const DrawParams& p, const Edges& e, const VSOut* vo, uint32_t material,
                                           int px, int py, float old_depth, uint32_t& bgra, float& z) {
    const PixelEval r = eval_pixel(e, px, py);
    if (!(r.z < old_depth)) return false;
    const f4 col = fragment_shader<S>(p.u, p.mesh.materials[material], mk3(r.alpha, r.beta, r.gamma), vo);
    bgra = pack_bgra(col);
    z = r.z;
    return true;
}

template <int S, bool kCoherent = false>
__device__ __forceinline__ bool shade_unclipped(const DrawParams& p, uint32_t tag, int px, int py, float old_depth,
                                                uint32_t& bgra, float& z) {
    VSOut vo[3];
    Edges e;
    uint32_t material;
    if (tag & kRecTag) {
        material = record_inputs<S, kCoherent>(p, tag, e, vo);
    } else {
        Screen s;
        material = winner_inputs<S, kCoherent>(p, tag, s, vo);
        if (!edge_setup(s, p.target.width, p.target.height, e)) return false;
    }
    return shade_from<S>(p, e, vo, material, px, py, old_depth, bgra, z);
}

// Winner that came out of the clipper: its inputs from the clipper re-run, then the
// fragment; kept out of line so that the clipper's state does not raise the register count
// of the shading loops that call it.
template <int S>
__device__ __noinline__ bool shade_clipped_px(const DrawParams& p, uint32_t tag, int px, int py, float old_depth,
                                              uint32_t* bgra, float* z) {
    Screen s;
    VSOut vo[3];
    uint32_t material;
    return clipped_inputs<S>(p, tag, s, vo, material) && shade_pixel<S>(p, px, py, material, s, vo, old_depth, *bgra, *z);
}

// Winner of the per-draw tile pass, clipped or not.
template <int S, bool kClip>
__device__ __forceinline__ bool shade_any(const DrawParams& p, uint32_t tag, int px, int py, float old_depth,
                                          uint32_t& bgra, float& z) {
    VSOut vo[3];
    Edges e;
    uint32_t material;
    if (kClip && (tag & 8u)) {
        const uint32_t base = __float_as_uint(p.scratch.rec[(size_t)kRecFloat4 * (tag >> 4)].x);
        if (base == kNoClipRec) {
            uint32_t c = 0u;
            float d = 0.0f;
            if (!shade_clipped_px<S>(p, tag, px, py, old_depth, &c, &d)) return false;
            bgra = c;
            z = d;
            return true;
        }
        const float4* r = p.scratch.crec + (size_t)(4 + 3 * VAttr<S>::n) * (base + (tag & 7u));
        material = unpack_raster(r[0], r[1], r[2], r[3], e);
#pragma unroll
        for (int k = 0; k < 3; ++k) vo[k] = unpack_vsout<S, true>(r + 4 + VAttr<S>::n * k);
    } else if (tag & kRecTag) {
        material = record_inputs<S, true>(p, tag, e, vo);
    } else {
        Screen s;
        material = winner_inputs<S, true>(p, tag, s, vo);
        if (!edge_setup(s, p.target.width, p.target.height, e)) return false;
    }
    return shade_from<S>(p, e, vo, material, px, py, old_depth, bgra, z);
}

}  // namespace
}  // namespace axr
