// Draw kernels for sm_103a.
//
// A draw is four launches on one stream (one more when faces may be clipped, and one in a larger
// frame), each set up while the one before drains (pdl.cuh):
//   vertex_kernel    one thread per vertex: clip position (mvp * pos), screen position and
//                    NDC depth (the per-vertex part of the reference's Triangle ctor,
//                    src/tiled_pipeline.cpp:53-72), clip-plane masks, and the shader's
//                    vertex outputs (IShader::vertex, include/shaders/shaders.hpp). The
//                    reference recomputes these for every face a vertex belongs to (clip
//                    stage) and every tile a triangle touches (processTile, cpp:407-409);
//                    they depend only on the vertex, so one evaluation gives the same bits.
//                    Its first thread zeroes the draw's counters.
//   geometry_kernel  one thread per face in draw order: clip classification from the vertex
//                    masks, backface cull and edge setup (cpp:195-236, 436-487), then the pixels
//                    of the smaller boxes (face_group, draw_body.cuh); larger boxes get one
//                    setup record and one work item per 16x16 tile, faces that straddle the
//                    clip volume go to a list
//   clip_kernel      one thread per listed face: the exact clipper, its output triangles
//                    rasterised or queued as above; not launched when the mesh's bounding sphere
//                    shows that no face can be clipped (never left out of a recorded draw)
//   large_kernel     warps take tile work items and evaluate 256 pixels each, 8 per lane
//   tile_kernel      a CTA per flagged tile: its covered pixels (non-empty depth keys) are
//                    listed and their keys reset, then one thread per covered pixel re-derives
//                    the winner from its key, shades it once and merges it into the framebuffer
//                    with the reference's strict less-than test. A larger frame (scan_pass) does
//                    it in two kernels, scan_kernel listing the covered pixels of all tiles in
//                    memory and shade_kernel shading them
// Visibility is order independent: every covered pixel does a fire-and-forget 64-bit
// atomicMin of (depth, draw-order position), so the surviving key is the reference's
// early-Z winner (minimum depth, earliest triangle on ties) whatever order the threads
// run in. Only the winning fragment is shaded; the reference shades every fragment that
// passes its early test at the time, with the same final colour.
#include <cuda_runtime.h>

#include <cstddef>
#include <cstring>

#include "batch_types.h"
#include "draw_body.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace axr {

namespace {

constexpr int kBlock = 256;
constexpr int kClipBlock = 64;

// Resident 128-thread CTAs per SM the geometry kernel is compiled for (register budget
// 65536 / (128 * n)): 56 registers, the fewest without spills. Its gathers' latency is the bound (2M-triangle
// terrain, us a frame: 7 CTAs 92.1, 8 88.4, 9 86.2, 10 98).
#ifndef AXR_GEOMETRY_MIN_BLOCKS
#define AXR_GEOMETRY_MIN_BLOCKS 9
#endif
// A CTA brings the face indices of the CTA this many further on into L2, so that of the two dependent
// loads before a face's setup the first no longer comes from HBM (the terrain 89.8 to 88.4 us; 1216 and
// 4864 CTAs ahead 88.5 and 89.1).
constexpr uint32_t kIndexAhead = 304;


template <int S>
__global__ void __launch_bounds__(kBlock) vertex_kernel(const __grid_constant__ DrawParams p) {
    pdl_wait();
    pdl_release();
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i == 0) {
        p.scratch.counters->large_count = 0u;
        p.scratch.counters->item_count = 0u;
        p.scratch.counters->cut_count = 0u;
        p.scratch.counters->crec_count = 0u;
        p.scratch.counters->shade_count = 0u;
    }
    if (i < p.mesh.num_vertices) vertex_one<S>(p, i);
}

__global__ void __launch_bounds__(kPhasedFaceUnit, AXR_GEOMETRY_MIN_BLOCKS)
    geometry_kernel(const __grid_constant__ DrawParams p, uint32_t faces_per_cta) {
    __shared__ __align__(16) FaceSmem<(int)kPhasedFaceUnit> sm;
    // 32 words, a line, per thread; with several material groups another CTA's faces may be meant
    const size_t ahead = 3ull * ((size_t)(blockIdx.x + kIndexAhead) * faces_per_cta) + 32u * threadIdx.x;
    if (32u * threadIdx.x < 3u * faces_per_cta && ahead < 3ull * p.mesh.num_faces)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p.mesh.idx + ahead));
    pdl_wait();
    pdl_release();
    face_cta<true, true>(p, blockIdx.x * faces_per_cta, faces_per_cta, p.scratch.counters, p.scratch.collect_stats != 0,
                         sm);
}

// The listed faces, spread over the warps of the grid first (lane 0 of each, then lane 1, ...):
// the lanes of a warp would run different planes' chains one after another.
template <int S>
__global__ void __launch_bounds__(kClipBlock) clip_kernel(const __grid_constant__ DrawParams p) {
    pdl_wait();
    pdl_release();
    DevCounters* c = p.scratch.counters;
    const uint32_t n = min(ld_volatile(&c->cut_count), p.mesh.num_drawn);
    const uint32_t warps = gridDim.x * (kClipBlock / 32);
    GeomStats st = {0, 0, 0, 0};
    for (uint32_t k = blockIdx.x * (kClipBlock / 32) + (threadIdx.x >> 5) + (threadIdx.x & 31u) * warps; k < n;
         k += 32 * warps)
        clip_listed<S>(p, p.scratch.cut[k], st);
    __syncwarp();
    geometry_warp_tail(p.target, c, p.scratch.collect_stats != 0, st, kNoTile);
}

__global__ void __launch_bounds__(kBlock) large_kernel(const __grid_constant__ DrawParams p) {
    pdl_wait();
    pdl_release();
    DevCounters* c = p.scratch.counters;
    const uint32_t n_items = min(ld_volatile(&c->item_count), p.scratch.item_cap);
    const uint32_t n_tris = min(ld_volatile(&c->large_count), p.scratch.large_cap);
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (kBlock / 32);
    uint32_t frags = 0, tested = 0;
    for (uint32_t it = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); it < n_items; it += warps) {
        const LargeItem item = p.scratch.items[it];
        if (item.tri >= n_tris) continue;  // reserved slot of a triangle rasterised elsewhere
        Edges e;
        uint32_t tag;
        load_large(&p.scratch.large[item.tri], e, tag);
        large_tile(p.target, e, tag, item.tile, frags, tested);
    }
    if (p.scratch.collect_stats) {
        uint32_t f = __reduce_add_sync(0xFFFFFFFFu, frags);
        const uint32_t te = __reduce_add_sync(0xFFFFFFFFu, tested);
        if (lane == 0 && f) atomicAdd(&c->stat_fragments, (unsigned long long)f);
        if (lane == 0 && te) atomicAdd(&c->stat_tested, (unsigned long long)te);
    }
}

// Resident 256-thread CTAs per SM the shading kernels are compiled for, by the shader's registers
// (frames, us: PBR close-up 102.8 / 96.2 / 96.7 at 2 / 3 / 4 CTAs, Blinn-Phong terrain 96.3 / 94.9 / 96.7
// at 3 / 4 / 5; without a bound PBR took 86 registers, so 2 CTAs).
constexpr int tile_blocks(int shader) {
    return shader == kPhong || shader == kPBR ? 3 : shader == kBlinnPhong ? 4 : 5;
}

// One covered pixel (x | y << 16) whose winner is `tag`: shaded and merged.
template <int S, bool kClip>
__device__ __forceinline__ void shade_listed(const DrawParams& p, uint2 w) {
    const DevTarget& t = p.target;
    const int px = (int)(w.x & 0xFFFFu), py = (int)(w.x >> 16);
    const size_t idx = (size_t)py * (size_t)t.width + (size_t)px;
    uint32_t bgra;
    float z;
    if (shade_any<S, kClip>(p, w.y, px, py, t.depth[idx], bgra, z)) {
        t.color[idx] = bgra;
        t.depth[idx] = z;
    }
}

// Tile pass of a small frame: a CTA per flagged tile, a thread per pixel. The covered pixels are
// listed in shared memory, so that a tile of few fills as few warps; a frame of this size is
// bound by latency, and one kernel has one start and one chain.
template <int S, bool kClip>
__global__ void __launch_bounds__(kBlock, tile_blocks(S)) tile_kernel(const __grid_constant__ DrawParams p) {
    __shared__ uint2 s_list[256];
    __shared__ uint32_t s_fill;
    const DevTarget& t = p.target;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) s_fill = 0u;
    pdl_wait();
    pdl_release();
    const uint32_t tile = blockIdx.x;
    if (ld_volatile(&t.tile_flag[tile]) == 0u) return;  // the same for every thread
    const uint32_t px = tile % (uint32_t)t.tiles_x * kTile + (uint32_t)(tid & 15);
    const uint32_t py = tile / (uint32_t)t.tiles_x * kTile + (uint32_t)(tid >> 4);
    unsigned long long key = kEmptyKey;
    const size_t idx = (size_t)py * (size_t)t.width + px;
    if (px < (uint32_t)t.width && py < (uint32_t)t.height) key = __ldcg(t.key + idx);
    const bool has = key != kEmptyKey;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, has);
    __syncthreads();  // s_fill; and every thread has read the flag
    if (tid == 0) t.tile_flag[tile] = 0u;
    uint32_t at = 0;
    if (lane == 0 && m) at = atomicAdd(&s_fill, (uint32_t)__popc(m));
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    if (has) {
        s_list[at + (uint32_t)__popc(m & ((1u << lane) - 1u))] = make_uint2(px | (py << 16), (uint32_t)key);
        t.key[idx] = kEmptyKey;  // for the next draw
    }
    __syncthreads();
    const uint32_t n = s_fill;
    if (p.scratch.collect_stats && tid == 0 && n) {
        atomicAdd(&p.scratch.counters->stat_tiles, 1ull);
        atomicAdd(&p.scratch.counters->stat_shaded, (unsigned long long)n);
    }
    if ((uint32_t)tid < n) shade_listed<S, kClip>(p, s_list[tid]);
}

// Key scan of a larger frame: a tile per warp, all its keys in flight at once; the covered pixels are
// appended to the shade list, their keys and the tile's flag reset. List space is taken once per CTA (a
// prefix over the warps), so the global counter sees few atomics.
// Bound by the keys' reads: many warps with a tile each hide them better than few with two (2M-triangle
// terrain / 200k small triangles at 3840x2160, us a frame: one tile, 6 CTAs per SM 85.4 / 95.9; two, 3 CTAs
// 86.2 / 97.5; two, 4 CTAs 86.5 / 95.0; one, 7 CTAs (spills) 89.4 / 103; four, 2 CTAs 87.5 / 102).
__global__ void __launch_bounds__(kBlock, 6) scan_kernel(const __grid_constant__ DrawParams p) {
    constexpr int kWarps = kBlock / 32;
    __shared__ uint32_t s_count[kWarps], s_base;
    DevCounters* c = p.scratch.counters;
    const DevTarget& t = p.target;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t ntiles = (uint32_t)t.tiles_x * (uint32_t)t.tiles_y, tile = blockIdx.x * kWarps + (uint32_t)warp;
    pdl_wait();
    pdl_release();
    const bool dirty = tile < ntiles && ld_volatile(&t.tile_flag[tile]) != 0u;
    const uint32_t pos = (tile % (uint32_t)t.tiles_x * kTile + (uint32_t)(lane & 15)) |
                         (tile / (uint32_t)t.tiles_x * kTile + (uint32_t)(lane >> 4)) << 16;  // the lane's first pixel
    unsigned long long keys[8];
    uint32_t count = 0;
    {
        const uint32_t px = pos & 0xFFFFu, py = pos >> 16;
        const unsigned long long* at = t.key + (size_t)py * (size_t)t.width + px;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            keys[r] = (dirty && px < (uint32_t)t.width && py + 2 * r < (uint32_t)t.height) ? __ldcg(at) : kEmptyKey;
            at += 2 * (size_t)t.width;
        }
    }
    if (dirty) {
#pragma unroll
        for (int r = 0; r < 8; ++r) count += (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, keys[r] != kEmptyKey));
    }
    if (lane == 0) s_count[warp] = count;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const uint32_t v = s_count[w];
        if (w < warp) before += v;
        total += v;
    }
    if (threadIdx.x == 0 && total) s_base = atomicAdd(&c->shade_count, total);
    __syncthreads();
    if (!dirty) return;
    uint32_t at = s_base + before;
    unsigned long long* key = t.key + (size_t)(pos >> 16) * (size_t)t.width + (pos & 0xFFFFu);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const bool has = keys[r] != kEmptyKey;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, has);
        if (has) {
            p.scratch.shade[at + (uint32_t)__popc(m & below)] = make_uint2(pos + ((uint32_t)(2 * r) << 16), (uint32_t)keys[r]);
            key[(size_t)(2 * r) * (size_t)t.width] = kEmptyKey;  // for the next draw
        }
        at += (uint32_t)__popc(m);
    }
    if (lane == 0) {
        t.tile_flag[tile] = 0u;
        if (p.scratch.collect_stats && count) {
            atomicAdd(&c->stat_tiles, 1ull);
            atomicAdd(&c->stat_shaded, (unsigned long long)count);
        }
    }
}

// The listed pixels, a thread each: covered areas are spread evenly over all SMs.
template <int S, bool kClip>
__global__ void __launch_bounds__(kBlock, tile_blocks(S)) shade_kernel(const __grid_constant__ DrawParams p) {
    pdl_wait();
    pdl_release();
    const uint32_t n = min(ld_volatile(&p.scratch.counters->shade_count), p.scratch.px_cap);
    const uint2* list = p.scratch.shade;
    for (uint32_t q = blockIdx.x * kBlock + threadIdx.x; q < n; q += gridDim.x * kBlock) shade_listed<S, kClip>(p, list[q]);
}

// Colour and/or depth fill, 16-byte stores (the planes are 256-byte aligned allocations).
__global__ void clear_kernel(uint32_t* color, float* depth, size_t n, uint32_t bgra, float dv, int do_color,
                             int do_depth) {
    pdl_wait();
    pdl_release();
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t n4 = n / 4;
    const uint4 cv = make_uint4(bgra, bgra, bgra, bgra);
    const float4 dv4 = make_float4(dv, dv, dv, dv);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
        if (do_color) reinterpret_cast<uint4*>(color)[i] = cv;
        if (do_depth) reinterpret_cast<float4*>(depth)[i] = dv4;
    }
    for (size_t i = 4 * n4 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (do_color) color[i] = bgra;
        if (do_depth) depth[i] = dv;
    }
}

__global__ void fill_u64_kernel(unsigned long long* dst, size_t n, unsigned long long v) {
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = v;
}

__device__ void debug_emit(float* out, uint32_t* count, uint32_t cap, const Screen& s, uint32_t tag) {
    if (is_backface(s)) return;
    uint32_t slot = atomicAdd(count, 1u);
    if (slot >= cap) return;
    float* o = out + 14ull * slot;
    o[0] = __uint_as_float(tag);
    for (int k = 0; k < 3; ++k) { o[1 + 2 * k] = s.x[k]; o[2 + 2 * k] = s.y[k]; o[7 + k] = s.z[k]; }
    o[10] = s.minx; o[11] = s.miny; o[12] = s.maxx; o[13] = s.maxy;
}

// Stage dump: the same clip / cull / setup as the geometry kernel, computed from the mesh
// directly (no vertex cache), writing one record per surviving triangle.
__global__ void debug_triangles_kernel(const __grid_constant__ DrawParams p, float* out, uint32_t* count,
                                       uint32_t cap) {
    uint32_t o = blockIdx.x * kBlock + threadIdx.x;
    if (o >= p.mesh.num_drawn || o > kMaxOrdinal) return;
    FaceRef fr = face_of(p.mesh, o);
    uint3 f = load_face(p.mesh, fr.face);
    const uint32_t nv = p.mesh.num_vertices;
    if (f.x >= nv || f.y >= nv || f.z >= nv) return;
    f4 c0 = load_clip(p.mesh, p.u.mvp, f.x), c1 = load_clip(p.mesh, p.u.mvp, f.y);
    f4 c2 = load_clip(p.mesh, p.u.mvp, f.z);
    int cls = clip_classify(c0, c1, c2);
    if (cls == 3) {
        Screen s;
        screen_setup(c0, c1, c2, p.target.width, p.target.height, s);
        debug_emit(out, count, cap, s, o << 4);
    } else if (cls < 0) {
        CVClip a[kMaxClipVerts], b[kMaxClipVerts];
        a[0].clip = c0; a[1].clip = c1; a[2].clip = c2;
        CVClip* res;
        int n = clip_triangle<0>(a, b, &res);
        for (int j = 0; 3 * j + 2 < n; ++j) {
            Screen s;
            screen_setup(res[3 * j].clip, res[3 * j + 1].clip, res[3 * j + 2].clip, p.target.width,
                         p.target.height, s);
            debug_emit(out, count, cap, s, (o << 4) | 8u | (uint32_t)j);
        }
    }
}

__global__ void debug_sample_kernel(DevTexture tex, const float2* uv, float4* out, uint32_t n) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 q = uv[i];
    f4 c = tex_sample(tex, mk2(q.x, q.y));
    out[i] = make_float4(c.x, c.y, c.z, c.w);
}

unsigned grid_for(size_t n, int block, unsigned cap = 65535u * 16u) {
    size_t g = (n + (size_t)block - 1) / (size_t)block;
    if (g == 0) g = 1;
    return (unsigned)(g < cap ? g : cap);
}

template <int S>
cudaError_t launch_shaded(const DrawParams& p, const LaunchConfig& cfg, cudaStream_t stream, cudaEvent_t* ev,
                          uint64_t* launches) {
    cudaError_t e;
    auto mark = [&](int k) { return ev ? cudaEventRecord(ev[k], stream) : cudaSuccess; };
    if ((e = mark(0)) != cudaSuccess) return e;
    if (p.mesh.num_drawn == 0) {  // nothing to draw: the framebuffer stays as it is
        for (int k = 1; k < kStageEvents; ++k)
            if ((e = mark(k)) != cudaSuccess) return e;
        return cudaSuccess;
    }
    e = launch_dependent(vertex_kernel<S>, grid_for(p.mesh.num_vertices, kBlock, 0x7FFFFFFFu), (unsigned)kBlock, stream, p);
    if (e != cudaSuccess) return e;
    if ((e = mark(1)) != cudaSuccess) return e;
    const uint32_t share = face_share(p.mesh.num_drawn, cfg.num_sms);
    e = launch_dependent(geometry_kernel, grid_for(p.mesh.num_drawn, (int)share, 0x7FFFFFFFu), kPhasedFaceUnit, stream, p,
                         share);
    if (e != cudaSuccess || (e = mark(2)) != cudaSuccess) return e;
    const bool clipped = !cfg.clip_free;
    if (clipped) {
        // a warp for each of the first num_sms * 8 faces
        e = launch_dependent(clip_kernel<S>, (unsigned)cfg.num_sms * 4u, (unsigned)kClipBlock, stream, p);
        if (e != cudaSuccess) return e;
    }
    if ((e = mark(3)) != cudaSuccess) return e;
    e = launch_dependent(large_kernel, (unsigned)(cfg.num_sms * cfg.large_ctas_per_sm), (unsigned)kBlock, stream, p);
    if (e != cudaSuccess || (e = mark(4)) != cudaSuccess) return e;
    const uint32_t tiles = (uint32_t)(p.target.tiles_x * p.target.tiles_y);
    const bool scan = scan_pass(tiles, cfg.num_sms);
    if (scan) {
        e = launch_dependent(scan_kernel, grid_for(tiles, kBlock / 32, 0x7FFFFFFFu), (unsigned)kBlock, stream, p);
        if (e != cudaSuccess) return e;
        *launches += 1;
    }
    if ((e = mark(5)) != cudaSuccess) return e;
    if (!scan) {
        e = clipped ? launch_dependent(tile_kernel<S, true>, tiles, (unsigned)kBlock, stream, p)
                    : launch_dependent(tile_kernel<S, false>, tiles, (unsigned)kBlock, stream, p);
    } else {
        const unsigned shade_ctas = (unsigned)(cfg.num_sms * tile_blocks(S));
        e = clipped ? launch_dependent(shade_kernel<S, true>, shade_ctas, (unsigned)kBlock, stream, p)
                    : launch_dependent(shade_kernel<S, false>, shade_ctas, (unsigned)kBlock, stream, p);
    }
    if (e != cudaSuccess) return e;
    *launches += clipped ? 5 : 4;
    return mark(6);
}

}  // namespace

// Up to 30 tiles per SM one kernel is faster (frames, us, one kernel / scan and shade: 96x96 icon 19.5 /
// 22.8, 512x512 sphere 22.6 / 26.2, 1365x767 close-up 93.6 / 96.2); in larger frames it is not, since it
// shades a tile where its CTA runs while a list spreads the covered pixels evenly over all
// threads, and its keys' reads wait for shading (1920x1080 terrain level; 200k small triangles at
// 3840x2160 120 to 139 with 8 tiles per CTA / 106).
bool scan_pass(uint32_t tiles, int num_sms) { return tiles > 30u * (uint32_t)num_sms; }

cudaError_t launch_draw(const DrawParams& p, const LaunchConfig& cfg, cudaStream_t stream, cudaEvent_t* stage_events,
                        uint64_t* launches) {
    switch (p.u.shader) {
        case kFlat: return launch_shaded<kFlat>(p, cfg, stream, stage_events, launches);
        case kPhong: return launch_shaded<kPhong>(p, cfg, stream, stage_events, launches);
        case kPBR: return launch_shaded<kPBR>(p, cfg, stream, stage_events, launches);
        case kBlinnPhong: return launch_shaded<kBlinnPhong>(p, cfg, stream, stage_events, launches);
        case kGouraud: return launch_shaded<kGouraud>(p, cfg, stream, stage_events, launches);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_clear(uint32_t* color, float* depth, size_t pixels, uint32_t bgra, float depth_value,
                         bool do_color, bool do_depth, cudaStream_t stream) {
    return launch_dependent(clear_kernel, grid_for(pixels, 256, 4096), 256u, stream, color, depth, pixels, bgra, depth_value,
                            do_color ? 1 : 0, do_depth ? 1 : 0);
}

cudaError_t launch_fill_u64(unsigned long long* dst, size_t n, unsigned long long v, cudaStream_t stream) {
    fill_u64_kernel<<<grid_for(n, 256, 4096), 256, 0, stream>>>(dst, n, v);
    return cudaGetLastError();
}

// ---- mesh uploads: float3 arrays widened to float4, with the positions' bounds after an update
// (batch planning's density classes, clip-free draws). One kernel for all arrays, each block's box
// in memory instead of atomics on a cleared word, and the result written to the host's memory: a
// copy, a kernel and a memset each, one after another, cost more than their work (65k-vertex
// mesh updated and drawn: 160 to 112 us).
constexpr int kPackBlock = 256;

// The block's box of its threads' boxes.
__device__ __forceinline__ void block_box(float lo[3], float hi[3], float* partial) {
    __shared__ float s_box[kPackBlock / 32][6];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[d] = fminf(lo[d], __shfl_xor_sync(0xFFFFFFFFu, lo[d], o));
            hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xFFFFFFFFu, hi[d], o));
        }
        if ((threadIdx.x & 31) == 0) {
            s_box[threadIdx.x >> 5][d] = lo[d];
            s_box[threadIdx.x >> 5][3 + d] = hi[d];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        float v = s_box[0][threadIdx.x];
        for (int w = 1; w < kPackBlock / 32; ++w)
            v = threadIdx.x < 3 ? fminf(v, s_box[w][threadIdx.x]) : fmaxf(v, s_box[w][threadIdx.x]);
        partial[6 * blockIdx.x + threadIdx.x] = v;
    }
}

__global__ void __launch_bounds__(kPackBlock) mesh_pack_kernel(const __grid_constant__ MeshPack p, float* partial) {
    if (partial) pdl_release();  // without the radius kernel, what follows may read the arrays
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (uint32_t i = blockIdx.x * kPackBlock + threadIdx.x; i < p.n; i += gridDim.x * kPackBlock) {
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            if (k >= p.arrays) break;
            const float* s = p.src[k] + 3ull * i;
            const float v[3] = {s[0], s[1], s[2]};
            p.dst[k][i] = make_float4(v[0], v[1], v[2], 0.0f);
            if (k == 0) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    lo[d] = fminf(lo[d], v[d]);
                    hi[d] = fmaxf(hi[d], v[d]);
                }
            }
        }
    }
    if (partial) block_box(lo, hi, partial);
}

// The same from pinned host memory, with the other arrays: the first vertex_blocks CTAs take 256 vertices
// at a time through shared memory (16-byte loads, all arrays' in flight together), the others copy
// the flat arrays. Bound by the link. Copies into a staging area, one after another and each with its
// start, and a kernel behind them took longer at every size (update and frame, us, copies / this kernel:
// 256 vertices 59 / 40, 4k 68 / 58, 65k 108 / 83, 262k 200 / 181, 1M 590 / 572).
__global__ void __launch_bounds__(kPackBlock) mesh_import_kernel(const __grid_constant__ MeshImport p, uint32_t vertex_blocks,
                                                                 float* partial) {
    if (partial) pdl_release();
    const int tid = threadIdx.x;
    if (blockIdx.x >= vertex_blocks) {
        const size_t first = (size_t)(blockIdx.x - vertex_blocks) * kPackBlock + tid;
        const size_t stride = (size_t)(gridDim.x - vertex_blocks) * kPackBlock;
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const size_t n = p.copy_bytes[a] / 16;
#pragma unroll 4
            for (size_t i = first; i < n; i += stride) p.copy_dst[a][i] = p.copy_src[a][i];
            const uint32_t* s = reinterpret_cast<const uint32_t*>(p.copy_src[a]);
            uint32_t* d = reinterpret_cast<uint32_t*>(p.copy_dst[a]);
            const size_t w = n * 4 + first;
            if (w < p.copy_bytes[a] / 4) d[w] = s[w];  // at most three words
        }
        return;
    }
    __shared__ __align__(16) float s_in[4][3 * kPackBlock];
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (uint32_t v0 = blockIdx.x * kPackBlock; v0 < p.pack.n; v0 += vertex_blocks * kPackBlock) {
        const uint32_t floats = 3u * min((uint32_t)kPackBlock, p.pack.n - v0);
        const uint32_t whole = floats / 4;
        float4 r[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
            if (k < p.pack.arrays && (uint32_t)tid < whole)
                r[k] = reinterpret_cast<const float4*>(p.pack.src[k] + 3ull * v0)[tid];
        __syncthreads();  // the previous vertices have been read
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            if (k >= p.pack.arrays) break;
            if ((uint32_t)tid < whole) reinterpret_cast<float4*>(s_in[k])[tid] = r[k];
            const uint32_t w = 4 * whole + (uint32_t)tid;
            if (w < floats) s_in[k][w] = p.pack.src[k][3ull * v0 + w];
        }
        __syncthreads();
        if (3u * (uint32_t)tid < floats) {
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                if (k >= p.pack.arrays) break;
                const float v[3] = {s_in[k][3 * tid], s_in[k][3 * tid + 1], s_in[k][3 * tid + 2]};
                p.pack.dst[k][v0 + tid] = make_float4(v[0], v[1], v[2], 0.0f);
                if (k == 0) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        lo[d] = fminf(lo[d], v[d]);
                        hi[d] = fmaxf(hi[d], v[d]);
                    }
                }
            }
        }
    }
    if (partial) block_box(lo, hi, partial);
}

// The box of all blocks, then each block's largest squared distance from its centre.
__global__ void __launch_bounds__(kPackBlock) mesh_radius_kernel(const float4* pos, uint32_t n, const float* partial,
                                                                 MeshBounds* out) {
    __shared__ float s_box[6];
    __shared__ double s_r2[kPackBlock / 32];
    pdl_wait();
    pdl_release();
    if (threadIdx.x < 192) {  // a warp per bound
        const uint32_t d = threadIdx.x >> 5, lane = threadIdx.x & 31;
        float v = d < 3 ? INFINITY : -INFINITY;
        for (uint32_t b = lane; b < gridDim.x; b += 32) {
            const float w = partial[6 * b + d];
            v = d < 3 ? fminf(v, w) : fmaxf(v, w);
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float w = __shfl_xor_sync(0xFFFFFFFFu, v, o);
            v = d < 3 ? fminf(v, w) : fmaxf(v, w);
        }
        if (lane == 0) {
            s_box[d] = v;
            if (blockIdx.x == 0) (d < 3 ? out->lo : out->hi)[d % 3] = v;
        }
    }
    __syncthreads();
    float c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = __fmul_rn(0.5f, __fadd_rn(s_box[k], s_box[3 + k]));
    double r2 = 0.0;
    for (uint32_t i = blockIdx.x * kPackBlock + threadIdx.x; i < n; i += gridDim.x * kPackBlock) {
        const float4 p = pos[i];
        const float v[3] = {p.x, p.y, p.z};
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double t = __dsub_rn((double)v[k], (double)c[k]);
            s = __dadd_rn(s, __dmul_rn(t, t));
        }
        r2 = fmax(r2, s);
    }
    for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(0xFFFFFFFFu, r2, o));
    if ((threadIdx.x & 31) == 0) s_r2[threadIdx.x >> 5] = r2;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kPackBlock / 32; ++w) r2 = fmax(r2, s_r2[w]);
        out->r2[blockIdx.x] = r2;
        if (blockIdx.x == 0) out->blocks = gridDim.x;
    }
}

cudaError_t launch_mesh_pack(const MeshPack& p, float* partial, MeshBounds* bounds, cudaStream_t stream, uint64_t* launches) {
    if (p.n == 0) return cudaSuccess;
    const unsigned g = grid_for(p.n, kPackBlock, kBoundsBlocks);
    mesh_pack_kernel<<<g, kPackBlock, 0, stream>>>(p, partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    *launches += 1;
    if (!partial) return cudaSuccess;
    *launches += 1;
    return launch_dependent(mesh_radius_kernel, g, (unsigned)kPackBlock, stream, (const float4*)p.dst[0], p.n,
                            (const float*)partial, bounds);
}

cudaError_t launch_mesh_import(const MeshImport& p, float* partial, MeshBounds* bounds, cudaStream_t stream, uint64_t* launches) {
    const unsigned vb = p.pack.n ? grid_for(p.pack.n, kPackBlock, kBoundsBlocks) : 0u;
    const size_t bytes = p.copy_bytes[0] + p.copy_bytes[1];
    const unsigned cb = bytes ? grid_for(bytes / 16, kPackBlock * 4, kBoundsBlocks) : 0u;
    if (vb + cb == 0) return cudaSuccess;
    mesh_import_kernel<<<vb + cb, kPackBlock, 0, stream>>>(p, vb, vb ? partial : nullptr);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    *launches += 1;
    if (!partial || !vb) return cudaSuccess;
    *launches += 1;
    return launch_dependent(mesh_radius_kernel, vb, (unsigned)kPackBlock, stream, (const float4*)p.pack.dst[0], p.pack.n,
                            (const float*)partial, bounds);
}

cudaError_t launch_debug_triangles(const DrawParams& p, float* out, uint32_t* count, uint32_t capacity,
                                   cudaStream_t stream) {
    if (p.mesh.num_drawn == 0) return cudaSuccess;
    debug_triangles_kernel<<<grid_for(p.mesh.num_drawn, kBlock, 0x7FFFFFFFu), kBlock, 0, stream>>>(p, out, count,
                                                                                                   capacity);
    return cudaGetLastError();
}

cudaError_t launch_debug_sample(DevTexture tex, const float2* uv, float4* out, uint32_t n, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    debug_sample_kernel<<<grid_for(n, 256, 0x7FFFFFFFu), 256, 0, stream>>>(tex, uv, out, n);
    return cudaGetLastError();
}

}  // namespace axr
