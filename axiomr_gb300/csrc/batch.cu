// Batched form: one persistent, cooperative launch renders many independent draws.
//
// The reference issues one drawMesh per mesh, each a full pass of its pipeline
// (src/tiled_pipeline.cpp:143-322). Here every draw of a batch has its own framebuffer,
// so the draws share nothing but the GPU, and one launch walks four phases over the
// work units of all draws, separated by grid barriers:
//   1. vertices   256-vertex units of every draw: screen cache + vertex-shader outputs
//   2. faces      units of faces in draw order (256; in the phased form up to 128): clip, cull, setup,
//                 raster of the smaller boxes; large triangles go to one shared list with one
//                 item per 16x16 tile
//   3. large      warps take items of the shared list, strided over the grid, any draw
//   4. tiles      tile units, one warp per 16x16 tile: a warp reads the tile's depth keys,
//                 shades the winners (compacted across the warp through shared memory),
//                 and writes the whole tile once. A draw that asks for a clear gets it
//                 fused here: the tile is staged in shared memory with the clear colour
//                 and depth, the winners are merged into it, and the 16x16 colour and
//                 depth boxes go out with two TMA tensor stores
//                 (cp.async.bulk.tensor, clipped at the framebuffer edge by the hardware),
//                 so every pixel of the frame is written exactly once.
// Units are handed out round-robin (unit u to CTA u mod grid); a table built by the host
// names each unit's draw, and the CTA stages that draw's DrawParams in shared memory
// (double-buffered, one __syncthreads per unit).
// Results are those of the per-draw path: the same device functions compute every
// value (draw_body.cuh), and the visibility keys give the same winners.
#include <cuda_runtime.h>

#include "batch.h"
#include "draw_body.cuh"
#include "pdl.cuh"
#include "tma.cuh"
#include "unit.cuh"

namespace axr {
namespace {

constexpr int kBatchBlock = 256;
constexpr int kBatchWarps = kBatchBlock / 32;
constexpr int kBatchMinBlocks = 3;  // 256 threads x 3 CTAs: at most 85 registers
constexpr unsigned long long kBarrierTimeoutNs = 2000000000ull;

// Resident 128-thread CTAs per SM the phased face kernel is compiled for (8: at most 64
// registers; its shared memory, 16.9 KB per CTA, allows 9 and more).
#ifndef AXR_FACE_MIN_BLOCKS
#define AXR_FACE_MIN_BLOCKS 8
#endif

// Resident 256-thread CTAs per SM the phased tile kernel is compiled for (4: at most 64
// registers; its shared memory, 39.7 KB per CTA, allows 5 at most).
#ifndef AXR_TILE_MIN_BLOCKS
#define AXR_TILE_MIN_BLOCKS 4
#endif

static_assert(sizeof(DrawParams) % 16 == 0, "DrawParams is copied as 16-byte words");
static_assert(offsetof(BatchDraw, p) % 16 == 0, "DrawParams is copied as 16-byte words");

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid-wide barrier of the cooperative launch (all CTAs are co-resident). The wait is
// bounded: after timeout_ns (kBarrierTimeoutNs unless a caller passes less) it sets
// kErrBarrier and returns false, and the CTA leaves the kernel.
// With phase timing on, the last CTA to arrive at barrier k records the time.
__device__ bool grid_barrier(DevCounters* c, BatchProfile* prof, int k,
                             unsigned long long timeout_ns = kBarrierTimeoutNs) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const uint32_t gen = ld_acquire(&c->bar_gen);
        __threadfence();
        if (atomicAdd(&c->bar_count, 1u) == gridDim.x - 1) {
            if (prof) prof->barrier_ns[k] = global_ns();
            atomicExch(&c->bar_count, 0u);
            __threadfence();
            atomicAdd(&c->bar_gen, 1u);
        } else {
            const unsigned long long t0 = global_ns();
            while (ld_acquire(&c->bar_gen) == gen) {
                if (global_ns() - t0 > timeout_ns) {
                    atomicOr(&c->error, kErrBarrier);
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Phase timing at kernel exit: the last CTA out adds the four phase durations of this
// launch to the accumulators.
__device__ void profile_exit(BatchProfile* prof) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&prof->exits, 1ull) != gridDim.x - 1) return;
    __threadfence();
    const unsigned long long end = global_ns();
    const volatile unsigned long long* b = prof->barrier_ns;
    const unsigned long long t0 = *reinterpret_cast<volatile unsigned long long*>(&prof->start);
    const unsigned long long t[5] = {t0, b[0], b[1], b[2], end};
    for (int k = 0; k < 4; ++k) atomicAdd(&prof->phase_ns[k], t[k + 1] > t[k] ? t[k + 1] - t[k] : 0ull);
    atomicAdd(&prof->launches, 1ull);
    prof->exits = 0ull;
}

// ---- the tile pass, in three steps over one 16x16 tile of draw `p`:
//   tile_scan    (warp) keys -> entries (slot << 8 | pixel) in a list in shared memory:
//                unclipped winners from its front, clipped ones from its back, their tags
//                parked in the colour staging slots; keys and flag reset; pixels without a key
//                get the requested clear (staged when both planes are cleared, else written)
//   shade_winner (thread) one winner: fragment, merged into the staging slots or written to
//                the framebuffer
//   tile_store   (warp) the staged tile out with two TMA tensor stores (or plain stores when
//                the pitch has no tensor map)
// `stage` is the tile's staging buffer: colour plane [256] then depth plane [256].
constexpr int kAnyShader = kMixedShaders;  // template argument: the draw's own shader kind, looked up per CTA

struct TileCtx {
    uint32_t tile;
    int tx, ty;
    bool clear_c, clear_d, full;
};

__device__ __forceinline__ TileCtx tile_ctx_at(const UnitInfo& ui, uint32_t tile, int tx, int ty) {
    TileCtx c;
    c.tile = tile;
    c.tx = tx;
    c.ty = ty;
    c.clear_c = (ui.flags & kBatchClearColor) != 0u;
    c.clear_d = (ui.flags & kBatchClearDepth) != 0u;
    c.full = c.clear_c && c.clear_d;
    return c;
}

__device__ __forceinline__ TileCtx tile_ctx(const DevTarget& t, const UnitInfo& ui, uint32_t tile) {
    return tile_ctx_at(ui, tile, (int)(tile % (uint32_t)t.tiles_x), (int)(tile / (uint32_t)t.tiles_x));
}

// `cap`: entries of the list; `fill` (NULL: an empty list of the warp's own): the list's fill,
// unclipped | clipped << 16, advanced by this tile's. Returns the tile's own counts, packed the
// same way (lane-uniform).
__device__ __forceinline__ uint32_t tile_scan(const DrawParams& p, const UnitInfo& ui, const TileCtx& c, bool dirty,
                                              uint32_t* stage, uint32_t slot, uint16_t* list, uint32_t cap,
                                              uint32_t* fill, DevCounters* counters, bool stats) {
    const DevTarget& t = p.target;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int lx = lane & 15, ly0 = lane >> 4;
    const int px = c.tx * kTile + lx;
    uint32_t* s_col = stage;
    float* s_dep = reinterpret_cast<float*>(stage + 256);
    // all eight keys first: the resets below would otherwise keep the compiler from
    // issuing a row's load before the previous row's store (one load in flight)
    unsigned long long keys[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int py = c.ty * kTile + ly0 + 2 * r;
        const bool in = px < t.width && py < t.height;
        keys[r] = (dirty && in) ? __ldcg(t.key + (size_t)py * (size_t)t.width + (size_t)px) : kEmptyKey;
    }
    uint32_t count = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const bool has = keys[r] != kEmptyKey, clipped = has && (((uint32_t)keys[r]) & 8u) != 0u;
        count += (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, has && !clipped)) +
                 ((uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, clipped)) << 16);
    }
    uint32_t at = 0;  // the list's fill before this tile
    if (fill) {
        if (lane == 0 && count) at = atomicAdd(fill, count);
        at = __shfl_sync(0xFFFFFFFFu, at, 0);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int ly = ly0 + 2 * r, py = c.ty * kTile + ly, pix = ly * kTile + lx;
        const bool in = px < t.width && py < t.height;
        const size_t idx = (size_t)py * (size_t)t.width + (size_t)px;
        const unsigned long long key = keys[r];
        const bool has = key != kEmptyKey;
        const bool clipped = has && (((uint32_t)key) & 8u) != 0u;
        const unsigned mw = __ballot_sync(0xFFFFFFFFu, has && !clipped);
        const unsigned mc = __ballot_sync(0xFFFFFFFFu, clipped);
        if (has) {
            t.key[idx] = kEmptyKey;  // reset for the next draw into this framebuffer
            s_col[pix] = (uint32_t)key;
            const uint32_t k = clipped ? cap - 1u - ((at >> 16) + (uint32_t)__popc(mc & below))
                                       : (at & 0xFFFFu) + (uint32_t)__popc(mw & below);
            list[k] = (uint16_t)((slot << 8) | (uint32_t)pix);
        } else if (c.full) {
            s_col[pix] = ui.clear_bgra;
            s_dep[pix] = ui.clear_depth;
        } else if (in) {
            if (c.clear_c) t.color[idx] = ui.clear_bgra;
            if (c.clear_d) t.depth[idx] = ui.clear_depth;
        }
        at += (uint32_t)__popc(mw) + ((uint32_t)__popc(mc) << 16);
    }
    if (dirty && lane == 0) {
        t.tile_flag[c.tile] = 0u;
        if (stats && count) {
            atomicAdd(&counters->stat_tiles, 1ull);
            atomicAdd(&counters->stat_shaded, (unsigned long long)((count & 0xFFFFu) + (count >> 16)));
        }
    }
    return count;
}

// Merge one shaded (or rejected) fragment of pixel `pix` of the tile.
__device__ __forceinline__ void tile_put(const DevTarget& t, const UnitInfo& ui, const TileCtx& c, uint32_t* stage,
                                         uint32_t pix, size_t idx, bool ok, uint32_t bgra, float z) {
    if (c.full) {
        stage[pix] = ok ? bgra : ui.clear_bgra;
        reinterpret_cast<float*>(stage + 256)[pix] = ok ? z : ui.clear_depth;
    } else if (ok) {
        t.color[idx] = bgra;
        t.depth[idx] = z;
    } else {
        if (c.clear_c) t.color[idx] = ui.clear_bgra;
        if (c.clear_d) t.depth[idx] = ui.clear_depth;
    }
}

template <int S, bool kClipped>
__device__ __forceinline__ void shade_winner(const DrawParams& p, const UnitInfo& ui, const TileCtx& c, uint32_t* stage,
                                             uint32_t pix) {
    const DevTarget& t = p.target;
    const uint32_t tag = stage[pix];
    const int gx = c.tx * kTile + (int)(pix & 15u), gy = c.ty * kTile + (int)(pix >> 4);
    const size_t idx = (size_t)gy * (size_t)t.width + (size_t)gx;
    const float old = c.clear_d ? ui.clear_depth : t.depth[idx];
    uint32_t bgra = 0u;
    float z = 0.0f;
    const bool ok = kClipped ? shade_clipped_px<S>(p, tag, gx, gy, old, &bgra, &z)
                             : shade_unclipped<S, true>(p, tag, gx, gy, old, bgra, z);
    tile_put(t, ui, c, stage, pix, idx, ok, bgra, z);
}

// Returns whether a TMA store was committed.
__device__ __forceinline__ bool tile_store(const DrawParams& p, const UnitInfo& ui, const BatchDraw* bd, const TileCtx& c,
                                           uint32_t* stage) {
    const DevTarget& t = p.target;
    const int lane = threadIdx.x & 31;
    if (!c.full) return false;
    __syncwarp();
    if (ui.flags & kBatchTma) {
        tma_fence_smem();  // this lane's shared-memory writes -> visible to the TMA unit
        __syncwarp();
        if (lane == 0) {
            tma_store_tile(&bd->color_map, stage, c.tx * kTile, c.ty * kTile);
            tma_store_tile(&bd->depth_map, stage + 256, c.tx * kTile, c.ty * kTile);
            tma_commit();
        }
        return true;
    }
    const int lx = lane & 15, ly0 = lane >> 4, px = c.tx * kTile + lx;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int py = c.ty * kTile + ly0 + 2 * r;
        if (px >= t.width || py >= t.height) continue;
        const size_t idx = (size_t)py * (size_t)t.width + (size_t)px;
        t.color[idx] = stage[(ly0 + 2 * r) * kTile + lx];
        t.depth[idx] = reinterpret_cast<const float*>(stage + 256)[(ly0 + 2 * r) * kTile + lx];
    }
    return false;
}

// The whole tile pass by one warp (persistent form). Returns whether a TMA store was committed.
template <int S>
__device__ bool tile_pass(const DrawParams& p, const UnitInfo& ui, const BatchDraw* bd, uint32_t tile, bool dirty,
                          uint32_t* stage, uint16_t* list, DevCounters* counters, bool stats) {
    const TileCtx c = tile_ctx(p.target, ui, tile);
    const uint32_t n = tile_scan(p, ui, c, dirty, stage, 0u, list, 256u, nullptr, counters, stats);
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();
#pragma unroll 1
    for (uint32_t q = lane; q < (n & 0xFFFFu); q += 32) shade_winner<S, false>(p, ui, c, stage, list[q]);
#pragma unroll 1
    for (uint32_t q = lane; q < n >> 16; q += 32) shade_winner<S, true>(p, ui, c, stage, list[255u - q]);
    __syncwarp();
    return tile_store(p, ui, bd, c, stage);
}

// ---- phase bodies, shared by the persistent and the phased forms
template <int S>
__device__ __forceinline__ void vertex_unit(const DrawParams& p, const UnitInfo& ui) {
    const uint32_t i = ui.local * kVertUnit + threadIdx.x;
    if (i < p.mesh.num_vertices) vertex_one<S>(p, i);
}

// Large-triangle tile items of all draws, strided over every warp of the grid (items are
// alike, 256 pixels each, so a static split balances without a shared counter).
__device__ __forceinline__ void large_items(const BatchParams& bp, bool stats) {
    const int lane = threadIdx.x & 31;
    DevCounters* c = bp.counters;
    const uint32_t n_items = min(ld_acquire(&c->item_count), bp.item_cap);
    const uint32_t n_tris = min(ld_acquire(&c->large_count), bp.large_cap);
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    uint32_t frags = 0, tested = 0;
    for (uint32_t it = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < n_items; it += warps) {
        const LargeItem item = bp.items[it];
        if (item.tri >= n_tris) continue;  // reserved slot of a triangle rasterised elsewhere
        const DevTarget t = bp.draws[bp.large_draw[item.tri]].p.target;
        Edges e;
        uint32_t tag;
        load_large(&bp.large[item.tri], e, tag);
        large_tile(t, e, tag, item.tile, frags, tested);
    }
    if (stats) {
        const uint32_t f = __reduce_add_sync(0xFFFFFFFFu, frags);
        const uint32_t te = __reduce_add_sync(0xFFFFFFFFu, tested);
        if (lane == 0 && f) atomicAdd(&c->stat_fragments, (unsigned long long)f);
        if (lane == 0 && te) atomicAdd(&c->stat_tested, (unsigned long long)te);
    }
}

// Both planes of a tile without keys set to the clear values with direct stores: 8 pixels
// of one row per lane (two 16-byte stores per plane) when the tile lies inside a
// framebuffer whose width is a multiple of 4, one pixel per store otherwise.
__device__ __forceinline__ void clear_tile(const DevTarget& t, uint32_t tile, uint32_t cc, float cd) {
    const int lane = threadIdx.x & 31;
    const int tx = (int)(tile % (uint32_t)t.tiles_x), ty = (int)(tile / (uint32_t)t.tiles_x);
    const int x0 = tx * kTile, y0 = ty * kTile;
    if ((t.width & 3) == 0 && x0 + kTile <= t.width && y0 + kTile <= t.height) {
        const int py = y0 + (lane >> 1), px = x0 + 8 * (lane & 1);
        const size_t idx = (size_t)py * (size_t)t.width + (size_t)px;
        const uint4 c4 = make_uint4(cc, cc, cc, cc);
        const float4 d4 = make_float4(cd, cd, cd, cd);
        uint4* c = reinterpret_cast<uint4*>(t.color + idx);
        float4* d = reinterpret_cast<float4*>(t.depth + idx);
        c[0] = c4;
        c[1] = c4;
        d[0] = d4;
        d[1] = d4;
        return;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int px = x0 + (lane & 15), py = y0 + (lane >> 4) + 2 * r;
        if (px >= t.width || py >= t.height) continue;
        const size_t idx = (size_t)py * (size_t)t.width + (size_t)px;
        t.color[idx] = cc;
        t.depth[idx] = cd;
    }
}

// A warp's tiles of a tile unit: their flags with one load per lane, then tile_pass on each
// tile that is dirty or to be cleared. *sbuf alternates the warp's two staging buffers.
template <int S>
__device__ __forceinline__ void tile_unit(const BatchParams& bp, const DrawParams& p, const UnitInfo& ui,
                                          uint32_t* stage2, uint16_t* list, int* sbuf, bool stats) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tpw = bp.tiles_per_warp;
    const uint32_t ntiles = (uint32_t)p.target.tiles_x * (uint32_t)p.target.tiles_y;
    const uint32_t first = (ui.local * kUnitWarps + (uint32_t)warp) * tpw;
    const bool clears = (ui.flags & (kBatchClearColor | kBatchClearDepth)) != 0u;
    const bool flag = (uint32_t)lane < tpw && first + (uint32_t)lane < ntiles &&
                      ld_volatile(&p.target.tile_flag[first + (uint32_t)lane]) != 0u;
    const unsigned dirty = __ballot_sync(0xFFFFFFFFu, flag);
    const bool full_clear = (ui.flags & (kBatchClearColor | kBatchClearDepth)) == (kBatchClearColor | kBatchClearDepth);
    for (uint32_t j = 0; j < tpw; ++j) {
        const uint32_t tile = first + j;
        if (tile >= ntiles) break;
        const bool d = (dirty >> j) & 1u;
        if (!d && !clears) continue;
        if (!d && full_clear) {
            clear_tile(p.target, tile, ui.clear_bgra, ui.clear_depth);
            continue;
        }
        // the store issued from this buffer two tiles ago must have read it
        if (lane == 0) tma_wait_read_1();
        __syncwarp();
        if (tile_pass<S>(p, ui, &bp.draws[ui.draw], tile, d, stage2 + 512 * *sbuf, list, bp.counters, stats))
            *sbuf ^= 1;
    }
}

// ---- persistent form: one cooperative launch, phases behind grid barriers
// Shared memory of the persistent kernel. The face and the tile phase have a grid barrier between them, so
// their parts lie over one another: 37 KB a CTA. One beside the other they took 69 KB, which left
// the gathers of the three resident CTAs little L1 (a step of 20 small / 30 / 120 / 512 mixed draws, us: 195 /
// 531 / 1,999 / 7,640 with 69 KB, 159 / 467 / 1,734 / 6,455 with 37).
struct PersistentSmem {
    __align__(16) DrawParams p[2];
    UnitInfo u[2];
    union {
        FaceSmem<kBatchBlock> face;
        struct {
            __align__(128) uint32_t stage[kBatchWarps][2 * 512];  // warp: 2 x (colour | depth)
            uint16_t list[kBatchWarps][256];
        } tile;
    };
};
static_assert(sizeof(PersistentSmem) <= 40 * 1024, "the phases' parts share their memory");

template <int S>
__global__ void __launch_bounds__(kBatchBlock, kBatchMinBlocks) batch_kernel(const __grid_constant__ BatchParams bp) {
    __shared__ PersistentSmem sm;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool stats = bp.collect_stats != 0;
    BatchProfile* prof = bp.prof;
    if (prof && blockIdx.x == 0 && threadIdx.x == 0) prof->start = global_ns();
    const uint32_t face_base = bp.vert_units, tile_base = bp.vert_units + bp.face_units;
    int buf = 0;
    for (uint32_t u = blockIdx.x; u < bp.vert_units; u += gridDim.x, buf ^= 1) {
        stage_unit(bp, u, &sm.p[buf], &sm.u[buf]);
        __syncthreads();
        vertex_unit<S>(sm.p[buf], sm.u[buf]);
    }
    if (!grid_barrier(bp.counters, prof, 0)) return;
    for (uint32_t u = blockIdx.x; u < bp.face_units; u += gridDim.x, buf ^= 1) {
        stage_unit(bp, face_base + u, &sm.p[buf], &sm.u[buf]);
        __syncthreads();
        face_cta<true, false>(sm.p[buf], sm.u[buf].local * kFaceUnit, kFaceUnit, bp.counters, stats, sm.face);
    }
    if (!grid_barrier(bp.counters, prof, 1)) return;
    large_items(bp, stats);
    if (!grid_barrier(bp.counters, prof, 2)) return;
    int sbuf = 0;
    for (uint32_t u = blockIdx.x; u < bp.tile_units; u += gridDim.x, buf ^= 1) {
        stage_unit(bp, tile_base + u, &sm.p[buf], &sm.u[buf]);
        __syncthreads();
        tile_unit<S>(bp, sm.p[buf], sm.u[buf], sm.tile.stage[warp], sm.tile.list[warp], &sbuf, stats);
    }
    if (lane == 0) tma_wait_all();
    if (prof) profile_exit(prof);
}

// ---- phased form: one launch per phase, one CTA per work unit (large: persistent warps)
// (the vertices, faces and large triangles of every shader kind of a launch set together).
// Each kernel starts while the one before it drains: its CTAs stage their unit, which no kernel
// writes, and wait there.
__global__ void __launch_bounds__(kBatchBlock) batch_vertex_kernel(const __grid_constant__ BatchParams bp) {
    __shared__ __align__(16) DrawParams s_p;
    __shared__ UnitInfo s_u;
    stage_unit(bp, blockIdx.x, &s_p, &s_u);
    pdl_wait();
    pdl_release();
    if (blockIdx.x == 0 && threadIdx.x < kBatchCountersReset / 4)  // first read by the face kernel
        reinterpret_cast<uint32_t*>(bp.counters)[threadIdx.x] = 0u;
    __syncthreads();
    switch (s_p.u.shader) {
        case kFlat: vertex_unit<kFlat>(s_p, s_u); break;
        case kPhong: vertex_unit<kPhong>(s_p, s_u); break;
        case kPBR: vertex_unit<kPBR>(s_p, s_u); break;
        case kBlinnPhong: vertex_unit<kBlinnPhong>(s_p, s_u); break;
        default: vertex_unit<kGouraud>(s_p, s_u); break;
    }
}

__global__ void __launch_bounds__(kPhasedFaceUnit, AXR_FACE_MIN_BLOCKS) batch_face_kernel(const __grid_constant__ BatchParams bp) {
    __shared__ __align__(16) DrawParams s_p;
    __shared__ UnitInfo s_u;
    __shared__ __align__(16) FaceSmem<(int)kPhasedFaceUnit> s_face;
    stage_unit(bp, bp.vert_units + blockIdx.x, &s_p, &s_u);
    pdl_wait();
    pdl_release();
    __syncthreads();
    face_cta<true, false>(s_p, s_u.local * bp.face_unit, bp.face_unit, bp.counters, bp.collect_stats != 0, s_face);
}

__global__ void __launch_bounds__(kBatchBlock) batch_large_kernel(const __grid_constant__ BatchParams bp) {
    pdl_wait();
    pdl_release();
    large_items(bp, bp.collect_stats != 0);
}

// Shared memory of the phased tile kernel.
struct TileSmem {
    __align__(16) DrawParams p;
    UnitInfo u;
    __align__(128) uint32_t stage[kBatchWarps][2][512];
    __align__(128) uint32_t clear[2][256];  // a cleared tile: colour, depth (TMA source)
    uint16_t list[kBatchWarps * 256];       // a round's winners: unclipped from the front, clipped from the back
    uint32_t buf[kBatchWarps];              // each slot's staging buffer and tile (x | y << 16)
    uint32_t pos[kBatchWarps];
    uint32_t fill[2];                       // the list's fill, by round parity
    uint32_t dirty;
};

// Winner `v` of the round's list.
template <int S, bool kClipped>
__device__ __forceinline__ void shade_entry(TileSmem& sm, uint32_t v) {
    const uint32_t w = v >> 8, pos = sm.pos[w];
    const TileCtx c = tile_ctx_at(sm.u, 0u, (int)(pos & 0xFFFFu), (int)(pos >> 16));
    shade_winner<S, kClipped>(sm.p, sm.u, c, sm.stage[w][sm.buf[w]], v & 255u);
}

// The clipped winners of a round, out of line (rare).
template <int S>
__device__ __noinline__ void shade_clipped_list(TileSmem& sm, uint32_t n) {
    for (uint32_t q = threadIdx.x; q < n; q += kBatchBlock)
        shade_entry<S, true>(sm, sm.list[kBatchWarps * 256 - 1 - q]);
}

// A round's winners, shaded by the whole CTA.
template <int S>
__device__ __forceinline__ void shade_list(TileSmem& sm, uint32_t fill) {
#pragma unroll 1
    for (uint32_t q = threadIdx.x; q < (fill & 0xFFFFu); q += kBatchBlock) shade_entry<S, false>(sm, sm.list[q]);
    if (fill >> 16) shade_clipped_list<S>(sm, fill >> 16);
}

// Tile pass of the phased form: one CTA per unit of bp.tile_unit consecutive tiles (at most
// 32). Warp 0 reads the unit's tile flags with one load per lane. Tiles without keys whose two
// planes are to be cleared are cleared directly by the warps (no staging, no barrier). The
// other tiles go through the staged pass in rounds of eight, one per warp: each warp scans its
// tile into the round's winner list, then all 256 threads shade the list (balanced across the
// eight tiles), then each warp stores its tile. A warp's two staging buffers alternate after
// each committed TMA store, so a tile's store overlaps the next round.
template <int S>
__global__ void __launch_bounds__(kBatchBlock, AXR_TILE_MIN_BLOCKS)
    batch_tile_kernel(const __grid_constant__ BatchParams bp) {
    __shared__ TileSmem sm;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool stats = bp.collect_stats != 0;
    stage_unit(bp, bp.vert_units + bp.face_units + blockIdx.x, &sm.p, &sm.u);
    if (threadIdx.x == 0) sm.fill[0] = 0u;
    pdl_wait();
    pdl_release();
    __syncthreads();
    const DrawParams& p = sm.p;
    const UnitInfo& ui = sm.u;
    // a fully cleared draw with tensor maps: its key-less tiles go out as TMA stores of one
    // cleared tile in shared memory (no clear kernel; every pixel of the frame written once)
    const bool tma_clear = (ui.flags & (kBatchClearColor | kBatchClearDepth)) == (kBatchClearColor | kBatchClearDepth) &&
                           (ui.flags & kBatchTma) && !(ui.flags & kBatchClearedApart);
    if (tma_clear) {
        sm.clear[0][threadIdx.x] = ui.clear_bgra;
        sm.clear[1][threadIdx.x] = __float_as_uint(ui.clear_depth);
        tma_fence_smem();  // visible to the TMA unit after the barrier below
    }
    const uint32_t ntiles = (uint32_t)p.target.tiles_x * (uint32_t)p.target.tiles_y;
    const uint32_t unit = bp.tile_unit;  // <= 32
    const uint32_t first = ui.local * unit;
    const uint32_t count = min(unit, ntiles - first);
    if (warp == 0) {
        const bool f = (uint32_t)lane < count && ld_volatile(&p.target.tile_flag[first + (uint32_t)lane]) != 0u;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, f);
        if (lane == 0) sm.dirty = m;
    }
    __syncthreads();
    const unsigned all = count >= 32u ? 0xFFFFFFFFu : ((1u << count) - 1u);
    const unsigned dirty = sm.dirty;
    const bool clears = (ui.flags & (kBatchClearColor | kBatchClearDepth)) != 0u;
    const bool full = (ui.flags & (kBatchClearColor | kBatchClearDepth)) == (kBatchClearColor | kBatchClearDepth);
    // key-less tiles with a full clear, spread over the warps (unless the clear kernel has
    // written them already): TMA stores of the cleared tile, issued by the warp's lane 0 and
    // read back from shared memory before the CTA exits (one issuing thread per tile
    // measured 1% slower); direct stores without tensor maps
    if (full && !(ui.flags & kBatchClearedApart)) {
        unsigned clean = all & ~dirty;
        const BatchDraw* bd = &bp.draws[ui.draw];
        for (int k = 0; clean; ++k) {
            const int t = __ffs(clean) - 1;
            clean &= clean - 1u;
            if ((k & (kBatchWarps - 1)) != warp) continue;
            const uint32_t tile = first + (uint32_t)t;
            if (tma_clear) {
                if (lane == 0) {
                    const int x = (int)(tile % (uint32_t)p.target.tiles_x) * kTile;
                    const int y = (int)(tile / (uint32_t)p.target.tiles_x) * kTile;
                    tma_store_tile(&bd->color_map, sm.clear[0], x, y);
                    tma_store_tile(&bd->depth_map, sm.clear[1], x, y);
                    tma_commit();
                }
            } else {
                clear_tile(p.target, tile, ui.clear_bgra, ui.clear_depth);
            }
        }
    }
    // staged tiles: the dirty ones, plus the key-less ones when only one plane is cleared
    unsigned work = full ? dirty : (clears ? all : dirty);
    uint32_t sbuf = 0;  // the buffer this warp stages into; never the newest committed store's
    for (uint32_t round = 0; work; ++round) {
        // this round: the next eight tiles of `work`, the w-th to warp w
        int mine = -1;
#pragma unroll
        for (int w = 0; w < kBatchWarps; ++w) {
            if (!work) break;
            const int t = __ffs(work) - 1;
            work &= work - 1u;
            if (w == warp) mine = t;
        }
        const uint32_t tile = first + (uint32_t)(mine < 0 ? 0 : mine);
        uint32_t* stage = sm.stage[warp][sbuf];
        const TileCtx c = tile_ctx(p.target, ui, tile);
        if (mine >= 0) {
            if (lane == 0) {
                tma_wait_read_1();  // an older store from this buffer has read it
                sm.buf[warp] = sbuf;
                sm.pos[warp] = (uint32_t)c.tx | ((uint32_t)c.ty << 16);
            }
            __syncwarp();
            tile_scan(p, ui, c, (dirty >> mine) & 1u, stage, (uint32_t)warp, sm.list, kBatchWarps * 256,
                      &sm.fill[round & 1], bp.counters, stats);
        }
        __syncthreads();
        const uint32_t fill = sm.fill[round & 1];
        if (threadIdx.x == 0) sm.fill[(round + 1) & 1] = 0u;  // its last reader passed the barrier above
        if constexpr (S == kAnyShader) {
            switch (p.u.shader) {
                case kFlat: shade_list<kFlat>(sm, fill); break;
                case kPhong: shade_list<kPhong>(sm, fill); break;
                case kPBR: shade_list<kPBR>(sm, fill); break;
                case kBlinnPhong: shade_list<kBlinnPhong>(sm, fill); break;
                default: shade_list<kGouraud>(sm, fill); break;
            }
        } else {
            shade_list<S>(sm, fill);
        }
        __syncthreads();
        if (mine >= 0 && tile_store(p, ui, &bp.draws[ui.draw], c, stage)) sbuf ^= 1u;
    }
    // the staging buffers and the cleared tile must have been read before the CTA exits
    // (a thread that committed no store group passes at once)
    tma_wait_read_0();
}

// Clear of both planes of the phased form's fully cleared draws, in spans of bp.clear_unit
// pixels of one draw with 16-byte stores (planes are 256-byte aligned and spans start at
// multiples of 4 pixels). One CTA per SM walks the spans: 16-byte stores from 256 threads
// per SM reach the HBM write rate.
__global__ void __launch_bounds__(kBatchBlock) batch_clear_kernel(const __grid_constant__ BatchParams bp) {
    pdl_wait();
    pdl_release();
    const uint2* units = reinterpret_cast<const uint2*>(bp.units) + bp.vert_units + bp.face_units + bp.tile_units;
    for (uint32_t u = blockIdx.x; u < bp.clear_units; u += gridDim.x) {
        const uint2 r = __ldg(units + u);
        const BatchDraw* bd = &bp.draws[r.x];
        uint32_t* color = bd->p.target.color;
        float* depth = bd->p.target.depth;
        const size_t n = (size_t)bd->p.target.width * (size_t)bd->p.target.height;
        const uint32_t cc = __ldg(&bd->clear_bgra);
        const float cd = __ldg(&bd->clear_depth);
        const size_t lo = (size_t)r.y * bp.clear_unit, hi = min(n, lo + (size_t)bp.clear_unit);
        const uint4 c4 = make_uint4(cc, cc, cc, cc);
        const float4 d4 = make_float4(cd, cd, cd, cd);
        const size_t v_hi = lo + ((hi - lo) & ~size_t(3));
        for (size_t i = lo + 4 * (size_t)threadIdx.x; i < v_hi; i += 4 * (size_t)kBatchBlock) {
            *reinterpret_cast<uint4*>(color + i) = c4;
            *reinterpret_cast<float4*>(depth + i) = d4;
        }
        for (size_t i = v_hi + threadIdx.x; i < hi; i += kBatchBlock) {
            color[i] = cc;
            depth[i] = cd;
        }
    }
}

__global__ void merge_counters_kernel(DevCounters* dst, DevCounters* src) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const uint32_t err = src->error;
    if (err) atomicOr(&dst->error, err);
    src->error = 0u;
    unsigned long long* d = &dst->stat_triangles;
    unsigned long long* s = &src->stat_triangles;
    for (int k = 0; k < 6; ++k) {  // stat_triangles .. stat_shaded
        if (s[k]) atomicAdd(&d[k], s[k]);
        s[k] = 0ull;
    }
}

// Failure-path probe: CTA 0 waits at a grid barrier that CTA 1 never reaches, so the
// bounded wait gives up after timeout_ns and sets kErrBarrier.
__global__ void barrier_probe_kernel(DevCounters* c, unsigned long long timeout_ns) {
    if (blockIdx.x != 0) return;
    grid_barrier(c, nullptr, 0, timeout_ns);
}

cudaError_t launch_tiles(int shader, const BatchParams& bp, cudaStream_t stream) {
    switch (shader) {
        case kAnyShader: return launch_dependent(batch_tile_kernel<kAnyShader>, bp.tile_units, (unsigned)kBatchBlock, stream, bp);
        case kFlat: return launch_dependent(batch_tile_kernel<kFlat>, bp.tile_units, (unsigned)kBatchBlock, stream, bp);
        case kPhong: return launch_dependent(batch_tile_kernel<kPhong>, bp.tile_units, (unsigned)kBatchBlock, stream, bp);
        case kPBR: return launch_dependent(batch_tile_kernel<kPBR>, bp.tile_units, (unsigned)kBatchBlock, stream, bp);
        case kBlinnPhong: return launch_dependent(batch_tile_kernel<kBlinnPhong>, bp.tile_units, (unsigned)kBatchBlock, stream, bp);
        case kGouraud: return launch_dependent(batch_tile_kernel<kGouraud>, bp.tile_units, (unsigned)kBatchBlock, stream, bp);
        default: return cudaErrorInvalidValue;
    }
}

// One launch set of the phased form, all its shader kinds together, each kernel a dependent launch
// (30 mixed draws 157.4 to 145.8 us, 20 small draws in one call 62 to 51; batches of hundreds of draws are unchanged).
cudaError_t launch_phased(int shader, const BatchParams& bp, int num_sms, cudaStream_t stream, cudaEvent_t* ev,
                          uint64_t* launches, bool clear_late) {
    cudaError_t e = cudaSuccess;
    // zeroed by the vertex kernel where there is one
    if (!bp.vert_units && (e = cudaMemsetAsync(bp.counters, 0, kBatchCountersReset, stream)) != cudaSuccess) return e;
    auto mark = [&](int k) { return ev ? cudaEventRecord(ev[k], stream) : cudaSuccess; };
    // at the HBM write rate; running it beside the vertex and face phases of the same
    // draws (a side stream) measured no faster, since their key atomics then wait on its
    // writes. The raster phases touch only keys and tile flags, so the clear may also
    // run just before the tile pass (clear_late).
    auto clear = [&]() -> cudaError_t {
        if (!bp.clear_units) return cudaSuccess;
        const unsigned g = min(bp.clear_units, (unsigned)num_sms);
        *launches += 1;
        return launch_dependent(batch_clear_kernel, g, (unsigned)kBatchBlock, stream, bp);
    };
    if ((e = mark(0)) != cudaSuccess) return e;
    if (!clear_late && (e = clear()) != cudaSuccess) return e;
    if ((e = mark(1)) != cudaSuccess) return e;
    if (bp.vert_units && (e = launch_dependent(batch_vertex_kernel, bp.vert_units, (unsigned)kBatchBlock, stream, bp)) != cudaSuccess)
        return e;
    if ((e = mark(2)) != cudaSuccess) return e;
    if (bp.face_units && (e = launch_dependent(batch_face_kernel, bp.face_units, kPhasedFaceUnit, stream, bp)) != cudaSuccess)
        return e;
    if ((e = mark(3)) != cudaSuccess) return e;
    // up to 16 CTAs per SM, about three waves of the 5 resident: the items are strided over
    // all warps of the grid, and the later waves even out the first waves' tails (5 per SM
    // measured 3.041 ms per 512-draw step, 8: 3.027, 10: 3.022, 16: 3.018, 32: 3.020); no more
    // CTAs than a small batch has groups of 4 tiles, since CTAs without an item only cost
    const unsigned large_ctas = max((unsigned)num_sms, min((unsigned)num_sms * 16u, bp.tile_units * bp.tile_unit / 4u));
    if (bp.face_units && (e = launch_dependent(batch_large_kernel, large_ctas, (unsigned)kBatchBlock, stream, bp)) != cudaSuccess)
        return e;
    if (clear_late && (e = clear()) != cudaSuccess) return e;
    if ((e = mark(4)) != cudaSuccess) return e;
    if (bp.tile_units && (e = launch_tiles(shader, bp, stream)) != cudaSuccess) return e;
    if ((e = mark(5)) != cudaSuccess) return e;
    *launches += (bp.vert_units ? 1 : 0) + (bp.face_units ? 2 : 0) + (bp.tile_units ? 1 : 0);
    return cudaSuccess;
}

template <int S>
cudaError_t launch_persistent(const BatchParams& bp, int num_sms, cudaStream_t stream, uint64_t* launches) {
    cudaError_t e = cudaMemsetAsync(bp.counters, 0, kBatchCountersReset, stream);
    if (e != cudaSuccess) return e;
    // resident CTAs per SM of this instantiation, per device (a cooperative launch must not
    // exceed it)
    constexpr int kMaxDev = 64;
    static int blocks_per_sm[kMaxDev] = {};
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
    if (blocks_per_sm[dev] == 0) {
        int n = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel<S>, kBatchBlock, 0);
        if (e != cudaSuccess) return e;
        if (n < 1) return cudaErrorInvalidConfiguration;
        blocks_per_sm[dev] = n;
    }
    const unsigned grid = (unsigned)(blocks_per_sm[dev] * num_sms);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kBatchBlock);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (bp.prof && (e = cudaMemsetAsync(&bp.prof->exits, 0, sizeof(bp.prof->exits), stream)) != cudaSuccess) return e;
    e = cudaLaunchKernelEx(&cfg, batch_kernel<S>, bp);
    if (e == cudaSuccess) *launches += 1;
    return e;
}

}  // namespace

cudaError_t launch_batch(int shader, const BatchParams& bp, int form, int num_sms, cudaStream_t stream,
                         cudaEvent_t* phase_events, uint64_t* launches, bool clear_late) {
    if (form == kFormPhased) return launch_phased(shader, bp, num_sms, stream, phase_events, launches, clear_late);
    switch (shader) {
        case kFlat: return launch_persistent<kFlat>(bp, num_sms, stream, launches);
        case kPhong: return launch_persistent<kPhong>(bp, num_sms, stream, launches);
        case kPBR: return launch_persistent<kPBR>(bp, num_sms, stream, launches);
        case kBlinnPhong: return launch_persistent<kBlinnPhong>(bp, num_sms, stream, launches);
        case kGouraud: return launch_persistent<kGouraud>(bp, num_sms, stream, launches);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_merge_counters(DevCounters* dst, DevCounters* src, cudaStream_t stream) {
    merge_counters_kernel<<<1, 32, 0, stream>>>(dst, src);
    return cudaGetLastError();
}

cudaError_t launch_barrier_probe(DevCounters* counters, unsigned long long timeout_ns, cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(counters, 0, kBatchCountersReset, stream);
    if (e != cudaSuccess) return e;
    barrier_probe_kernel<<<2, 32, 0, stream>>>(counters, timeout_ns);
    return cudaGetLastError();
}

}  // namespace axr
