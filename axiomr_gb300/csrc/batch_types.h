// Batched form: many independent draws (each with its own mesh, camera, shader and
// framebuffer) in one persistent kernel launch. Shared by the host planner (batch.cpp)
// and the kernel (batch.cu).
//
// Layout of one batch in HBM (one allocation, 256-byte aligned sections):
//   BatchDraw[count]      per draw: tensor maps of the framebuffer planes, DrawParams whose
//                         scratch points into this batch, clear request
//   UnitRef[units]        per work unit (vertex units, then face units, then tile units,
//                         then clear units): the draw it belongs to and its index inside it
//   vertex caches         per draw: vscreen[V] float4 + vattr[n*V] float4 (n = VAttr<S>::n)
//                         + shading records (kRecFloat4 float4 per face in draw order)
//   LargeTri[large_cap], large_draw[large_cap], LargeItem[item_cap]: shared by all draws
// Work units: 256 vertices (vertex phase), up to 256 faces in draw order (geometry phase),
// up to 64 tiles of 16x16 (key-scan + shade phase); the large-triangle phase takes items
// from the shared list.
#pragma once
#include <stdint.h>

#include "device_types.h"

namespace axr {

// Opaque CUtensorMap (128 bytes, 64-byte aligned), filled by cuTensorMapEncodeTiled.
struct alignas(64) TensorMap128 {
    unsigned char bytes[128];
};

constexpr uint32_t kBatchClearColor = 1u;  // clear the colour plane before the draw
constexpr uint32_t kBatchClearDepth = 2u;  // clear the depth plane before the draw
constexpr uint32_t kBatchTma = 4u;         // the tensor maps are valid (width % 4 == 0)
constexpr uint32_t kBatchClearedApart = 8u; // phased form: the clear kernel writes both planes

constexpr uint32_t kVertUnit = 256;
constexpr uint32_t kFaceUnit = 256;        // persistent and binned forms
constexpr uint32_t kPhasedFaceUnit = 128;  // phased form: at most this (the threads of its face
                                           // kernel), fewer in a batch of few faces (face_share)
constexpr uint32_t kPhasedTileUnit = 32;   // phased form: most tiles per tile unit (32-bit tile masks)
constexpr uint32_t kUnitWarps = 8;  // warps of a 256-thread CTA
constexpr uint32_t kClearUnit = 1u << 16;  // most pixels per unit of the phased form's clear kernel

struct alignas(64) BatchDraw {
    TensorMap128 color_map;  // uint32 [height][width], 16x16 box
    TensorMap128 depth_map;  // float  [height][width], 16x16 box
    DrawParams p;
    uint32_t flags;          // kBatch*
    uint32_t clear_bgra;
    float clear_depth;
    uint32_t pad_[13];
};

constexpr uint32_t kErrBarrier = 4u;  // a grid barrier of the batched kernel timed out

struct UnitRef {
    uint32_t draw;   // index into the launch's draw table
    uint32_t local;  // unit index inside the draw
};

// Device-side phase timing of the batched kernel (enabled with the context's profiling):
// accumulated nanoseconds of the four phases and the launches they cover, plus per-launch
// scratch (start, exit counter, barrier completion times).
struct BatchProfile {
    unsigned long long phase_ns[4];
    unsigned long long launches;
    unsigned long long start;
    unsigned long long exits;
    unsigned long long pad_;
    unsigned long long barrier_ns[3];
    unsigned long long pad2_[5];
};

struct BatchParams {
    const BatchDraw* draws;
    const UnitRef* units;         // vert_units + face_units + tile_units entries
    DevCounters* counters;        // the context's counters (grid barrier in bar_count/bar_gen)
    BatchProfile* prof;           // NULL: no phase timing
    const LargeTri* large;
    const LargeItem* items;
    const uint32_t* large_draw;
    uint32_t count;
    uint32_t vert_units, face_units, tile_units;
    uint32_t clear_units;         // phased form: clear_unit-pixel spans of the full clears
    uint32_t large_cap, item_cap;
    int32_t collect_stats;
    uint32_t tiles_per_warp;      // persistent form: tiles a warp takes per tile unit (unit = 8 warps x this)
    uint32_t face_unit;           // faces per face unit
    uint32_t tile_unit;           // tiles per tile unit
    uint32_t clear_unit;          // pixels per clear unit
    BinSet bins;                  // binned form: the launch set's bin counts and clipped records
};

// Faces per CTA of a face launch over `faces` faces with CTAs of kPhasedFaceUnit threads: one
// per thread where that gives every SM four CTAs or more; otherwise fewer, so that a small
// draw's setup chains run side by side on all SMs and each CTA's threads share the pixels of
// its few boxes (frames, us, at 16 / 128 faces per CTA: 4k-triangle sphere 30.8 / 36.9, 200k
// triangles 148 / 119, 2M triangles 322 / 102).
constexpr uint32_t kTileShareCtas = 16;  // CTAs per SM that a tile pass should have
constexpr uint32_t kMinFaceShare = 16;
inline uint32_t face_share(uint64_t faces, int num_sms) {
    uint32_t n = kPhasedFaceUnit;
    while (n > kMinFaceShare && faces < 4ull * (uint64_t)num_sms * n) n /= 2;
    return n;
}

// Most pixels of a box that the face phase of a keyed batch of `faces` faces rasterises where no
// limit was set or tuned: with few CTAs, those with large boxes outlast the others, while the large-triangle
// pass spreads such boxes over all SMs. The lines lie at 4 and 64 CTAs of faces per SM (78k and 1.2M faces);
// the draws' resolution moves the best limit as well, so they are compromises that the
// autotuner betters. A step in us at limits of 64 / 96 / 256, phased: 90k faces 81 / 88 / 92, 326k 161 / 157 /
// 172, 660k 379 / 362 / 340, at a quarter of the resolution 86 / 86 / 94, 1.2M 747 / 721 / 678, at a quarter
// 143 / 141 / 145, 5.4M 3,223 / 3,156 / 2,883. Persistent: 90k 216 / 208 / 217, 326k 466 / 455 / 471, 660k 908 /
// 880 / 857, at a quarter 284 / 283 / 293, 1.2M 1,764 / 1,700 / 1,601, 5.4M 7,130 / 6,949 / 6,461.
inline int32_t face_pixels(uint64_t faces, int num_sms) {
    const uint64_t ctas = faces / kPhasedFaceUnit;
    return ctas < 4ull * (uint64_t)num_sms ? 64 : ctas < 64ull * (uint64_t)num_sms ? 96 : INT32_MAX;
}

// Tiles per CTA of a phased tile pass over `tiles` tiles: 32 where that leaves enough CTAs for
// every SM many times over; fewer in a smaller batch, whose tile pass would otherwise end with
// a few CTAs that still shade their covered tiles one round of eight after another
// (30 mixed draws, 57k tiles: tile pass 115 to 94 us at 16 tiles; fewer cost more in CTA starts,
// 183 against 170 us a step at 4).
inline uint32_t tile_share(uint64_t tiles, int num_sms) {
    uint32_t n = kPhasedTileUnit;
    while (n > 1 && tiles < (uint64_t)kTileShareCtas * (uint64_t)num_sms * n) n /= 2;
    return n;
}

// Pixels per CTA of the phased form's clear kernel over `pixels` pixels: spread over all SMs,
// in multiples of what 256 threads store at once.
inline uint32_t clear_share(uint64_t pixels, int num_sms) {
    const uint64_t n = (pixels / (uint64_t)num_sms + 1023) & ~uint64_t(1023);
    return (uint32_t)(n < 4096 ? 4096 : n > kClearUnit ? kClearUnit : n);
}

// Launch forms of a batch (chosen per batch by the autotuner):
//   kFormPersistent  one cooperative launch: the four phases behind grid barriers
//   kFormPhased      four launches (one per phase), each over the work units of all draws
//   kFormBinned      three launches over the work units of all draws: vertices, faces
//                    (setup and binning), bins (raster, shading and write-out in shared
//                    memory); tile units are bins of 8 tiles, one CTA each
constexpr int kFormPersistent = 0;
constexpr int kFormPhased = 1;
constexpr int kFormBinned = 2;
constexpr uint32_t kPersistentTilesPerWarp = 8;
constexpr uint32_t kSplitMinDraws = 128;  // phased batches of this many draws run as two launch sets
static_assert(kPhasedTileUnit <= 32, "a phased tile unit is described by 32-bit tile masks");

// The shader argument of a phased launch set whose draws are of several kinds.
constexpr int kMixedShaders = -1;

}  // namespace axr
