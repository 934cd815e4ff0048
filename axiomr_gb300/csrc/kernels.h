// Host-side launchers for the draw kernels (kernels.cu). All launches go to `stream`.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_types.h"

namespace axr {

// Side stream and events of a context: the second launch set of a split batch (fork before its
// first launch, join after its last).
struct AuxStream {
    cudaStream_t stream;
    cudaEvent_t fork, join;
};

struct LaunchConfig {
    int num_sms;
    int large_ctas_per_sm;
    // no vertex of the draw can lie outside or on a clip plane (checked on the host from the
    // mesh's bounding sphere): no triangle is clipped, so the clip pass is not run
    bool clip_free = false;
};

// Whether a draw into a frame of so many tiles lists its covered pixels in scratch.shade (a scan
// and a shade kernel) instead of tile by tile in shared memory.
bool scan_pass(uint32_t tiles, int num_sms);

// One draw: vertices, faces (clip classification, cull, setup, raster of the smaller boxes), the
// clip pass, large-triangle tiles, key scan (larger frames), shading and merge (the tile pass).
// `stage_events` (optional, kStageEvents events) are recorded before the first kernel and after each of
// these six stages. Adds the number of kernels launched to *launches.
constexpr int kStageEvents = 7;
cudaError_t launch_draw(const DrawParams& p, const LaunchConfig& cfg, cudaStream_t stream, cudaEvent_t* stage_events,
                        uint64_t* launches);

cudaError_t launch_clear(uint32_t* color, float* depth, size_t pixels, uint32_t bgra, float depth_value,
                         bool do_color, bool do_depth, cudaStream_t stream);
cudaError_t launch_fill_u64(unsigned long long* dst, size_t n, unsigned long long v, cudaStream_t stream);
// The packed float3 arrays of a mesh upload -> float4 (x, y, z, 0), src[k] to dst[k] for the first
// `arrays` (src[0]: positions). With `partial` (6 * kBoundsBlocks floats on the device) also the
// positions' bounds into *bounds (pinned host memory, complete when the stream gets past); the
// box centre and squared radius follow the host's mesh_bounds operation for operation. Adds the
// number of kernels launched to *launches.
struct MeshPack {
    const float* src[4];
    float4* dst[4];
    uint32_t n, arrays;
};
cudaError_t launch_mesh_pack(const MeshPack& p, float* partial, MeshBounds* bounds, cudaStream_t stream, uint64_t* launches);

// A mesh's arrays read by the GPU straight from pinned host memory (all 16-byte aligned): float3
// arrays widened as above, texture coordinates and indices copied.
struct MeshImport {
    MeshPack pack;
    const uint4* copy_src[2];  // uvs, indices
    uint4* copy_dst[2];
    size_t copy_bytes[2];      // multiples of 4
};
cudaError_t launch_mesh_import(const MeshImport& p, float* partial, MeshBounds* bounds, cudaStream_t stream, uint64_t* launches);

// Stage dump for parity tests: every triangle that survives clip + cull, unordered, as
// (tag, screen x0 y0 x1 y1 x2 y2, ndcZ0..2, minX, minY, maxX, maxY) = 14 words.
cudaError_t launch_debug_triangles(const DrawParams& p, float* out, uint32_t* count, uint32_t capacity,
                                   cudaStream_t stream);
cudaError_t launch_debug_sample(DevTexture tex, const float2* uv, float4* out, uint32_t n, cudaStream_t stream);

}  // namespace axr
