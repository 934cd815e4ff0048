// Device-side mesh ingest: the part of AxiomR's OBJ loader after text parsing, on the GPU.
//
// Mesh::parseModelFile (src/mesh.cpp:300-415) turns every face-line corner into a Vertex
// (position, uv or (0,0), normal or (0,0,0)), numbers distinct vertices in order of first
// appearance (std::unordered_map with Vertex::operator==, include/mesh.hpp:15-17: all eight
// floats compare equal, so +0 == -0 and a NaN never matches) and fans each polygon into
// triangles; Mesh::calculateTangentBitangent (src/mesh.cpp:222-298) then sums per-face
// tangents and bitangents per vertex in face order and orthonormalises them. Here:
//   corner_keys     one thread per corner: its eight floats
//   insert          open-addressing hash table of corner indices; a slot keeps the smallest
//                   corner index of its key (atomicMin), i.e. the key's first appearance
//   first_flags     a corner is a vertex's first appearance when its slot holds itself
//   scan            exclusive prefix sum of the flags: vertex numbers in appearance order (and
//                   polygon offsets from their sizes)
//   emit_vertices / fan_faces / face_frames / incidence + vertex_frames
// The per-vertex sums run in face order (each vertex's incident (face, corner) entries are
// sorted before summing), so every float is the reference's. The text itself is parsed on
// the host (the reference's parser, or any other that produces the same pools). Of a
// 65k-triangle model's call the kernels are 150 us; the rest was allocations (19 stream-ordered ones from
// a pool that every synchronisation emptied, 9 plain ones and their frees) and host passes over
// corners and positions. Now: one allocation for the scratch and one for the arrays, from a pool that
// the context keeps, and those passes on the device (model ingested and its first 800x600 frame drawn:
// 1070 to 264 us).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "api_internal.h"
#include "api_types.h"
#include "fmath.cuh"

using namespace axr;
using namespace axr_internal;

namespace {

constexpr int kBlock = 256;

struct Key {
    float4 a;  // position x, y, z, uv.x
    float4 b;  // uv.y, normal x, y, z
};

__device__ __forceinline__ bool key_nan(const Key& k) {
    return k.a.x != k.a.x || k.a.y != k.a.y || k.a.z != k.a.z || k.a.w != k.a.w || k.b.x != k.b.x ||
           k.b.y != k.b.y || k.b.z != k.b.z || k.b.w != k.b.w;
}

__device__ __forceinline__ bool key_eq(const Key& p, const Key& q) {
    return p.a.x == q.a.x && p.a.y == q.a.y && p.a.z == q.a.z && p.a.w == q.a.w && p.b.x == q.b.x &&
           p.b.y == q.b.y && p.b.z == q.b.z && p.b.w == q.b.w;
}

__device__ __forceinline__ uint32_t key_hash(const Key& k) {
    const float f[8] = {k.a.x, k.a.y, k.a.z, k.a.w, k.b.x, k.b.y, k.b.z, k.b.w};
    uint32_t h = 2166136261u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t b = f[i] == 0.0f ? 0u : __float_as_uint(f[i]);  // +0 and -0 alike
        h = (h ^ b) * 16777619u;
        h ^= h >> 15;
    }
    return h;
}

// A corner that names no position (the caller is told of the first) gets the pool's first one.
__global__ void corner_keys_kernel(const float* __restrict__ pos, uint32_t n_pos, const float* __restrict__ uv, uint32_t n_uv,
                                   const float* __restrict__ nrm, uint32_t n_nrm, const int* __restrict__ corners,
                                   uint32_t nc, Key* keys, uint32_t* first_bad) {
    const uint32_t c = blockIdx.x * kBlock + threadIdx.x;
    if (c >= nc) return;
    int v = corners[3 * (size_t)c], t = corners[3 * (size_t)c + 1], n = corners[3 * (size_t)c + 2];
    if (v < 0 || (uint32_t)v >= n_pos) {
        atomicMin(first_bad, c);
        if (n_pos == 0) return;  // no vertex comes of it: the call fails
        v = 0;
    }
    const bool tv = t >= 0 && (uint32_t)t < n_uv, nv = n >= 0 && (uint32_t)n < n_nrm;
    Key k;
    k.a = make_float4(pos[3 * (size_t)v], pos[3 * (size_t)v + 1], pos[3 * (size_t)v + 2], tv ? uv[2 * (size_t)t] : 0.0f);
    k.b = make_float4(tv ? uv[2 * (size_t)t + 1] : 0.0f, nv ? nrm[3 * (size_t)n] : 0.0f,
                      nv ? nrm[3 * (size_t)n + 1] : 0.0f, nv ? nrm[3 * (size_t)n + 2] : 0.0f);
    keys[c] = k;
}

// Slot of corner c's key (inserting c when the key is new); -1 for a key with a NaN, which
// never matches. Probing visits every slot at most once.
__device__ int probe(const Key* keys, int* table, uint32_t mask, uint32_t c, bool insert) {
    const Key k = keys[c];
    if (key_nan(k)) return -1;
    uint32_t slot = key_hash(k) & mask;
    for (uint32_t step = 0; step <= mask; ++step) {
        int cur = atomicAdd(&table[slot], 0);
        if (cur < 0) {
            if (!insert) return -1;  // cannot happen after the insert pass
            const int prev = atomicCAS(&table[slot], -1, (int)c);
            if (prev < 0) return (int)slot;
            cur = prev;
        }
        if (key_eq(keys[cur], k)) {
            if (insert) atomicMin(&table[slot], (int)c);
            return (int)slot;
        }
        slot = (slot + 1) & mask;
    }
    return -1;
}

__global__ void insert_kernel(const Key* keys, int* table, uint32_t mask, uint32_t nc) {
    const uint32_t c = blockIdx.x * kBlock + threadIdx.x;
    if (c < nc) probe(keys, table, mask, c, true);
}

// first[c] = 1 when corner c is its vertex's first appearance; rep[c] = that first corner.
__global__ void first_flags_kernel(const Key* keys, int* table, uint32_t mask, uint32_t nc, uint32_t* first,
                                   uint32_t* rep) {
    const uint32_t c = blockIdx.x * kBlock + threadIdx.x;
    if (c >= nc) return;
    const int slot = probe(keys, table, mask, c, false);
    const uint32_t r = slot < 0 ? c : (uint32_t)table[slot];
    rep[c] = r;
    first[c] = r == c ? 1u : 0u;
}

// ---- exclusive prefix sum: block scans, then each block adds the totals of the blocks before it
constexpr int kScanBlock = 1024;

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// dst (may be src): each block's own exclusive sums; the block's total to block_sums. kFan: the
// elements are polygon sizes and count as their fan's triangles.
template <bool kFan>
__global__ void scan_block_kernel(const uint32_t* src, uint32_t* dst, uint32_t n, uint32_t* block_sums) {
    __shared__ uint32_t warp_sums[kScanBlock / 32];
    const uint32_t i = blockIdx.x * kScanBlock + threadIdx.x;
    uint32_t x = i < n ? src[i] : 0u;
    if (kFan) x = x >= 3u ? x - 2u : 0u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t incl = warp_inclusive(x, lane);
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) warp_sums[lane] = warp_inclusive(warp_sums[lane], lane);  // inclusive over warps
    __syncthreads();
    if (i < n) dst[i] = (warp > 0 ? warp_sums[warp - 1] : 0u) + incl - x;
    if (threadIdx.x == 0) block_sums[blockIdx.x] = warp_sums[kScanBlock / 32 - 1];
}

// Block b adds the totals of the blocks before it (a model of 1M corners has 1000);
// `host`: the total (the last element's prefix and `last`, the element itself) and *first_bad go
// there.
__global__ void scan_add_kernel(uint32_t* data, uint32_t n, const uint32_t* block_sums, const uint32_t* last,
                                const uint32_t* first_bad, IngestHost* host) {
    __shared__ uint32_t warp_sums[kScanBlock / 32];
    uint32_t v = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kScanBlock) v += block_sums[b];
    v = __reduce_add_sync(0xFFFFFFFFu, v);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = v;
    __syncthreads();
    v = __reduce_add_sync(0xFFFFFFFFu, warp_sums[threadIdx.x & 31]);
    const uint32_t i = blockIdx.x * kScanBlock + threadIdx.x;
    if (i < n) {
        const uint32_t p = data[i] + v;
        data[i] = p;
        if (host && i == n - 1) {
            host->vertices = p + *last;
            host->first_bad = *first_bad;
        }
    }
}

uint32_t scan_blocks(size_t n) { return (uint32_t)((n + kScanBlock - 1) / kScanBlock); }

// Exclusive sums of src[0, n) into dst; sums: scan_blocks(n) words of scratch.
template <bool kFan = false>
cudaError_t scan_exclusive(const uint32_t* src, uint32_t* dst, uint32_t n, uint32_t* sums, cudaStream_t st,
                           const uint32_t* last = nullptr, const uint32_t* first_bad = nullptr,
                           IngestHost* host = nullptr) {
    if (n == 0) return cudaSuccess;
    const uint32_t blocks = scan_blocks(n);
    scan_block_kernel<kFan><<<blocks, kScanBlock, 0, st>>>(src, dst, n, sums);
    if (blocks > 1 || host) scan_add_kernel<<<blocks, kScanBlock, 0, st>>>(dst, n, sums, last, first_bad, host);
    return cudaGetLastError();
}

// first corners -> vertex arrays (position, uv, normal); every corner -> its vertex number
__global__ void emit_vertices_kernel(const Key* keys, const uint32_t* first, const uint32_t* prefix,
                                     const uint32_t* rep, uint32_t nc, float4* pos, float2* uv, float4* nrm,
                                     uint32_t* vid) {
    const uint32_t c = blockIdx.x * kBlock + threadIdx.x;
    if (c >= nc) return;
    vid[c] = prefix[rep[c]];
    if (!first[c]) return;
    const Key k = keys[c];
    const uint32_t v = prefix[c];
    pos[v] = make_float4(k.a.x, k.a.y, k.a.z, 0.0f);
    uv[v] = make_float2(k.a.w, k.b.x);
    nrm[v] = make_float4(k.b.y, k.b.z, k.b.w, 0.0f);
}

// polygon p (corner offset, face offset) -> its fan (c0, ci, ci+1)
__global__ void fan_faces_kernel(const uint32_t* vid, const uint32_t* poly_corner, const uint32_t* poly_face,
                                 const uint32_t* poly_size, uint32_t np, uint32_t* idx) {
    const uint32_t p = blockIdx.x * kBlock + threadIdx.x;
    if (p >= np) return;
    const uint32_t n = poly_size[p], o = poly_corner[p], f0 = poly_face[p];
    for (uint32_t i = 1; i + 1 < n; ++i) {
        uint32_t* f = idx + 3 * (size_t)(f0 + i - 1);
        f[0] = vid[o];
        f[1] = vid[o + i];
        f[2] = vid[o + i + 1];
    }
}

// per-face tangent and bitangent (src/mesh.cpp:226-257), and each corner's incidence count
__global__ void face_frames_kernel(const uint32_t* idx, uint32_t nf, const float4* pos, const float2* uv,
                                   const float4* nrm, float4* ft, float4* fb, uint32_t* count) {
    const uint32_t f = blockIdx.x * kBlock + threadIdx.x;
    if (f >= nf) return;
    const uint32_t i0 = idx[3 * (size_t)f], i1 = idx[3 * (size_t)f + 1], i2 = idx[3 * (size_t)f + 2];
    const float4 p0 = pos[i0], p1 = pos[i1], p2 = pos[i2];
    const f3 e1 = sub(mk3(p1.x, p1.y, p1.z), mk3(p0.x, p0.y, p0.z));
    const f3 e2 = sub(mk3(p2.x, p2.y, p2.z), mk3(p0.x, p0.y, p0.z));
    const float2 u0 = uv[i0], u1 = uv[i1], u2 = uv[i2];
    const float d1x = fsub(u1.x, u0.x), d1y = fsub(u1.y, u0.y), d2x = fsub(u2.x, u0.x), d2y = fsub(u2.y, u0.y);
    const float den = fsub(fmul(d1x, d2y), fmul(d2x, d1y));
    const float4 n0v = nrm[i0];
    const f3 n0 = mk3(n0v.x, n0v.y, n0v.z);
    f3 t, b;
    if (fabsf(den) < 1e-8f) {
        t = fabsf(n0.x) > 0.8f ? mk3(0.0f, 1.0f, 0.0f) : mk3(1.0f, 0.0f, 0.0f);
        b = cross(n0, t);
    } else {
        const float r = frcp(den);
        t = mul(r, sub(mul(d2y, e1), mul(d1y, e2)));
        b = mul(r, add(mul(-d2x, e1), mul(d1x, e2)));
        if (dot(cross(n0, t), b) < 0.0f) b = neg(b);
    }
    ft[f] = make_float4(t.x, t.y, t.z, 0.0f);
    fb[f] = make_float4(b.x, b.y, b.z, 0.0f);
    atomicAdd(&count[i0], 1u);
    atomicAdd(&count[i1], 1u);
    atomicAdd(&count[i2], 1u);
}

// incidence lists: entry f*3+k of face f's corner k in its vertex's list (unordered)
__global__ void incidence_kernel(const uint32_t* idx, uint32_t nf, const uint32_t* offset, uint32_t* cursor,
                                 uint32_t* entries) {
    const uint32_t f = blockIdx.x * kBlock + threadIdx.x;
    if (f >= nf) return;
    for (int k = 0; k < 3; ++k) {
        const uint32_t v = idx[3 * (size_t)f + k];
        entries[offset[v] + atomicAdd(&cursor[v], 1u)] = 3u * f + (uint32_t)k;
    }
}

// per vertex: its entries sorted (face order), the sums, then the orthonormal frame
// (src/mesh.cpp:260-297; the reference's two fallbacks test glm's vec3::length(), which is
// the component count 3, and never run)
__global__ void vertex_frames_kernel(uint32_t nv, const uint32_t* offset, const uint32_t* count, uint32_t* entries,
                                     const float4* ft, const float4* fb, const float4* nrm, float4* tan, float4* bit) {
    const uint32_t v = blockIdx.x * kBlock + threadIdx.x;
    if (v >= nv) return;
    uint32_t* e = entries + offset[v];
    const uint32_t n = count[v];
    for (uint32_t i = 1; i < n; ++i) {  // insertion sort: lists are short
        const uint32_t x = e[i];
        uint32_t j = i;
        while (j > 0 && e[j - 1] > x) {
            e[j] = e[j - 1];
            --j;
        }
        e[j] = x;
    }
    f3 ts = mk3(0.0f, 0.0f, 0.0f), bs = mk3(0.0f, 0.0f, 0.0f);
    for (uint32_t i = 0; i < n; ++i) {
        const uint32_t f = e[i] / 3u;
        const float4 a = ft[f], b = fb[f];
        ts = add(ts, mk3(a.x, a.y, a.z));
        bs = add(bs, mk3(b.x, b.y, b.z));
    }
    const float4 nv4 = nrm[v];
    const f3 nn = mk3(nv4.x, nv4.y, nv4.z);
    f3 t = n > 0 ? ts : mk3(1.0f, 0.0f, 0.0f);
    t = sub(t, mul(nn, dot(nn, t)));
    t = normalize(t);
    f3 b = cross(nn, t);
    const float hand = dot(bs, b) < 0.0f ? -1.0f : 1.0f;
    b = mul(b, hand);
    tan[v] = make_float4(t.x, t.y, t.z, 0.0f);
    bit[v] = make_float4(b.x, b.y, b.z, 0.0f);
}

unsigned grid(size_t n) { return (unsigned)std::max<size_t>(1, (n + kBlock - 1) / kBlock); }

}  // namespace

extern "C" axr_status axr_mesh_create_from_obj(axr_context* ctx, const axr_obj_desc* d, axr_mesh** out) {
    NvtxRange nvtx_range("axr_mesh_create_from_obj");
    if (!ctx || !d || !out) return fail(ctx, AXR_E_INVALID, "NULL argument");
    *out = nullptr;
    if ((d->num_positions && !d->positions) || (d->num_uvs && !d->uvs) || (d->num_normals && !d->normals) ||
        (d->num_corners && !d->corners) || (d->num_polygons && !d->polygon_sizes) ||
        (d->num_groups && !d->groups) || (d->num_materials && !d->materials))
        return fail(ctx, AXR_E_INVALID, "OBJ descriptor arrays missing");
    const uint32_t nc = d->num_corners, np = d->num_polygons;
    uint64_t corners = 0, faces = 0;
    for (uint32_t p = 0; p < np; ++p) {
        const uint32_t k = d->polygon_sizes[p];
        corners += k;
        faces += k >= 3u ? k - 2u : 0u;
    }
    if (corners != nc) return fail(ctx, AXR_E_INVALID, "polygon sizes add up to %llu corners, not %u",
                                   (unsigned long long)corners, nc);
    if (faces > kMaxOrdinal + 1ull) return fail(ctx, AXR_E_CAPACITY, "a draw is limited to %u faces", kMaxOrdinal + 1u);
    // the corners' positions are checked on the device with the keys; here only where another
    // fault would be reported before theirs
    auto bad_corner = [&](uint64_t i) {
        return fail(ctx, AXR_E_INVALID, "corner %llu names position %d of %u", (unsigned long long)i, d->corners[3 * i],
                    d->num_positions);
    };
    auto check_corners = [&]() -> axr_status {
        for (uint64_t i = 0; i < nc; ++i)
            if (d->corners[3 * i] < 0 || (uint32_t)d->corners[3 * i] >= d->num_positions) return bad_corner(i);
        return AXR_OK;
    };
    const uint32_t nf = (uint32_t)faces;
    for (uint32_t g = 0; g < d->num_groups; ++g) {
        const bool beyond = (uint64_t)d->groups[g].start_face + d->groups[g].face_count > nf;
        if (!beyond && d->groups[g].material < d->num_materials) continue;
        axr_status st = check_corners();
        if (st != AXR_OK) return st;
        if (beyond) return fail(ctx, AXR_E_INVALID, "group %u covers faces beyond the mesh", g);
        return fail(ctx, AXR_E_INVALID, "group %u names material %u of %u", g, d->groups[g].material, d->num_materials);
    }
    std::lock_guard<std::mutex> lk(ctx->mu);
    DeviceGuard g(ctx->device);
    cudaStream_t st = ctx->stream;
    uint32_t cap = 16;
    while (cap < 2u * std::max<uint32_t>(nc, 1u)) cap <<= 1;
    if (!ctx->ingest_host) AXR_CUDA(ctx, cudaMallocHost(&ctx->ingest_host, sizeof(IngestHost)));
    if (!ctx->ingest_pool) {
        // the context's own pool: what it keeps between calls (at most kIngestKept bytes; without it
        // every call maps fresh memory) goes back when the context is destroyed and the last mesh in
        // it is gone
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = ctx->device;
        AXR_CUDA(ctx, cudaMemPoolCreate(&ctx->ingest_pool, &props));
        uint64_t keep = kIngestKept;
        AXR_CUDA(ctx, cudaMemPoolSetAttribute(ctx->ingest_pool, cudaMemPoolAttrReleaseThreshold, &keep));
    }

    // device inputs and scratch in one allocation (vertices: at most one per corner)
    size_t bytes = 0;
    auto place = [&](size_t n) {
        const size_t at = bytes;
        bytes += (std::max<size_t>(n, 16) + 255) & ~size_t(255);
        return at;
    };
    const uint32_t sums_n = std::max({scan_blocks(nc), scan_blocks(np), 1u});
    const size_t o_pos = place(12ull * d->num_positions), o_uv = place(8ull * d->num_uvs), o_nrm = place(12ull * d->num_normals);
    const size_t o_corners = place(12ull * nc), o_sizes = place(4ull * np), o_pc = place(4ull * np), o_pf = place(4ull * np);
    const size_t o_keys = place(sizeof(Key) * nc), o_table = place(4ull * cap + 4), o_first = place(4ull * nc);
    const size_t o_prefix = place(4ull * nc), o_rep = place(4ull * nc), o_vid = place(4ull * nc), o_sums = place(4ull * sums_n);
    const size_t o_ft = place(16ull * nf), o_fb = place(16ull * nf), o_entries = place(12ull * nf);
    const size_t o_count = place(4ull * nc), o_cursor = place(4ull * nc), o_offset = place(4ull * nc);  // count, cursor: zeroed together
    const size_t o_pool4 = place(16ull * d->num_positions), o_partial = place(24ull * kBoundsBlocks);
    unsigned char* mem = nullptr;
    cudaError_t e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&mem), bytes, ctx->ingest_pool, st);
    auto at = [&](auto* type, size_t offset) { return reinterpret_cast<decltype(type)>(mem + offset); };
    float *dpos = at((float*)nullptr, o_pos), *duv = at((float*)nullptr, o_uv), *dnrm = at((float*)nullptr, o_nrm);
    int *dcorners = at((int*)nullptr, o_corners), *table = at((int*)nullptr, o_table);
    Key* keys = at((Key*)nullptr, o_keys);
    auto words = [&](size_t offset) { return at((uint32_t*)nullptr, offset); };
    uint32_t *dps = words(o_sizes), *dpc = words(o_pc), *dpf = words(o_pf), *first = words(o_first), *prefix = words(o_prefix),
             *rep = words(o_rep), *vid = words(o_vid), *sums = words(o_sums), *count = words(o_count),
             *cursor = words(o_cursor), *offset = words(o_offset), *entries = words(o_entries);
    float4 *ft = at((float4*)nullptr, o_ft), *fb = at((float4*)nullptr, o_fb);
    auto put = [&](void* dst, const void* src, size_t n) {
        if (e == cudaSuccess && n) e = cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st);
    };
    IngestHost* host = ctx->ingest_host;  // written by the kernels
    host->first_bad = 0xFFFFFFFFu;
    host->vertices = 0;
    uint32_t* first_bad = words(o_table) + cap;  // all-ones with the table
    put(dpos, d->positions, 12ull * d->num_positions);
    // bounding sphere for batch planning: over the position pool (a superset of the vertices)
    host->bounds.blocks = 0;
    if (e == cudaSuccess && d->num_positions) {
        MeshPack pack{};
        pack.src[0] = dpos;
        pack.dst[0] = at((float4*)nullptr, o_pool4);
        pack.n = d->num_positions;
        pack.arrays = 1;
        e = launch_mesh_pack(pack, at((float*)nullptr, o_partial), &host->bounds, st, &ctx->launches);
    }
    put(duv, d->uvs, 8ull * d->num_uvs);
    put(dnrm, d->normals, 12ull * d->num_normals);
    put(dcorners, d->corners, 12ull * nc);
    put(dps, d->polygon_sizes, 4ull * np);
    if (e == cudaSuccess) e = cudaMemsetAsync(table, 0xFF, 4ull * cap + 4, st);
    if (e == cudaSuccess && nc) {
        corner_keys_kernel<<<grid(nc), kBlock, 0, st>>>(dpos, d->num_positions, duv, d->num_uvs, dnrm, d->num_normals, dcorners,
                                                        nc, keys, first_bad);
        insert_kernel<<<grid(nc), kBlock, 0, st>>>(keys, table, cap - 1, nc);
        first_flags_kernel<<<grid(nc), kBlock, 0, st>>>(keys, table, cap - 1, nc, first, rep);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = scan_exclusive(first, prefix, nc, sums, st, first + nc - 1, first_bad, host);
        ctx->launches += 3;
    }
    cudaEvent_t counted = nullptr;  // the vertex count is on the host
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&counted, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(counted, st);
    // what does not need the count runs while the host waits for it
    if (e == cudaSuccess && np) {
        e = scan_exclusive(dps, dpc, np, sums, st);
        if (e == cudaSuccess) e = scan_exclusive<true>(dps, dpf, np, sums, st);
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(count, 0, o_offset - o_count, st);
    if (counted) {
        const cudaError_t w = cudaEventSynchronize(counted);
        if (e == cudaSuccess) e = w;
        cudaEventDestroy(counted);
    }
    const uint32_t nv = e == cudaSuccess ? host->vertices : 0u;
    if (e == cudaSuccess && host->first_bad != 0xFFFFFFFFu) {
        cudaFreeAsync(mem, st);
        cudaStreamSynchronize(st);
        return bad_corner(host->first_bad);
    }
    // the mesh's arrays in one allocation from the pool; its groups and materials in a plain one
    // (cudaFree of which waits for what still draws the mesh, as for any other mesh)
    auto* m = new axr_mesh();
    m->device = ctx->device;
    m->num_vertices = nv;
    m->num_faces = nf;
    m->num_groups = d->num_groups;
    m->num_materials = d->num_materials;
    const size_t ng = std::max<uint32_t>(1, d->num_groups), nm = std::max<uint32_t>(1, d->num_materials);
    bytes = 0;
    const size_t m_pos = place(16ull * nv), m_nrm = place(16ull * nv), m_tan = place(16ull * nv), m_bit = place(16ull * nv);
    const size_t m_uv = place(8ull * nv), m_idx = place(12ull * nf), m_staging = place(4 * m->staging_floats());
    const size_t mem_bytes = bytes;
    bytes = 0;
    const size_t m_groups = place(sizeof(DevGroup) * ng), m_mats = place(sizeof(DevMaterial) * nm);
    unsigned char* tables = nullptr;
    if (e == cudaSuccess) e = dmalloc(&tables, bytes);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&m->mem, mem_bytes, ctx->ingest_pool, st);
    if (e == cudaSuccess) {
        unsigned char* b = static_cast<unsigned char*>(m->mem);
        m->pos = reinterpret_cast<float4*>(b + m_pos);
        m->nrm = reinterpret_cast<float4*>(b + m_nrm);
        m->tan = reinterpret_cast<float4*>(b + m_tan);
        m->bit = reinterpret_cast<float4*>(b + m_bit);
        m->uv = reinterpret_cast<float2*>(b + m_uv);
        m->idx = reinterpret_cast<uint32_t*>(b + m_idx);
        m->staging = reinterpret_cast<float*>(b + m_staging);
        m->groups = reinterpret_cast<DevGroup*>(tables + m_groups);
        m->materials = reinterpret_cast<DevMaterial*>(tables + m_mats);
    }
    if (e == cudaSuccess && nc) {
        emit_vertices_kernel<<<grid(nc), kBlock, 0, st>>>(keys, first, prefix, rep, nc, m->pos, m->uv, m->nrm, vid);
        fan_faces_kernel<<<grid(np), kBlock, 0, st>>>(vid, dpc, dpf, dps, np, m->idx);
        e = cudaGetLastError();
        ctx->launches += 2;
    }
    if (e == cudaSuccess && nf) {
        face_frames_kernel<<<grid(nf), kBlock, 0, st>>>(m->idx, nf, m->pos, m->uv, m->nrm, ft, fb, count);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = scan_exclusive(count, offset, nv, sums, st);
        if (e == cudaSuccess) {
            incidence_kernel<<<grid(nf), kBlock, 0, st>>>(m->idx, nf, offset, cursor, entries);
            e = cudaGetLastError();
        }
        ctx->launches += 2;
    }
    if (e == cudaSuccess && nv) {
        vertex_frames_kernel<<<grid(nv), kBlock, 0, st>>>(nv, offset, count, entries, ft, fb, m->nrm, m->tan, m->bit);
        e = cudaGetLastError();
        ctx->launches += 1;
    }
    // groups and materials as axr_mesh_create builds them
    std::vector<DevGroup> groups(ng);
    uint32_t base = 0;
    for (uint32_t k = 0; k < d->num_groups; ++k) {
        groups[k] = DevGroup{d->groups[k].start_face, d->groups[k].face_count, base, d->groups[k].material};
        base += d->groups[k].face_count;
    }
    m->num_drawn = base;
    std::vector<DevMaterial> mats(nm);
    for (uint32_t k = 0; k < d->num_materials; ++k) {
        const axr_material_desc& md = d->materials[k];
        DevMaterial& dm = mats[k];
        dm = DevMaterial{};
        auto view = [](const axr_texture* t) {
            DevTexture v{};
            if (t) {
                v.texels = t->texels;
                v.width = t->width;
                v.height = t->height;
            }
            return v;
        };
        dm.diffuse = view(md.diffuse);
        dm.bump = view(md.bump);
        dm.metallic = view(md.metallic);
        dm.roughness = view(md.roughness);
        dm.ao = view(md.ao);
        dm.specular_exponent = md.specular_exponent;
    }
    put(m->groups, groups.data(), sizeof(DevGroup) * groups.size());
    put(m->materials, mats.data(), sizeof(DevMaterial) * mats.size());
    if (mem) cudaFreeAsync(mem, st);
    const cudaError_t done = cudaStreamSynchronize(st);  // also after a failure: kernels write to `host`
    if (e == cudaSuccess) e = done;
    if (e != cudaSuccess) {
        dfree(tables);
        if (m->mem) cudaFree(m->mem);
        delete m;
        return cuda_fail(ctx, e, "mesh ingest");
    }
    take_bounds(m, host->bounds);
    *out = m;
    return AXR_OK;
}

extern "C" axr_status axr_mesh_read(axr_context* ctx, const axr_mesh* m, float* vertices14, uint32_t* indices3) {
    if (!ctx || !m) return fail(ctx, AXR_E_INVALID, "NULL argument");
    std::lock_guard<std::mutex> lk(ctx->mu);
    DeviceGuard g(ctx->device);
    const uint32_t nv = m->num_vertices;
    std::vector<float4> pos(nv), nrm(nv), tan(nv), bit(nv);
    std::vector<float2> uv(nv);
    auto get = [&](void* dst, const void* src, size_t bytes) {
        if (src && bytes) AXR_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
        return AXR_OK;
    };
    axr_status s = AXR_OK;
    if (vertices14) {
        if ((s = get(pos.data(), m->pos, 16ull * nv)) != AXR_OK) return s;
        if ((s = get(nrm.data(), m->nrm, 16ull * nv)) != AXR_OK) return s;
        if ((s = get(uv.data(), m->uv, 8ull * nv)) != AXR_OK) return s;
        if ((s = get(tan.data(), m->tan, 16ull * nv)) != AXR_OK) return s;
        if ((s = get(bit.data(), m->bit, 16ull * nv)) != AXR_OK) return s;
    }
    if (indices3 && (s = get(indices3, m->idx, 12ull * m->num_faces)) != AXR_OK) return s;
    AXR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (vertices14)
        for (uint32_t i = 0; i < nv; ++i) {
            float* o = vertices14 + 14ull * i;
            const float f[14] = {pos[i].x, pos[i].y, pos[i].z, uv[i].x, uv[i].y, nrm[i].x, nrm[i].y, nrm[i].z,
                                 m->tan ? tan[i].x : 0.f, m->tan ? tan[i].y : 0.f, m->tan ? tan[i].z : 0.f,
                                 m->bit ? bit[i].x : 0.f, m->bit ? bit[i].y : 0.f, m->bit ? bit[i].z : 0.f};
            std::memcpy(o, f, sizeof(f));
        }
    return AXR_OK;
}

extern "C" axr_status axr_mesh_counts(const axr_mesh* m, uint32_t* vertices, uint32_t* faces, uint32_t* drawn) {
    if (!m) return fail(nullptr, AXR_E_INVALID, "mesh is NULL");
    if (vertices) *vertices = m->num_vertices;
    if (faces) *faces = m->num_faces;
    if (drawn) *drawn = m->num_drawn;
    return AXR_OK;
}
