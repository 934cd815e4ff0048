// Output encoding: framebuffers as PNG files, built on the GPU.
//
// The reference shows a frame by copying the BGRA8 colour plane into a bottom-up 32-bit
// DIB and blitting it to a window (Window::present, src/window.cpp:70-84; the DIB header,
// src/windows_bitmap.cpp:15-30): the alpha byte is not shown and framebuffer row 0 is the
// bottom row of the picture. The headless counterpart here is one PNG file per framebuffer,
// top row first, RGB8 (what the window shows) or RGBA8.
//
// File layout (PNG: ISO/IEC 15948; zlib: RFC 1950; deflate: RFC 1951):
//   signature, IHDR, a tEXt chunk ("Software") whose length puts the first IDAT data byte
//   at file offset 80, IDAT chunks of kIdat data bytes each (the last one shorter), IEND.
//   From one IDAT chunk's data to the next is kChunkStride = 65536 bytes, so every 32-bit
//   word of the compressed stream lies at a 4-byte aligned file offset inside one chunk.
//   The IDAT data is one zlib stream: header 78 01, one deflate block with the fixed
//   Huffman codes, Adler-32. Every scanline has filter type 0 (None).
// Compression: per scanline, runs of pixels equal to their left neighbour become matches
//   at distance 3 / 4 bytes, runs of pixels equal to the ones above matches at one scanline,
//   everything else literals. Runs are cut every 32 pixels (one warp step), so that a warp
//   finds them with ballots and every step's bits are known without a sequential parse;
//   a flat 32-pixel step costs 12-13 bits.
//
// Four launches per call, each over all images of the call:
//   rows   : one warp per scanline, 32 pixels per step: runs, bit counts (warp scan), the
//            codes assembled in shared memory and written as whole words to the scanline's
//            slot in a staging buffer; the Adler-32 partial sums of the scanline
//   layout : one block per image; exclusive scan of the scanline bit counts, then
//            signature, IHDR, tEXt, the IDAT chunk headers, IEND, the Adler-32, file size
//   pack   : one block per 8 or 32 scanlines of an image, one thread per 32-bit word of the
//            compressed stream: gathers its bits from the staged scanlines (zlib and block
//            headers, end-of-block, Adler-32 included) and stores the word; no word is
//            written twice, so no atomics
//   crc    : one block per IDAT chunk: CRC-32 of its type and data
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "api_internal.h"
#include "api_types.h"
#include "pdl.cuh"

using namespace axr_internal;

namespace axr {

constexpr uint32_t kIdat = 65524;         // data bytes of a full IDAT chunk (multiple of 4)
constexpr uint32_t kChunkStride = 65536;  // kIdat + 12: chunk length, type and CRC
constexpr uint32_t kData0 = 80;           // file offset of the first IDAT data byte
constexpr uint32_t kHeadBytes = kData0 - 8;  // signature, IHDR, tEXt
constexpr uint32_t kIendCrc = 0xAE426082u;   // CRC-32 of "IEND"
constexpr uint32_t kHeaderBits = 19;      // zlib header (16 bits) + deflate block header (3)
constexpr uint32_t kCrcPoly = 0xEDB88320u;  // CRC-32 polynomial, bit-reflected
constexpr uint32_t kAdlerMod = 65521u;
constexpr int kPngWarps = 8;
constexpr int kLayoutThreads = 1024;
constexpr uint32_t kCrcThreads = 256;

struct PngJob {
    const uint32_t* color;          // BGRA8 plane, row 0 = bottom
    uint8_t* out;                   // file buffer (device)
    unsigned long long* size;       // file size out (device); 0 when the image did not fit
    unsigned long long capacity;
    unsigned long long stage_base;  // first staging word of this image's scanline slots
    uint32_t width, height, channels, row_bytes;
    uint32_t row_words;   // staging words per scanline slot
    uint32_t row_base;    // first scanline of this image in the call's scanline arrays
    uint32_t max_chunks;  // IDAT chunks of the worst case
    unsigned long long max_words;  // stream words of the worst case
    uint32_t header[kHeadBytes / 4];  // the file's bytes before the first IDAT chunk
};

struct PngLayout {
    unsigned long long end_bit;       // end of the last scanline's bits in the stream
    unsigned long long stream_bytes;  // zlib stream length (IDAT data bytes in all)
    uint32_t chunks;                  // IDAT chunks
    uint32_t adler;                   // Adler-32 of the scanline bytes
    uint32_t error;                   // the file would exceed the buffer
    uint32_t pad;
};

struct PngParams {
    const PngJob* jobs;
    PngLayout* layout;
    uint32_t* stage;           // scanline slots
    uint32_t* row_bits;        // per scanline: its bits (filter byte included)
    uint32_t* s0;              // per scanline: sum of its bytes
    unsigned long long* s1;    // per scanline: sum of (row_bytes - i) * byte_i
    unsigned long long* row_off;  // per scanline: first bit in the stream
    const uint2* groups;       // pack blocks: (image, first scanline) of group_rows scanlines
    uint32_t jobs_n, rows;
    uint32_t group_rows;       // scanlines per pack block
    // CRC-32 by powers of x mod P, bit-reflected (bit 31 holds x^0)
    uint32_t stride[32];       // 2^i * x^(32 * kCrcThreads): bit i of a word, kCrcThreads words on
    uint32_t words[kCrcThreads];  // x^(32 (d + 1))
    uint32_t bytes[4];         // x^(8 d)
};

constexpr uint32_t kGroupRows = 8, kMaxGroupRows = 32;  // scanlines per pack block (see group_share)

constexpr uint32_t kStep = 32, kSteps = 4;         // pixels per parse step, steps per block of the rows pass
constexpr uint32_t kBlockPixels = kStep * kSteps;
// shared words per warp: a block's codes (at most 36 bits a pixel and 31 a step) + carry
constexpr int kBufWords = 160;
constexpr uint32_t kCrcJobs = 1024;  // images whose chunk offsets a crc block keeps in shared memory

// ------------------------------------------------------------------ device helpers

// The last job with row_base <= row (the warp's row), 32 jobs compared at a time.
__device__ __forceinline__ uint32_t find_job(const PngJob* jobs, uint32_t n, uint32_t row, uint32_t lane) {
    uint32_t lo = 0, span = n;
    while (span > 1) {
        const uint32_t step = (span + 31) / 32, i = lane * step;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, i < span && __ldg(&jobs[lo + i].row_base) <= row);
        const uint32_t k = (31u - (uint32_t)__clz((int)m)) * step;
        lo += k;
        span = min(step, span - k);
    }
    return lo;
}

__device__ __forceinline__ uint32_t reverse_bits(uint32_t code, uint32_t len) { return __brev(code) >> (32 - len); }

// Fixed Huffman codes, bits reversed for the LSB-first stream, of matches of 1 to 86 (64) pixels of 3 (4)
// bytes at a distance of one pixel: length symbol (257..285), its extra bits, 5-bit distance code
// (2 or 3, without extra bits).
constexpr uint32_t reversed(uint32_t v, uint32_t n) {
    uint32_t r = 0;
    for (uint32_t i = 0; i < n; ++i) r |= (v >> i & 1u) << (n - 1 - i);
    return r;
}
constexpr uint2 left_match(uint32_t channels, uint32_t pixels) {
    const uint32_t len = pixels * channels, v = len - 3;
    uint32_t sym = 257 + v, extra_bits = 0, extra = 0;
    if (len == 258) {
        sym = 285;
    } else if (v >= 8) {
        while (v >> (extra_bits + 3)) ++extra_bits;  // the top three bits of v are 1xx
        sym = 257 + 4 * (extra_bits + 1) + (v >> extra_bits & 3u);
        extra = v & ((1u << extra_bits) - 1u);
    }
    const uint32_t n = sym < 280 ? 7 : 8;
    const uint32_t code = sym < 280 ? reversed(sym - 256, 7) : reversed(0xC0 + (sym - 280), 8);
    return uint2{code | extra << n | reversed(channels - 1, 5) << (n + extra_bits), n + extra_bits + 5};
}
struct LeftMatches {
    uint2 of[2][86];  // channels - 3, pixels - 1
};
constexpr LeftMatches left_matches() {
    LeftMatches t{};
    for (uint32_t c = 0; c < 2; ++c)
        for (uint32_t k = 0; k < 258 / (c + 3); ++k) t.of[c][k] = left_match(c + 3, k + 1);
    return t;
}
__device__ const LeftMatches g_left = left_matches();
template <int C>
constexpr uint32_t kLongestCode = left_match(C, 258u / C).x;
template <int C>
constexpr uint32_t kLongestBits = left_match(C, 258u / C).y;

// deflate distance code (0..29), its extra bits and their value, for 1 <= dist <= 32768
__device__ __forceinline__ void distance_code(uint32_t dist, uint32_t& code, uint32_t& ebits, uint32_t& extra) {
    const uint32_t v = dist - 1;
    if (v < 4) {
        code = v; ebits = 0; extra = 0;
        return;
    }
    const uint32_t e = (31 - __clz(v)) - 1, m = (v >> e) & 1u;
    code = 2 * (e + 1) + m;
    ebits = e;
    extra = v - ((2 + m) << e);
}

// fixed Huffman code of literal byte b, reversed for the LSB-first stream; returns its length
__device__ __forceinline__ uint32_t literal_code(uint32_t b, uint32_t& code) {
    const bool hi = b >= 144;
    code = hi ? (__brev(0x190u + b - 144u) >> 23) : (__brev(0x30u + b) >> 24);
    return hi ? 9u : 8u;
}

__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// ------------------------------------------------------------------ kernels

// A warp's code buffer: buf[0] holds staging word wbase of its scanline. After codes up
// to bit `end` are in, whole words go out to the staging slot and the partial one moves
// to buf[0]. Warp-uniform.
__device__ __forceinline__ void flush_words(uint32_t* buf, uint32_t* stage, uint32_t row_words, uint32_t& wbase,
                                            uint32_t& nbits, uint32_t end, int lane) {
    const uint32_t done = (end >> 5) - wbase;
    if (done) {
        for (uint32_t k = (uint32_t)lane; k < done; k += 32)
            if (wbase + k < row_words) stage[wbase + k] = buf[k];  // the slot holds the worst case
        const uint32_t carry = buf[done];
        __syncwarp();
        for (uint32_t k = (uint32_t)lane; k <= done; k += 32) buf[k] = 0u;
        __syncwarp();
        if (lane == 0) buf[0] = carry;
        __syncwarp();
        wbase += done;
    }
    nbits = end;
}

// A lane's code of n <= 31 bits, or (kWide) lo and up to 4 bits of hi, at bit `pos` of its
// warp's buffer (n = 0: none).
template <bool kWide>
__device__ __forceinline__ void put_code(uint32_t* buf, uint32_t pos, uint32_t lo, uint32_t hi, uint32_t n) {
    if (!n) return;
    const uint32_t k = pos >> 5, sh = pos & 31u;
    const uint32_t w1 = __funnelshift_l(lo, kWide ? hi : 0u, sh);  // the bits past the word (none: 0)
    atomicOr(&buf[k], lo << sh);
    if (w1) atomicOr(&buf[k + 1], w1);
    if (kWide) {
        const uint32_t w2 = __funnelshift_l(hi, 0u, sh);
        if (w2) atomicOr(&buf[k + 2], w2);
    }
}

// One warp per scanline, parsed in steps of 32 pixels: lane i takes pixel x = step + i. It is in
// a left run when it equals pixel x-1, else in an up run when it equals the pixel above; a run
// starts where its kind starts in the step and ends where it ends or at the step's end. A run
// start emits one match of the run's length, a lone up-run pixel whose match would cost at least
// its literals emits literals instead, other pixels emit literals. Steps that lie wholly in a
// left run (flat regions) are merged into matches of up to 258 bytes; a step wholly equal to the
// scanline above is one match.
//
// Issue bound on a batch, latency bound on one image (a warp per scanline leaves most of the GPU
// idle), so four steps are taken together: their loads, ballots and bit-position scans do not
// wait for one another, the codes go to the staging slot once per block, and the next block's
// pixels are loaded ahead. A block of one colour that goes on with the pixel before it, or starts the
// scanline (flat background, 78% of the 512-frame batch's blocks), costs its loads and one vote: its
// run and its checksum terms are taken in closed form when the run of such blocks ends. Match codes
// are looked up. Rows pass of the 512 frames of a mixed batch (415 Mpixel, RGB) 1.91 ms a step at a
// time, 1.16 with four steps and the vote, 0.98 with closed forms and tables; one 1920x1080 RGBA frame
// 67 to 22 us; at 5 or 3 resident CTAs instead of 4 (64 registers) 1.21 and 1.45 ms (of 1.16).
template <int C>
__global__ void __launch_bounds__(32 * kPngWarps, 4) png_rows_kernel(const __grid_constant__ PngParams p) {
    __shared__ uint32_t s_buf[kPngWarps][kBufWords];
    pdl_release();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * kPngWarps + (uint32_t)warp;
    if (row >= p.rows) return;
    const PngJob& j = p.jobs[find_job(p.jobs, p.jobs_n, row, (uint32_t)lane)];
    const uint32_t W = j.width, H = j.height, L = j.row_bytes, row_words = j.row_words;
    const uint32_t r = row - j.row_base;
    const uint32_t mask = C == 4 ? 0xFFFFFFFFu : 0x00FFFFFFu;
    const uint32_t* src = j.color + (size_t)(H - 1 - r) * W;
    const bool has_up = r > 0 && L <= 32768u;
    const uint32_t* up = src + W;  // the framebuffer row above = the previous scanline
    uint32_t* stage = p.stage + j.stage_base + (size_t)r * row_words;
    uint32_t up_code, up_eb, up_ex;
    distance_code(has_up ? L : 1u, up_code, up_eb, up_ex);
    constexpr uint32_t kMaxRun = 258u / C;  // pixels in the longest match
    constexpr uint32_t full_code = kLongestCode<C>, full_bits = kLongestBits<C>;
    const uint2* matches = g_left.of[C - 3];
    // lane i's codes of matches of i + 1 pixels (at most 31 bits): a step's runs look theirs up
    const uint2 mine = __ldg(matches + lane);
    const uint32_t left_tab = mine.x, left_bits = mine.y, len_bits = left_bits - 5u;
    const uint32_t up_bits = left_bits + up_eb;
    const uint32_t up_tab = (left_tab & ((1u << len_bits) - 1u)) | reverse_bits(up_code, 5) << len_bits | up_ex << (len_bits + 5u);

    uint32_t* buf = s_buf[warp];
    for (int k = lane; k < kBufWords; k += 32) buf[k] = 0u;
    __syncwarp();
    if (lane == 0) buf[0] = reverse_bits(0x30, 8);  // filter type 0 as a literal byte
    uint32_t nbits = 8;    // bits of this scanline so far
    uint32_t wbase = 0;    // staging word that buf[0] holds
    uint32_t prev = 0;     // the pixel before this block
    uint32_t pending = 0;  // pixels of a left run carried over whole steps, not yet emitted
    uint32_t whole = 0;    // longest matches of that run, not yet written
    uint32_t flat = 0;     // pixels of the blocks of one colour just parsed, not yet in the sums
    uint32_t left_run = 0; // and of their left run, not yet in `pending`
    // Adler-32 partial sums: byte i of the scanline (i = 0 is the filter byte, 0) adds
    // (L - i) * byte: (L - i) * (b0 + b1 + b2 [+ b3]) - (b1 + 2 b2 [+ 3 b3]) per pixel
    uint32_t a0 = 0, u0 = 0;            // this lane's bytes; flat blocks (lane-uniform)
    unsigned long long a1 = 0, u1 = 0;
    // (the bytes of a framebuffer word are B, G, R, A; the scanline's R, G, B [, A])
    auto byte_sums = [](uint32_t word, uint32_t& sum, uint32_t& lag) {
        sum = __dp4a(word, C == 4 ? 0x01010101u : 0x00010101u, 0u);
        lag = __dp4a(word, C == 4 ? 0x03000102u : 0x00000102u, 0u);
    };
    // the counted longest matches, 32 at a time
    auto write_whole = [&]() {
        for (; whole; whole -= min(whole, 32u)) {
            const uint32_t n = min(whole, 32u);
            if ((uint32_t)lane < n) 
                put_code<false>(buf, nbits - wbase * 32 + (uint32_t)lane * full_bits, full_code, 0u, full_bits);
            __syncwarp();
            flush_words(buf, stage, row_words, wbase, nbits, nbits + n * full_bits, lane);
        }
    };
    const uint32_t up0 = has_up ? __ldg(up) & mask : 0u;
    // the one-colour blocks that end at pixel x; what is left of `left_run` is the scanline's last part of a step
    auto fold = [&](uint32_t x) {
        if (!flat) return;
        uint32_t sum, lag;
        byte_sums(prev, sum, lag);  // the sum over their pixels of (L - 1 - x C) sum - lag
        const unsigned long long n = flat, x0 = x - flat;
        u0 += flat * sum;
        u1 += n * ((unsigned long long)(L - 1) * sum - lag) - (unsigned long long)(C * sum) * (n * x0 + n * (n - 1) / 2);
        flat = 0;
        pending += left_run & ~(kStep - 1);
        whole += pending / kMaxRun;
        pending %= kMaxRun;
        left_run &= kStep - 1;
    };
    uint32_t raw[kSteps];
#pragma unroll
    for (uint32_t k = 0; k < kSteps; ++k) raw[k] = kStep * k + (uint32_t)lane < W ? __ldg(src + kStep * k + lane) : 0u;
    __syncwarp();
    for (uint32_t c0 = 0; c0 < W; c0 += kBlockPixels) {
        uint32_t next[kSteps];
#pragma unroll
        for (uint32_t k = 0; k < kSteps; ++k) {
            const uint32_t x = c0 + kBlockPixels + kStep * k + (uint32_t)lane;
            next[k] = x < W ? __ldg(src + x) : 0u;
        }
        const uint32_t ref = c0 > 0 ? prev : __shfl_sync(0xFFFFFFFFu, raw[0], 0) & mask;
        bool same = true;
#pragma unroll
        for (uint32_t k = 0; k < kSteps; ++k)
            same = same && ((raw[k] & mask) == ref || c0 + kStep * k + (uint32_t)lane >= W);
        if (__all_sync(0xFFFFFFFFu, same)) {  // one colour, a left run but for the scanline's first pixel
            const uint32_t n = min(W - c0, kBlockPixels);
            flat += n;
            left_run += n;
            if (c0 == 0) {  // the first step: lane 0 the first pixel's code, lane 1 the run after it
                const uint32_t first = min(W, kStep);
                const uint32_t lit[4] = {(ref >> 16) & 255u, (ref >> 8) & 255u, ref & 255u, ref >> 24};
                unsigned long long code = 0;
                uint32_t bits = 0;
#pragma unroll
                for (int q = 0; q < C; ++q) {
                    uint32_t c;
                    const uint32_t l = literal_code(lit[q], c);
                    code |= (unsigned long long)c << bits;
                    bits += l;
                }
                if (has_up && up0 == ref && 12u + up_eb < bits) {
                    code = __shfl_sync(0xFFFFFFFFu, up_tab, 0);
                    bits = __shfl_sync(0xFFFFFFFFu, up_bits, 0);
                }
                const int at = first > 1 ? (int)first - 2 : 0;
                const uint32_t cl = __shfl_sync(0xFFFFFFFFu, left_tab, at);
                const uint32_t nl = first > 1 ? __shfl_sync(0xFFFFFFFFu, left_bits, at) : 0u;
                const uint32_t pos = nbits - wbase * 32;
                if (lane < 2)
                    put_code<C == 4>(buf, lane == 0 ? pos : pos + bits, lane == 0 ? (uint32_t)code : cl,
                                     lane == 0 ? (uint32_t)(code >> 32) : 0u, lane == 0 ? bits : nl);
                __syncwarp();
                flush_words(buf, stage, row_words, wbase, nbits, nbits + bits + nl, lane);
                left_run -= first;
            }
            prev = ref;
#pragma unroll
            for (uint32_t k = 0; k < kSteps; ++k) raw[k] = next[k];
            continue;
        }
        fold(c0);
        write_whole();
        uint32_t u[kSteps], v[kSteps], m_l[kSteps];
#pragma unroll
        for (uint32_t k = 0; k < kSteps; ++k) {
            const uint32_t x = c0 + kStep * k + (uint32_t)lane;
            u[k] = (has_up && x < W) ? (__ldg(up + x) & mask) : 0u;
        }
        uint32_t terms = 0;  // of a1: four at most, each below 131072 * 4 * 1020
#pragma unroll
        for (uint32_t k = 0; k < kSteps; ++k) {
            const uint32_t x = c0 + kStep * k + (uint32_t)lane;
            v[k] = raw[k] & mask;
            uint32_t sum, lag;  // (0 past the scanline's end)
            byte_sums(raw[k], sum, lag);
            a0 += sum;
            terms += (L - 1 - x * C) * sum - lag;
            uint32_t left = __shfl_up_sync(0xFFFFFFFFu, v[k], 1);
            if (lane == 0) left = prev;
            prev = __shfl_sync(0xFFFFFFFFu, v[k], 31);
            m_l[k] = __ballot_sync(0xFFFFFFFFu, x < W && x > 0 && v[k] == left);
        }
        a1 += terms;
        // each step's match before its own codes (the run carried to it, in pixels; lane k keeps
        // step k's) and each lane's code per step
        uint32_t ahead = 0, n[kSteps], lo[kSteps], hi[kSteps];  // hi: RGBA literals' bits past 32
#pragma unroll
        for (uint32_t k = 0; k < kSteps; ++k) {
            const uint32_t x = c0 + kStep * k + (uint32_t)lane;
            const bool valid = x < W;
            lo[k] = hi[k] = n[k] = 0;
            uint32_t before = 0;
            if (m_l[k] == 0xFFFFFFFFu) {  // the whole step continues a left run
                pending += kStep;
                if (pending >= kMaxRun) {
                    before = kMaxRun;
                    pending -= kMaxRun;
                }
            } else if (c0 + kStep * k < W) {
                before = pending;
                pending = 0;
                const bool eq_l = m_l[k] >> lane & 1u;
                const bool eq_u = valid && has_up && !eq_l && v[k] == u[k];
                const unsigned m_u = __ballot_sync(0xFFFFFFFFu, eq_u);
                if (valid) {  // as literals
                    uint32_t c, q;
                    q = literal_code((v[k] >> 16) & 255u, c); lo[k] = c; n[k] = q;
                    q = literal_code((v[k] >> 8) & 255u, c);  lo[k] |= c << n[k]; n[k] += q;
                    q = literal_code(v[k] & 255u, c);         lo[k] |= c << n[k]; n[k] += q;
                    if (C == 4) {
                        q = literal_code(v[k] >> 24, c);
                        lo[k] |= c << n[k];
                        hi[k] = c >> (32u - n[k]);  // n is 24 to 27 here
                        n[k] += q;
                    }
                }
                if (m_l[k] | m_u) {  // some pixels are in runs
                    const unsigned m = eq_l ? m_l[k] : m_u;
                    const bool start = (eq_l || eq_u) && !((m << 1) >> lane & 1u);
                    const uint32_t run = (uint32_t)__clz((int)__brev(~(m >> lane)));  // at a start: 1 to 32
                    const int at = start ? (int)run - 1 : 0;
                    const uint32_t cl = __shfl_sync(0xFFFFFFFFu, left_tab, at), nl = __shfl_sync(0xFFFFFFFFu, left_bits, at);
                    const uint32_t cu = __shfl_sync(0xFFFFFFFFu, up_tab, at), nu = __shfl_sync(0xFFFFFFFFu, up_bits, at);
                    const bool lone_up = eq_u && start && run == 1 && 12u + up_eb >= n[k];
                    if ((eq_l || eq_u) && !lone_up) {
                        lo[k] = eq_l ? cl : cu;
                        hi[k] = 0;
                        n[k] = !start ? 0u : eq_l ? nl : nu;
                    }
                }
            }
            if ((uint32_t)lane == k) ahead = before;
        }
        const uint2 ahead_code = ahead ? __ldg(matches + ahead - 1) : make_uint2(0u, 0u);
        // bit positions of the lanes' codes, two steps' sums (below 2^11) in a word
        static_assert(kSteps == 4, "two words");
        uint32_t in01 = n[0] | n[1] << 16, in23 = n[2] | n[3] << 16;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t01 = __shfl_up_sync(0xFFFFFFFFu, in01, o), t23 = __shfl_up_sync(0xFFFFFFFFu, in23, o);
            if (lane >= o) {
                in01 += t01;
                in23 += t23;
            }
        }
        const uint32_t all01 = __shfl_sync(0xFFFFFFFFu, in01, 31), all23 = __shfl_sync(0xFFFFFFFFu, in23, 31);
        const uint32_t incl[kSteps] = {in01 & 0xFFFFu, in01 >> 16, in23 & 0xFFFFu, in23 >> 16};
        const uint32_t all[kSteps] = {all01 & 0xFFFFu, all01 >> 16, all23 & 0xFFFFu, all23 >> 16};
        uint32_t pos = nbits - wbase * 32, ahead_pos = 0;
#pragma unroll
        for (uint32_t k = 0; k < kSteps; ++k) {
            if ((uint32_t)lane == k) ahead_pos = pos;
            pos += __shfl_sync(0xFFFFFFFFu, ahead_code.y, (int)k);
            put_code<C == 4>(buf, pos + incl[k] - n[k], lo[k], hi[k], n[k]);
            pos += all[k];
        }
        put_code<false>(buf, ahead_pos, ahead_code.x, 0u, ahead_code.y);
        __syncwarp();
        flush_words(buf, stage, row_words, wbase, nbits, wbase * 32 + pos, lane);
#pragma unroll
        for (uint32_t k = 0; k < kSteps; ++k) raw[k] = next[k];
    }
    fold(W);
    write_whole();
    if (pending | left_run) {  // lane 0: what the run carried over; lane 1: its part of the last step
        const uint32_t px = lane == 0 ? pending : lane == 1 ? left_run : 0u;
        const uint2 c = px ? __ldg(matches + px - 1) : make_uint2(0u, 0u);
        const uint32_t nb = __shfl_sync(0xFFFFFFFFu, c.y, 0), nl = __shfl_sync(0xFFFFFFFFu, c.y, 1);
        put_code<false>(buf, nbits - wbase * 32 + (lane == 0 ? 0u : nb), c.x, 0u, c.y);
        __syncwarp();
        flush_words(buf, stage, row_words, wbase, nbits, nbits + nb + nl, lane);
    }
    if (lane == 0 && (nbits & 31u) && wbase < row_words) stage[wbase] = buf[0];
    uint32_t s0 = u0;
    if (__any_sync(0xFFFFFFFFu, a0 != 0u)) {  // (a lane without bytes has no a1 either)
        s0 += __reduce_add_sync(0xFFFFFFFFu, a0);
        a1 = warp_sum64(a1);
    }
    a1 += u1;
    if (lane == 0) {
        p.row_bits[row] = nbits;
        p.s0[row] = s0;
        p.s1[row] = a1;
    }
}

__device__ __forceinline__ void put_be32(uint8_t* p, uint32_t v) {
    p[0] = (uint8_t)(v >> 24);
    p[1] = (uint8_t)(v >> 16);
    p[2] = (uint8_t)(v >> 8);
    p[3] = (uint8_t)v;
}

__global__ void __launch_bounds__(kLayoutThreads) png_layout_kernel(const __grid_constant__ PngParams p) {
    __shared__ unsigned long long s_warp[kLayoutThreads / 32];
    __shared__ unsigned long long s_a[kLayoutThreads / 32], s_b[kLayoutThreads / 32];
    __shared__ unsigned long long s_carry;
    pdl_wait();
    pdl_release();
    const PngJob& j = p.jobs[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_carry = kHeaderBits;
    __syncthreads();
    // exclusive scan of the scanline bit counts
    for (uint32_t c0 = 0; c0 < j.height; c0 += kLayoutThreads) {
        const uint32_t r = c0 + (uint32_t)tid;
        const unsigned long long v = r < j.height ? p.row_bits[j.row_base + r] : 0ull;
        unsigned long long incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            unsigned long long w = s_warp[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, w, o);
                if (lane >= o) w += t;
            }
            s_warp[lane] = w;  // inclusive over warps
        }
        __syncthreads();
        const unsigned long long base = s_carry + (warp ? s_warp[warp - 1] : 0ull);
        if (r < j.height) p.row_off[j.row_base + r] = base + incl - v;
        __syncthreads();
        if (tid == 0) s_carry += s_warp[31];
        __syncthreads();
    }
    const unsigned long long end_bit = s_carry;
    const unsigned long long data_bytes = (end_bit + 7 + 7) / 8;  // end-of-block code: 7 zero bits
    const unsigned long long stream_bytes = data_bytes + 4;       // + Adler-32
    const uint32_t chunks = (uint32_t)((stream_bytes + kIdat - 1) / kIdat);
    const uint32_t last_len = (uint32_t)(stream_bytes - (unsigned long long)kIdat * (chunks - 1));
    const unsigned long long file_bytes = kData0 + (unsigned long long)(chunks - 1) * kChunkStride + last_len + 4 + 12;
    const bool error = file_bytes > j.capacity || chunks > j.max_chunks || (stream_bytes + 3) / 4 > j.max_words;
    // Adler-32 of the scanline bytes: a = 1 + sum d, b = N + sum (N - k) d_k over stream
    // byte k; scanline r (bytes k = r*L + i) adds (N - r*L - L) * s0 + s1
    const unsigned long long n_bytes = (unsigned long long)j.height * j.row_bytes;
    unsigned long long a = 0, b = 0;
    for (uint32_t r = tid; r < j.height; r += kLayoutThreads) {
        const unsigned long long s0 = p.s0[j.row_base + r];
        const unsigned long long rest = (n_bytes - (unsigned long long)(r + 1) * j.row_bytes) % kAdlerMod;
        a = (a + s0) % kAdlerMod;
        b = (b + rest * (s0 % kAdlerMod) + p.s1[j.row_base + r] % kAdlerMod) % kAdlerMod;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        a += __shfl_xor_sync(0xFFFFFFFFu, a, o);
        b += __shfl_xor_sync(0xFFFFFFFFu, b, o);
    }
    if (lane == 0) {
        s_a[warp] = a % kAdlerMod;
        s_b[warp] = b % kAdlerMod;
    }
    __syncthreads();
    if (error) {
        if (tid == 0) {
            p.layout[blockIdx.x] = PngLayout{end_bit, stream_bytes, chunks, 0u, 1u, 0u};
            *j.size = 0ull;
        }
        return;
    }
    if ((uint32_t)tid < kHeadBytes / 4) reinterpret_cast<uint32_t*>(j.out)[tid] = j.header[tid];  // out is 16-byte aligned
    // IDAT chunk headers (length, type)
    for (uint32_t c = tid; c < chunks; c += kLayoutThreads) {
        uint8_t* h = j.out + kData0 + (size_t)c * kChunkStride - 8;
        put_be32(h, c + 1 < chunks ? kIdat : last_len);
        h[4] = 'I'; h[5] = 'D'; h[6] = 'A'; h[7] = 'T';
    }
    if (tid != 0) return;
    unsigned long long at = 0, bt = 0;
    for (int k = 0; k < kLayoutThreads / 32; ++k) {
        at += s_a[k];
        bt += s_b[k];
    }
    const uint32_t adler_a = (uint32_t)((1 + at) % kAdlerMod);
    const uint32_t adler_b = (uint32_t)((n_bytes % kAdlerMod + bt) % kAdlerMod);
    // IEND after the last chunk's CRC
    uint8_t* ie = j.out + kData0 + (size_t)(chunks - 1) * kChunkStride + last_len + 4;
    put_be32(ie, 0);
    ie[4] = 'I'; ie[5] = 'E'; ie[6] = 'N'; ie[7] = 'D';
    put_be32(ie + 8, kIendCrc);
    p.layout[blockIdx.x] = PngLayout{end_bit, stream_bytes, chunks, (adler_b << 16) | adler_a, 0u, 0u};
    *j.size = file_bytes;
}

// bits [b, b + n) (n <= 32) of a staged scanline
__device__ __forceinline__ uint32_t staged_bits(const uint32_t* __restrict__ slot, uint32_t b, uint32_t n) {
    const uint32_t k = b >> 5, sh = b & 31u;
    const unsigned long long two = (unsigned long long)__ldg(slot + k) | ((unsigned long long)__ldg(slot + k + 1) << 32);
    const uint32_t v = (uint32_t)(two >> sh);
    return n >= 32 ? v : (v & ((1u << n) - 1u));
}

// One block per group of p.group_rows scanlines of one image. The block writes the stream words
// that start inside the group's bits (the last group also the tail: end-of-block code, padding,
// Adler-32), each from the zlib and block headers (bits 0-18), the staged bits of the scanlines it
// covers and zeros. Positions are relative to the group's first bit, in 32 bits (a group holds at
// most 32 * (8 + 9 * 131072) = 37.7M bits): the stream's own are 64-bit, and their division into IDAT
// chunks cost more than the gather. 200 MB of files: 0.38 to 0.21 ms.
__global__ void __launch_bounds__(256, 6) png_pack_kernel(const __grid_constant__ PngParams p) {
    __shared__ uint32_t s_off[kMaxGroupRows + 1];  // each scanline's first bit; the group's end
    pdl_wait();
    pdl_release();
    const uint2 g = p.groups[blockIdx.x];
    const PngLayout& L = p.layout[g.x];
    if (L.error) return;
    const PngJob& j = p.jobs[g.x];
    const uint32_t r0 = g.y, nr = min(p.group_rows, j.height - r0);
    const unsigned long long* off = p.row_off + j.row_base;
    const uint32_t* bits = p.row_bits + j.row_base;
    const int tid = threadIdx.x;
    const unsigned long long base = off[r0];  // the scanlines' bits follow one another without gaps
    const bool last = r0 + nr >= j.height;
    const unsigned long long end = last ? L.end_bit : off[r0 + nr];
    if ((uint32_t)tid < nr) s_off[tid] = (uint32_t)(off[r0 + tid] - base);
    if (tid == 0) s_off[nr] = (uint32_t)(end - base);
    __syncthreads();
    const unsigned long long words = (L.stream_bytes + 3) / 4, data_bytes = L.stream_bytes - 4;
    const unsigned long long w_lo = r0 == 0 ? 0ull : (base + 31) / 32;
    const unsigned long long w_hi = last ? words : (end + 31) / 32;
    const uint32_t count = w_hi > w_lo ? (uint32_t)(w_hi - w_lo) : 0u;
    const uint32_t* slots = p.stage + j.stage_base + (size_t)r0 * j.row_words;
    const unsigned long long chunk0 = w_lo * 4 / kIdat;
    const uint32_t in_chunk = (uint32_t)(w_lo * 4 - chunk0 * kIdat);
    uint8_t* out = j.out + kData0 + (size_t)chunk0 * kChunkStride;
    const int skew = (int)(long long)(w_lo * 32 - base);  // word w_lo's first bit in the group (negative: the headers before it)
    uint32_t k = 0;  // this thread's scanline in the group, advanced as its words advance
    for (uint32_t i = (uint32_t)tid; i < count; i += 256) {
        const int b0 = skew + 32 * (int)i, b1 = b0 + 32;
        uint32_t word = 0u;
        while (k + 1 < nr && (int)s_off[k + 1] <= b0) ++k;
        if (b0 >= 0 && b1 <= (int)s_off[k + 1]) {  // inside one scanline
            word = staged_bits(slots + (size_t)k * j.row_words, (uint32_t)b0 - s_off[k], 32u);
        } else {
            if (r0 == 0 && i == 0) word = 0x78u | (0x01u << 8) | (0x3u << 16);
            for (uint32_t rr = k; r0 + rr < j.height; ++rr) {
                // past the group's scanlines only short ones can end inside this word
                const int rs = rr <= nr ? (int)s_off[rr] : (int)(off[r0 + rr] - base);
                if (rs >= b1) break;
                const int re = rr < nr ? (int)s_off[rr + 1] : rs + (int)bits[r0 + rr];
                const int s = max(rs, b0), e = min(re, b1);
                if (e <= s) continue;
                word |= staged_bits(slots + (size_t)rr * j.row_words, (uint32_t)(s - rs), (uint32_t)(e - s)) << (uint32_t)(s - b0);
            }
            const unsigned long long at = (w_lo + i) * 4;
            if (at + 4 > data_bytes) {  // Adler-32, most significant byte first, after the data
                for (int q = 0; q < 4; ++q) {
                    const unsigned long long byte = at + q;
                    if (byte >= data_bytes && byte < L.stream_bytes) {
                        const uint32_t v = (L.adler >> (24 - 8 * (uint32_t)(byte - data_bytes))) & 255u;
                        word = (word & ~(255u << (8 * q))) | (v << (8 * q));
                    }
                }
            }
        }
        const uint32_t to = in_chunk + 4 * i, c = to / kIdat;
        *reinterpret_cast<uint32_t*>(out + (size_t)c * kChunkStride + (to - c * kIdat)) = word;
    }
}

// a * b mod P, bit-reflected (bit 31 holds x^0)
__device__ __forceinline__ uint32_t gf_mul(uint32_t a, uint32_t b) {
    uint32_t prod = 0;
    for (int i = 0; i < 32; ++i) {
        if (a & (0x80000000u >> i)) prod ^= b;
        b = (b >> 1) ^ ((b & 1u) ? kCrcPoly : 0u);  // b * x
    }
    return prod;
}

// One block per IDAT chunk; the blocks walk the chunks of all images in order (image by
// image, so no block is launched for a chunk that does not exist). With the first word inverted
// (the initial value 0xFFFFFFFF), the CRC of N words is the sum of w_i x^(32 (N - i)): thread t takes
// the words t, t + 256, ... (whole lines per load), acc = acc x^(32 * 256) + w by four 256-entry
// tables, then shifts its sum to the end by one product; up to three last bytes follow. Each
// thread on a 256-byte part of its own, as a plain CRC needs it, read a line per lane and word
// and shifted its part by a chain of up to 20 products (200 MB of files 0.26 to 0.09 ms, one of
// 0.6 MB 26 to 11 us).
__global__ void __launch_bounds__(kCrcThreads) png_crc_kernel(const __grid_constant__ PngParams p) {
    __shared__ uint32_t s_t[4][256];
    __shared__ uint32_t s_part[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int t = 0; t < 4; ++t) {  // byte t of a word, kCrcThreads words on
        uint32_t v = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) v ^= (tid >> i & 1) ? p.stride[8 * t + i] : 0u;
        s_t[t][tid] = v;
    }
    pdl_wait();
    pdl_release();
    // chunks before each image (exclusive prefix) for images [tile, tile + kCrcJobs), and
    // the end of the tile; every block walks the same tiles in order
    __shared__ unsigned long long s_before[kCrcJobs + 1];
    __shared__ unsigned long long s_w[8];
    auto load_tile = [&](uint32_t first, unsigned long long before) {
        __syncthreads();  // the previous tile is no longer read
        const uint32_t n = min(kCrcJobs, p.jobs_n - first);
        constexpr int kPer = kCrcJobs / 256;
        uint32_t cnt[kPer];  // this thread's images
        unsigned long long mine = 0;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t i = (uint32_t)tid * kPer + q;
            cnt[q] = 0;
            if (i < n) {
                const PngLayout& L = p.layout[first + i];
                cnt[q] = L.error ? 0u : L.chunks;
            }
            mine += cnt[q];
        }
        unsigned long long incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_w[warp] = incl;
        __syncthreads();
        unsigned long long run = before + incl - mine;
        for (int q = 0; q < warp; ++q) run += s_w[q];
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t i = (uint32_t)tid * kPer + q;
            if (i < n) s_before[i] = run;
            run += cnt[q];
        }
        if ((uint32_t)tid == (n - 1) / kPer) s_before[n] = run;  // images past n added nothing
        __syncthreads();
    };
    uint32_t tile = 0;
    load_tile(0, 0);
    for (unsigned long long item = blockIdx.x;; item += gridDim.x) {
        uint32_t nt = min(kCrcJobs, p.jobs_n - tile);
        while (item >= s_before[nt] && tile + nt < p.jobs_n) {
            const unsigned long long end = s_before[nt];
            tile += nt;
            load_tile(tile, end);
            nt = min(kCrcJobs, p.jobs_n - tile);
        }
        if (item >= s_before[nt]) break;  // past the last chunk
        // the image of this item: the last one whose first chunk is <= item (images with no
        // chunks share their first-chunk index with the next one)
        uint32_t lo = 0, hi = nt;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s_before[mid] <= item) lo = mid; else hi = mid;
        }
        const uint32_t job = tile + lo;
        const unsigned long long first_chunk = s_before[lo];
        const PngLayout& L = p.layout[job];
        const uint32_t c = (uint32_t)(item - first_chunk);
        uint8_t* out = p.jobs[job].out;
        const uint32_t len = c + 1 < L.chunks ? kIdat : (uint32_t)(L.stream_bytes - (unsigned long long)kIdat * c);
        const uint8_t* start = out + kData0 + (size_t)c * kChunkStride - 4;  // type + data, 4-byte aligned
        const uint32_t n = (len + 4) / 4;  // whole words, the first of them the type
        const uint32_t* wp = reinterpret_cast<const uint32_t*>(start);
        uint32_t acc = 0, at = (uint32_t)tid;
        auto add = [&](uint32_t w) {
            acc = s_t[0][acc & 255u] ^ s_t[1][(acc >> 8) & 255u] ^ s_t[2][(acc >> 16) & 255u] ^ s_t[3][acc >> 24] ^ w;
        };
        for (; at + 7 * kCrcThreads < n; at += 8 * kCrcThreads) {
            uint32_t w[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) w[q] = wp[at + q * kCrcThreads];
            if (at == 0) w[0] = ~w[0];
#pragma unroll
            for (int q = 0; q < 8; ++q) add(w[q]);
        }
        for (; at < n; at += kCrcThreads) add(at == 0 ? ~wp[0] : wp[at]);
        // the thread's last word is d words before the end, 1 <= d <= kCrcThreads
        uint32_t part = at >= kCrcThreads ? gf_mul(acc, p.words[n - (at - kCrcThreads) - 1]) : 0u;
#pragma unroll
        for (int o = 16; o; o >>= 1) part ^= __shfl_xor_sync(0xFFFFFFFFu, part, o);
        if (lane == 0) s_part[warp] = part;
        __syncthreads();
        if (tid == 0) {
            uint32_t v = 0;
            for (int q = 0; q < 8; ++q) v ^= s_part[q];
            const uint32_t rest = (len + 4) & 3u;
            if (rest) {
                v = gf_mul(v, p.bytes[rest]);
                for (uint32_t q = 0; q < rest; ++q)  // byte q of `rest`: the low bits of a word, rest - q bytes before the end
                    v ^= gf_mul((uint32_t)start[4 * n + q], p.bytes[rest - q]);
            }
            v = ~v;
            uint8_t* o = out + kData0 + (size_t)c * kChunkStride + len;
            o[0] = (uint8_t)(v >> 24);
            o[1] = (uint8_t)(v >> 16);
            o[2] = (uint8_t)(v >> 8);
            o[3] = (uint8_t)v;
        }
        __syncthreads();  // s_part is rewritten by the next chunk
    }
}

}  // namespace axr

// ------------------------------------------------------------------ host side

using namespace axr;

namespace {

// CRC-32 on the host: the file headers' and the powers of x of the device's CRC pass.
struct Tables {
    uint32_t crc[256];
    uint32_t stride[32];
    uint32_t words[kCrcThreads];
    uint32_t bytes[4];
    static uint32_t mul(uint32_t a, uint32_t b) {
        uint32_t prod = 0;
        for (int i = 0; i < 32; ++i) {
            if (a & (0x80000000u >> i)) prod ^= b;
            b = (b >> 1) ^ ((b & 1u) ? kCrcPoly : 0u);
        }
        return prod;
    }
    Tables() {
        for (uint32_t n = 0; n < 256; ++n) {
            uint32_t c = n;
            for (int k = 0; k < 8; ++k) c = (c & 1u) ? (c >> 1) ^ kCrcPoly : c >> 1;
            crc[n] = c;
        }
        bytes[0] = 0x80000000u;  // x^0
        bytes[1] = 0x00800000u;  // x^8
        for (int k = 2; k < 4; ++k) bytes[k] = mul(bytes[k - 1], bytes[1]);
        words[0] = mul(bytes[2], bytes[2]);  // x^32
        for (uint32_t d = 1; d < kCrcThreads; ++d) words[d] = mul(words[d - 1], words[0]);
        for (int i = 0; i < 32; ++i) stride[i] = mul(1u << i, words[kCrcThreads - 1]);
    }
    // a PNG chunk of n data bytes at `at`: big-endian length, type and data (already there), CRC
    void seal(uint8_t* at, uint32_t n) const {
        auto be32 = [](uint8_t* to, uint32_t v) {
            for (int k = 0; k < 4; ++k) to[k] = (uint8_t)(v >> (24 - 8 * k));
        };
        be32(at, n);
        uint32_t c = 0xFFFFFFFFu;
        for (uint32_t i = 0; i < 4 + n; ++i) c = crc[(c ^ at[4 + i]) & 255u] ^ (c >> 8);
        be32(at + 8 + n, ~c);
    }
};

const Tables& tables() {
    static const Tables t;
    return t;
}

uint64_t row_bytes_of(uint32_t w, uint32_t ch) { return 1ull + (uint64_t)w * ch; }

// Signature, IHDR and tEXt chunks of a 1 x 1 RGB image: what every file's header starts from.
struct Header {
    uint8_t bytes[kHeadBytes] = {0x89, 'P', 'N', 'G', 0x0D, 0x0A, 0x1A, 0x0A};
    Header() {
        uint8_t* ih = bytes + 8;
        std::memcpy(ih + 4, "IHDR", 4);
        ih[11] = ih[15] = 1;
        ih[16] = 8;                      // bit depth
        ih[17] = 2;                      // colour type: RGB
        ih[18] = ih[19] = ih[20] = 0;    // deflate, adaptive filtering, no interlace
        tables().seal(ih, 13);
        uint8_t* tx = bytes + 33;
        std::memcpy(tx + 4, "tEXtSoftware\0AxiomR GB300 frame", 31);  // 27 data bytes after the type
        tables().seal(tx, 27);
    }
};

// The header of a width x height image: the size, the colour type and the IHDR's CRC. With all of it
// made anew for each, a call of many small images waited for the host (500 images of 64x64: 222 us a
// call, 186 with headers made on the device, 157 so).
void file_header(uint32_t width, uint32_t height, uint32_t channels, uint8_t* o) {
    static const Header base;
    std::memcpy(o, base.bytes, kHeadBytes);
    uint8_t* ih = o + 8;
    for (int k = 0; k < 4; ++k) {
        ih[8 + k] = (uint8_t)(width >> (24 - 8 * k));
        ih[12 + k] = (uint8_t)(height >> (24 - 8 * k));
    }
    ih[17] = channels == 4 ? 6 : 2;  // colour type: RGBA / RGB
    tables().seal(ih, 13);
}

// Scanlines per pack block of a call over `rows` scanlines: 8, or 32 where that leaves blocks for
// every SM several times over (a block's start is a chain of loads that 8 short scanlines do not
// pay for).
uint32_t group_share(uint64_t rows, int num_sms) {
    return rows >= 12ull * (uint64_t)num_sms * kMaxGroupRows ? kMaxGroupRows : kGroupRows;
}

}  // namespace

namespace {
void release_batch(axr_png_batch* b);
}

namespace axr_internal {

// Scanline scratch, the job table and the pinned staging of axr_framebuffers_encode_png,
// plus the device file buffers and pinned sizes of axr_framebuffers_read_png.
struct PngState {
    uint32_t row_cap = 0, job_cap = 0;
    size_t stage_cap = 0;  // words
    uint32_t* stage = nullptr;
    uint32_t* row_bits = nullptr;
    uint32_t* s0 = nullptr;
    unsigned long long* s1 = nullptr;
    unsigned long long* row_off = nullptr;
    PngJob* jobs = nullptr;
    PngLayout* layout = nullptr;
    uint32_t group_cap = 0;
    uint2* groups = nullptr;
    // pinned host tables, two used in turn so that a call does not wait for the upload of
    // the one before (that upload sits behind the work already on the stream)
    PngJob* jobs_host[2] = {};
    uint2* groups_host[2] = {};
    cudaEvent_t tables_free[2] = {};
    int next = 0;
    axr_png_batch* readback = nullptr;  // axr_framebuffers_read_png
    std::mutex readback_mu;             // held for a whole axr_framebuffers_read_png call
};

void free_png(axr_context* ctx) {
    PngState* s = ctx->png;
    if (!s) return;
    dfree(s->stage);
    dfree(s->row_bits);
    dfree(s->s0);
    dfree(s->s1);
    dfree(s->row_off);
    dfree(s->jobs);
    dfree(s->layout);
    dfree(s->groups);
    for (int t = 0; t < 2; ++t) {
        if (s->groups_host[t]) cudaFreeHost(s->groups_host[t]);
        if (s->jobs_host[t]) cudaFreeHost(s->jobs_host[t]);
        if (s->tables_free[t]) cudaEventDestroy(s->tables_free[t]);
    }
    if (s->readback) release_batch(s->readback);
    delete s;
    ctx->png = nullptr;
}

}  // namespace axr_internal

namespace {

// staging words per scanline: its worst case (filter byte + 9 bits per byte) + one word
// that the pack pass may read past the end
uint32_t row_words_of(uint32_t w, uint32_t ch) {
    return (uint32_t)((8 + 9ull * w * ch + 31) / 32 + 1);
}

axr_status grow_png(axr_context* ctx, uint32_t rows, uint32_t jobs, size_t stage_words, uint32_t groups) {
    if (!ctx->png) ctx->png = new PngState();
    PngState* s = ctx->png;
    for (int t = 0; t < 2; ++t)
        if (!s->tables_free[t]) AXR_CUDA(ctx, cudaEventCreateWithFlags(&s->tables_free[t], cudaEventDisableTiming));
    if (rows > s->row_cap) {
        AXR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        dfree(s->row_bits); dfree(s->s0); dfree(s->s1); dfree(s->row_off);
        s->row_bits = nullptr; s->s0 = nullptr; s->s1 = nullptr; s->row_off = nullptr;
        s->row_cap = 0;
        const uint32_t cap = std::max(rows, 4096u);
        AXR_CUDA(ctx, dmalloc(&s->row_bits, cap));
        AXR_CUDA(ctx, dmalloc(&s->s0, cap));
        AXR_CUDA(ctx, dmalloc(&s->s1, cap));
        AXR_CUDA(ctx, dmalloc(&s->row_off, cap));
        s->row_cap = cap;
    }
    if (stage_words > s->stage_cap) {
        AXR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        dfree(s->stage);
        s->stage = nullptr;
        s->stage_cap = 0;
        AXR_CUDA(ctx, dmalloc(&s->stage, stage_words));
        s->stage_cap = stage_words;
    }
    if (groups > s->group_cap) {
        AXR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        dfree(s->groups);
        s->groups = nullptr;
        for (int t = 0; t < 2; ++t) {
            if (s->groups_host[t]) cudaFreeHost(s->groups_host[t]);
            s->groups_host[t] = nullptr;
        }
        s->group_cap = 0;
        const uint32_t cap = std::max(groups, 1024u);
        AXR_CUDA(ctx, dmalloc(&s->groups, cap));
        for (int t = 0; t < 2; ++t)
            AXR_CUDA(ctx, cudaMallocHost(reinterpret_cast<void**>(&s->groups_host[t]), sizeof(uint2) * cap));
        s->group_cap = cap;
    }
    if (jobs > s->job_cap) {
        AXR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        dfree(s->jobs); dfree(s->layout);
        s->jobs = nullptr; s->layout = nullptr;
        for (int t = 0; t < 2; ++t) {
            if (s->jobs_host[t]) cudaFreeHost(s->jobs_host[t]);
            s->jobs_host[t] = nullptr;
        }
        s->job_cap = 0;
        const uint32_t cap = std::max(jobs, 64u);
        AXR_CUDA(ctx, dmalloc(&s->jobs, cap));
        AXR_CUDA(ctx, dmalloc(&s->layout, cap));
        for (int t = 0; t < 2; ++t)
            AXR_CUDA(ctx, cudaMallocHost(reinterpret_cast<void**>(&s->jobs_host[t]), sizeof(PngJob) * cap));
        s->job_cap = cap;
    }
    return AXR_OK;
}

// The encode of `count` framebuffers into device buffers; the caller holds ctx->mu. `sized`: recorded
// where the sizes are known, before the files are.
axr_status encode_locked(axr_context* ctx, int32_t count, const axr_framebuffer* const* fbs, uint32_t channels,
                         void* const* out, const uint64_t* capacity, unsigned long long* sizes, cudaEvent_t sized = nullptr) {
    if (channels != 3 && channels != 4) return fail(ctx, AXR_E_INVALID, "channels must be 3 (RGB) or 4 (RGBA)");
    if (count < 0 || (count > 0 && (!fbs || !out || !capacity || !sizes)))
        return fail(ctx, AXR_E_INVALID, "bad framebuffer or buffer list");
    if (count == 0) return AXR_OK;
    uint64_t rows = 0, groups = 0;
    size_t stage_words = 0;
    for (int32_t i = 0; i < count; ++i) {
        const axr_framebuffer* fb = fbs[i];
        if (!fb) return fail(ctx, AXR_E_INVALID, "framebuffer %d is NULL", i);
        if (fb->device != ctx->device) return fail(ctx, AXR_E_INVALID, "framebuffer %d is on another device", i);
        if (!out[i] || (reinterpret_cast<uintptr_t>(out[i]) & 15u))
            return fail(ctx, AXR_E_INVALID, "output buffer %d is NULL or not 16-byte aligned", i);
        const uint64_t bound = axr_png_bound((uint32_t)fb->width, (uint32_t)fb->height, channels);
        if (capacity[i] < bound)
            return fail(ctx, AXR_E_INVALID, "output buffer %d holds %llu bytes, the encode may need %llu", i,
                        (unsigned long long)capacity[i], (unsigned long long)bound);
        rows += (uint64_t)fb->height;
        stage_words += (size_t)fb->height * row_words_of((uint32_t)fb->width, channels);
    }
    const uint32_t group_rows = group_share(rows, ctx->cfg.num_sms);
    for (int32_t i = 0; i < count; ++i) groups += ((uint64_t)fbs[i]->height + group_rows - 1) / group_rows;
    if (rows > 0xFFFFFFFFull || count > 65535) return fail(ctx, AXR_E_INVALID, "too many scanlines or images in one call");
    axr_status st = grow_png(ctx, (uint32_t)rows, (uint32_t)count, stage_words + 64, (uint32_t)groups);
    if (st != AXR_OK) return st;
    PngState* s = ctx->png;
    const int tb = s->next;
    s->next ^= 1;
    AXR_CUDA(ctx, cudaEventSynchronize(s->tables_free[tb]));  // the upload two calls ago has been read
    PngJob* jobs_host = s->jobs_host[tb];
    uint2* groups_host = s->groups_host[tb];
    uint32_t row = 0;
    uint64_t chunks = 0;
    unsigned long long stage = 0;
    for (int32_t i = 0; i < count; ++i) {
        const axr_framebuffer* fb = fbs[i];
        PngJob& j = jobs_host[i];
        const uint64_t bound = axr_png_bound((uint32_t)fb->width, (uint32_t)fb->height, channels);
        j.color = fb->color;
        j.out = static_cast<uint8_t*>(out[i]);
        j.size = sizes + i;
        j.capacity = capacity[i];
        j.width = (uint32_t)fb->width;
        j.height = (uint32_t)fb->height;
        j.channels = channels;
        j.row_bytes = (uint32_t)row_bytes_of(j.width, channels);
        j.row_words = row_words_of(j.width, channels);
        j.stage_base = stage;
        j.row_base = row;
        j.max_chunks = (uint32_t)((bound - kData0 - 16) / kChunkStride);
        j.max_words = ((unsigned long long)j.max_chunks * kIdat + 3) / 4;
        if (i > 0 && j.width == jobs_host[i - 1].width && j.height == jobs_host[i - 1].height)
            std::memcpy(j.header, jobs_host[i - 1].header, kHeadBytes);
        else
            file_header(j.width, j.height, channels, reinterpret_cast<uint8_t*>(j.header));
        chunks += j.max_chunks;
        row += j.height;
        stage += (unsigned long long)j.height * j.row_words;
    }
    uint32_t ng = 0;
    for (int32_t i = 0; i < count; ++i)
        for (uint32_t r = 0; r < jobs_host[i].height; r += group_rows) groups_host[ng++] = make_uint2((uint32_t)i, r);
    AXR_CUDA(ctx, cudaMemcpyAsync(s->jobs, jobs_host, sizeof(PngJob) * (size_t)count, cudaMemcpyHostToDevice, ctx->stream));
    AXR_CUDA(ctx, cudaMemcpyAsync(s->groups, groups_host, sizeof(uint2) * ng, cudaMemcpyHostToDevice, ctx->stream));
    AXR_CUDA(ctx, cudaEventRecord(s->tables_free[tb], ctx->stream));
    PngParams p{};
    p.jobs = s->jobs;
    p.layout = s->layout;
    p.stage = s->stage;
    p.row_bits = s->row_bits;
    p.s0 = s->s0;
    p.s1 = s->s1;
    p.row_off = s->row_off;
    p.jobs_n = (uint32_t)count;
    p.rows = row;
    p.group_rows = group_rows;
    std::memcpy(p.stride, tables().stride, sizeof(p.stride));
    std::memcpy(p.words, tables().words, sizeof(p.words));
    std::memcpy(p.bytes, tables().bytes, sizeof(p.bytes));
    p.groups = s->groups;
    const unsigned row_blocks = (row + kPngWarps - 1) / kPngWarps;
    if (channels == 4) png_rows_kernel<4><<<row_blocks, 32 * kPngWarps, 0, ctx->stream>>>(p);
    else png_rows_kernel<3><<<row_blocks, 32 * kPngWarps, 0, ctx->stream>>>(p);
    AXR_CUDA(ctx, cudaGetLastError());
    AXR_CUDA(ctx, launch_dependent(png_layout_kernel, (unsigned)count, (unsigned)kLayoutThreads, ctx->stream, p));
    if (sized) AXR_CUDA(ctx, cudaEventRecord(sized, ctx->stream));
    AXR_CUDA(ctx, launch_dependent(png_pack_kernel, (unsigned)ng, 256u, ctx->stream, p));
    // a block per chunk, up to 8 per SM (each builds its tables first)
    AXR_CUDA(ctx, launch_dependent(png_crc_kernel, (unsigned)std::min<uint64_t>(chunks, (uint64_t)ctx->cfg.num_sms * 8u),
                                   (unsigned)kCrcThreads, ctx->stream, p));
    ctx->launches += 4;
    return AXR_OK;
}

}  // namespace

extern "C" uint64_t axr_png_bound(uint32_t width, uint32_t height, uint32_t channels) {
    if (width == 0 || height == 0 || (channels != 3 && channels != 4)) return 0;
    // a literal costs at most 9 bits and a match is taken only when it costs fewer bits
    // than the literals it replaces
    const uint64_t bits = kHeaderBits + (uint64_t)height * (8 + 9 * (uint64_t)width * channels);
    const uint64_t stream = (bits + 7 + 7) / 8 + 4;
    const uint64_t chunks = (stream + kIdat - 1) / kIdat;
    return kData0 + chunks * kChunkStride + 16;
}

extern "C" axr_status axr_framebuffers_encode_png(axr_context* ctx, int32_t count, const axr_framebuffer* const* fbs,
                                                  uint32_t channels, void* const* out, const uint64_t* capacity,
                                                  uint64_t* sizes) {
    NvtxRange nvtx_range("axr_framebuffers_encode_png");
    if (!ctx) return fail(nullptr, AXR_E_INVALID, "context is NULL");
    std::lock_guard<std::mutex> lk(ctx->mu);
    DeviceGuard g(ctx->device);
    static_assert(sizeof(uint64_t) == sizeof(unsigned long long), "size array element");
    return encode_locked(ctx, count, fbs, channels, out, capacity, reinterpret_cast<unsigned long long*>(sizes));
}

// A set of PNG files on the device, their sizes written to pinned memory by the layout pass, and
// its own copy streams, so that the files of one batch come back to the host while the next batch
// renders and encodes on the context stream. The sizes are known before the files are written, so that a
// caller's copies are enqueued while the last passes run (1080p screenshot 87.5 to 69.7 us,
// with the copy of the sizes and the waits on unused streams gone).
struct axr_png_batch {
    int device = 0;
    uint8_t* files = nullptr;
    size_t files_cap = 0;
    unsigned long long* sizes_host = nullptr;  // pinned
    uint32_t sizes_cap = 0;
    std::vector<size_t> at;  // file i at files + at[i]
    int32_t count = 0;
    bool encoded = false;
    cudaEvent_t sized = nullptr;  // the sizes are on the host (context stream)
    cudaEvent_t done = nullptr;   // the files are written (context stream)
    static constexpr int kStreams = 4;
    cudaStream_t copy[kStreams] = {};
    cudaEvent_t copied[kStreams] = {};
};

namespace {

void release_batch(axr_png_batch* b) {
    for (int k = 0; k < axr_png_batch::kStreams; ++k) {
        if (b->copy[k]) {
            cudaStreamSynchronize(b->copy[k]);
            cudaStreamDestroy(b->copy[k]);
        }
        if (b->copied[k]) cudaEventDestroy(b->copied[k]);
    }
    if (b->done) {
        cudaEventSynchronize(b->done);
        cudaEventDestroy(b->done);
    }
    if (b->sized) cudaEventDestroy(b->sized);
    dfree(b->files);
    if (b->sizes_host) cudaFreeHost(b->sizes_host);
    delete b;
}

axr_status create_batch(axr_context* ctx, axr_png_batch** out) {
    axr_png_batch* b = new axr_png_batch();
    b->device = ctx->device;
    cudaError_t e = cudaEventCreateWithFlags(&b->done, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->sized, cudaEventDisableTiming);
    for (int k = 0; e == cudaSuccess && k < axr_png_batch::kStreams; ++k) {
        e = cudaStreamCreateWithFlags(&b->copy[k], cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->copied[k], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) {
        release_batch(b);
        return cuda_fail(ctx, e, "PNG batch streams");
    }
    *out = b;
    return AXR_OK;
}

// Enqueue the encode of `count` framebuffers into b on the context stream; the caller holds
// ctx->mu.
axr_status batch_encode_locked(axr_context* ctx, axr_png_batch* b, int32_t count, const axr_framebuffer* const* fbs,
                               uint32_t channels) {
    if (channels != 3 && channels != 4) return fail(ctx, AXR_E_INVALID, "channels must be 3 (RGB) or 4 (RGBA)");
    if (count < 0 || (count > 0 && !fbs)) return fail(ctx, AXR_E_INVALID, "bad framebuffer list");
    std::vector<uint64_t> cap((size_t)count);
    b->at.assign((size_t)count + 1, 0);
    for (int32_t i = 0; i < count; ++i) {
        if (!fbs[i]) return fail(ctx, AXR_E_INVALID, "framebuffer %d is NULL", i);
        cap[i] = axr_png_bound((uint32_t)fbs[i]->width, (uint32_t)fbs[i]->height, channels);
        b->at[i + 1] = b->at[i] + ((cap[i] + 255) & ~uint64_t(255));
    }
    // the batch's earlier files must have been copied out before they are overwritten
    for (int k = 0; k < axr_png_batch::kStreams; ++k) AXR_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, b->copied[k], 0));
    if (b->at[count] > b->files_cap) {
        AXR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        dfree(b->files);
        b->files = nullptr;
        b->files_cap = 0;
        AXR_CUDA(ctx, dmalloc(&b->files, b->at[count]));
        b->files_cap = b->at[count];
    }
    if ((uint32_t)count > b->sizes_cap) {
        AXR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (b->sizes_host) cudaFreeHost(b->sizes_host);
        b->sizes_host = nullptr;
        b->sizes_cap = 0;
        AXR_CUDA(ctx, cudaMallocHost(reinterpret_cast<void**>(&b->sizes_host), sizeof(unsigned long long) * count));
        b->sizes_cap = (uint32_t)count;
    }
    b->count = count;
    b->encoded = false;
    if (count == 0) return AXR_OK;
    std::vector<void*> out((size_t)count);
    for (int32_t i = 0; i < count; ++i) out[i] = b->files + b->at[i];
    axr_status st = encode_locked(ctx, count, fbs, channels, out.data(), cap.data(), b->sizes_host, b->sized);
    if (st != AXR_OK) return st;
    AXR_CUDA(ctx, cudaEventRecord(b->done, ctx->stream));
    b->encoded = true;
    return AXR_OK;
}

axr_status batch_sizes(axr_context* ctx, axr_png_batch* b, uint64_t* sizes) {
    if (!b->encoded) return b->count == 0 ? AXR_OK : fail(ctx, AXR_E_INVALID, "the PNG batch holds no encode");
    DeviceGuard g(b->device);
    AXR_CUDA(ctx, cudaEventSynchronize(b->sized));
    for (int32_t i = 0; i < b->count; ++i) {
        if (b->sizes_host[i] == 0) return fail(ctx, AXR_E_CUDA, "framebuffer %d: encode overflow", i);
        if (sizes) sizes[i] = b->sizes_host[i];
    }
    return AXR_OK;
}

axr_status batch_read(axr_context* ctx, axr_png_batch* b, void* const* files, const uint64_t* capacity) {
    axr_status st = batch_sizes(ctx, b, nullptr);
    if (st != AXR_OK || b->count == 0) return st;
    if (!files) return fail(ctx, AXR_E_INVALID, "no host buffers");
    for (int32_t i = 0; i < b->count; ++i)
        if (files[i] && capacity && capacity[i] < b->sizes_host[i])
            return fail(ctx, AXR_E_INVALID, "host buffer %d holds %llu bytes, the file has %llu", i,
                        (unsigned long long)capacity[i], b->sizes_host[i]);
    DeviceGuard g(b->device);
    const int streams = std::min<int>(b->count, axr_png_batch::kStreams);
    for (int k = 0; k < streams; ++k) AXR_CUDA(ctx, cudaStreamWaitEvent(b->copy[k], b->done, 0));
    for (int32_t i = 0; i < b->count; ++i) {
        if (!files[i]) continue;
        AXR_CUDA(ctx, cudaMemcpyAsync(files[i], b->files + b->at[i], b->sizes_host[i], cudaMemcpyDeviceToHost,
                                      b->copy[i % axr_png_batch::kStreams]));
    }
    for (int k = 0; k < streams; ++k) AXR_CUDA(ctx, cudaEventRecord(b->copied[k], b->copy[k]));
    for (int k = 0; k < streams; ++k) AXR_CUDA(ctx, cudaEventSynchronize(b->copied[k]));
    return AXR_OK;
}

}  // namespace

namespace axr_internal {

axr_status png_batch_create(axr_context* ctx, axr_png_batch** out) { return create_batch(ctx, out); }

void png_batch_release(axr_png_batch* b) {
    if (b) release_batch(b);
}

axr_status png_batch_encode_locked(axr_context* ctx, axr_png_batch* b, int32_t count,
                                   const axr_framebuffer* const* fbs, uint32_t channels) {
    return batch_encode_locked(ctx, b, count, fbs, channels);
}

cudaError_t png_batch_query(const axr_png_batch* b) {
    return b->encoded ? cudaEventQuery(b->done) : cudaSuccess;
}

void png_batch_file(const axr_png_batch* b, int32_t i, const void** dev, uint64_t* size) {
    *dev = b->files + b->at[(size_t)i];
    *size = b->sizes_host[i];
}

}  // namespace axr_internal

extern "C" axr_status axr_png_batch_create(axr_context* ctx, axr_png_batch** out) {
    if (!ctx || !out) return fail(ctx, AXR_E_INVALID, "NULL argument");
    std::lock_guard<std::mutex> lk(ctx->mu);
    DeviceGuard g(ctx->device);
    return create_batch(ctx, out);
}

extern "C" void axr_png_batch_destroy(axr_context* ctx, axr_png_batch* b) {
    if (!b) return;
    DeviceGuard g(b->device);
    release_batch(b);
}

extern "C" axr_status axr_png_batch_encode(axr_context* ctx, axr_png_batch* b, int32_t count,
                                           const axr_framebuffer* const* fbs, uint32_t channels) {
    NvtxRange nvtx_range("axr_png_batch_encode");
    if (!ctx || !b) return fail(ctx, AXR_E_INVALID, "NULL argument");
    if (b->device != ctx->device) return fail(ctx, AXR_E_INVALID, "the PNG batch belongs to another device");
    std::lock_guard<std::mutex> lk(ctx->mu);
    DeviceGuard g(ctx->device);
    return batch_encode_locked(ctx, b, count, fbs, channels);
}

extern "C" axr_status axr_png_batch_sizes(axr_context* ctx, axr_png_batch* b, uint64_t* sizes) {
    if (!ctx || !b || !sizes) return fail(ctx, AXR_E_INVALID, "NULL argument");
    return batch_sizes(ctx, b, sizes);
}

extern "C" axr_status axr_png_batch_read(axr_context* ctx, axr_png_batch* b, void* const* files,
                                         const uint64_t* capacity) {
    if (!ctx || !b) return fail(ctx, AXR_E_INVALID, "NULL argument");
    return batch_read(ctx, b, files, capacity);
}

extern "C" axr_status axr_framebuffers_read_png(axr_context* ctx, int32_t count, const axr_framebuffer* const* fbs,
                                                uint32_t channels, void* const* files, const uint64_t* capacity,
                                                uint64_t* sizes) {
    NvtxRange nvtx_range("axr_framebuffers_read_png");
    if (!ctx) return fail(nullptr, AXR_E_INVALID, "context is NULL");
    if (count < 0 || (count > 0 && (!fbs || !sizes))) return fail(ctx, AXR_E_INVALID, "bad framebuffer list");
    if (channels != 3 && channels != 4) return fail(ctx, AXR_E_INVALID, "channels must be 3 (RGB) or 4 (RGBA)");
    if (count == 0) return AXR_OK;
    axr_png_batch* b;
    PngState* ps;
    {
        std::lock_guard<std::mutex> lk(ctx->mu);
        if (!ctx->png) ctx->png = new PngState();
        ps = ctx->png;
    }
    // the internal batch serves one call at a time (lock order: readback_mu, then ctx->mu)
    std::lock_guard<std::mutex> whole(ps->readback_mu);
    {
        std::lock_guard<std::mutex> lk(ctx->mu);
        DeviceGuard g(ctx->device);
        if (!ctx->png->readback) {
            axr_status st = create_batch(ctx, &ctx->png->readback);
            if (st != AXR_OK) return st;
        }
        b = ctx->png->readback;
        axr_status st = batch_encode_locked(ctx, b, count, fbs, channels);
        if (st != AXR_OK) return st;
    }
    axr_status st = batch_sizes(ctx, b, sizes);
    if (st != AXR_OK || !files) return st;
    for (int32_t i = 0; i < count; ++i)
        if (files[i] && capacity && capacity[i] < sizes[i])
            return fail(ctx, AXR_E_INVALID, "a host buffer is smaller than its file (sizes returned)");
    return batch_read(ctx, b, files, capacity);
}
