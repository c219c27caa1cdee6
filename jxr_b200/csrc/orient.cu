// orient.cu -- the presentation orientation of a decoded surface on the GPU.
//
// The reference applies an image's orientation (EXIF-like: mirrors,
// rotations, transposes) to the decoded host samples after the decode
// (apply_orientation, crates/jxr/src/decoder/orientation.rs:5-211, called by
// JxrDecoder::decode_oriented, crates/jxr/src/decoder.rs:327-333).  Here it is
// a device pass over the surface the engine left in HBM: each CTA writes one
// tile of the oriented surface, reading the source rectangle that tile comes
// from into shared memory first, so that both the reads and the writes run
// along rows.  Pixels move whole, their channels in order; one-bit luma (rows
// padded to bytes, most significant bit first) moves bit by bit.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/jxr_b200.h"
#include "orient_tile.h"

namespace jxr {
jxrb_status report_error(jxrb_status s, const char *why);
jxrb_status report_cuda(cudaError_t e, const char *what);
}  // namespace jxr

namespace {

using jxr::source_of;
using jxr::swaps_axes;

constexpr int kTile = 32;
constexpr uint32_t kMaxPixelBytes = 48;   // a 32 x 32 tile of them fills 48 KB of shared memory

// One destination tile of 32 x 32 pixels, `words` words of type W a pixel.
// The source pixels of a tile form a rectangle of at most 32 x 32 (every
// orientation maps rows and columns to rows or columns); it is staged in
// shared memory, then written out along destination rows.
template <typename W>
__global__ void __launch_bounds__(256) jxrb_orient_tiles(const W *__restrict__ src, W *__restrict__ dst, uint32_t w,
                                                        uint32_t h, uint32_t words, int o) {
    extern __shared__ __align__(16) unsigned char orient_smem[];
    W *tile = reinterpret_cast<W *>(orient_smem);
    const bool swap = swaps_axes(o);
    const uint32_t ow = swap ? h : w, oh = swap ? w : h;
    const uint32_t dx0 = blockIdx.x * kTile, dy0 = blockIdx.y * kTile;
    const uint32_t dx1 = min(dx0 + kTile, ow), dy1 = min(dy0 + kTile, oh);
    // the source rectangle: the extremes of the tile's corners
    uint32_t ax, ay, bx, by;
    source_of(o, w, h, dx0, dy0, ax, ay);
    source_of(o, w, h, dx1 - 1, dy1 - 1, bx, by);
    const uint32_t sx0 = min(ax, bx), sy0 = min(ay, by), sx1 = max(ax, bx) + 1, sy1 = max(ay, by) + 1;
    const uint32_t sw = sx1 - sx0, sh = sy1 - sy0;
    const uint32_t row_words = sw * words;
    for (uint32_t i = threadIdx.x; i < row_words * sh; i += blockDim.x) {
        const uint32_t r = i / row_words, c = i - r * row_words;
        tile[i] = src[((size_t)(sy0 + r) * w + sx0) * words + c];
    }
    __syncthreads();
    const uint32_t dw = dx1 - dx0, out_words = dw * words;
    for (uint32_t i = threadIdx.x; i < out_words * (dy1 - dy0); i += blockDim.x) {
        const uint32_t r = i / out_words, c = i - r * out_words;
        const uint32_t px = c / words, k = c - px * words;
        uint32_t sx, sy;
        source_of(o, w, h, dx0 + px, dy0 + r, sx, sy);
        dst[((size_t)(dy0 + r) * ow + dx0) * words + c] = tile[((sy - sy0) * sw + (sx - sx0)) * words + k];
    }
}

// Orientation of the usual pixel sizes (PB bytes, a template argument, so that
// no division by a runtime size is left).  The bound is the memory traffic;
// what has to be kept off the issue slots is the byte shuffling of pixels that
// are no whole words on rows that start at any byte.  Three passes over a
// T x T-pixel tile:
//   1. source rows into shared memory as the aligned words they lie in (bytes
//      only at a row's two ends).  Row r starts at byte (a + r * S), S chosen
//      equal to the source's row pitch modulo 4, so a pixel's address stays
//      linear in its row and column, and S / 4 about odd, so that walking a
//      column meets distinct banks;
//   2. each thread gathers G pixels that make whole destination words (four
//      3-byte pixels make three) and stores those words to a second tile laid
//      out as the destination rows are, alignment included;
//   3. that tile out to the destination rows in aligned words, bytes only at
//      the rows' ends: full sectors leave the SM once.
// T keeps both tiles in about 33 KB (6 to 8 CTAs an SM in flight) and a row
// segment of 128 bytes or more for most sizes.
// 3999 x 2999 RGB8, ROTATE90: 112.7 us with one byte a word and two divisions
// each (91.5 M warp instructions), 28.5 us here (18.4 M).
template <int PB>
struct OrientShape {
    static constexpr int kUnit = PB % 4 == 0 ? 4 : PB % 2 == 0 ? 2 : 1;   // bytes moved together
    static constexpr int kGroup = 4 / kUnit;                               // pixels of whole words
    static constexpr int kWords = kGroup * PB / 4;                         // words of a group
    static constexpr int kSide = PB <= 4 ? 64 : 32;                        // pixels across / down a tile
    static constexpr int kInWords = kSide * (kSide * PB + 8) / 4 + 1;      // S <= kSide * PB + 7, first byte <= 3
    static constexpr int kOutPitch = kSide * PB + 4;                       // bytes, whole words
};

template <int PB>
__global__ void __launch_bounds__(256) jxrb_orient_pixels(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst,
                                                         uint32_t w, uint32_t h, int o) {
    using Sh = OrientShape<PB>;
    constexpr int T = Sh::kSide, U = Sh::kUnit, G = Sh::kGroup, NW = Sh::kWords;
    __shared__ uint32_t in_words[Sh::kInWords];
    __shared__ uint32_t out_words[T * Sh::kOutPitch / 4];
    uint8_t *const in = reinterpret_cast<uint8_t *>(in_words);
    uint8_t *const outb = reinterpret_cast<uint8_t *>(out_words);
    const bool swap = swaps_axes(o);
    const uint32_t ow = swap ? h : w;
    const uint32_t dx0 = blockIdx.x * T, dy0 = blockIdx.y * T;
    const jxr::OrientTile tile = jxr::orient_tile(o, w, h, T, dx0, dy0);
    const int dw = tile.dw, dh = tile.dh, sw = tile.sw, sh = tile.sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // pass 1: a lane's words of all its rows are loaded before the first is
    // stored, so that they are in flight together (one row at a time, with the
    // rows' ends by the byte, took 88 us: a chain of load latencies).  A word
    // may hold bytes of the neighbouring pixels too; a tile whose first or last
    // word reaches outside the surface (words_inside) reads it by the byte.
    // A warp's rows are eight apart, so they all start at the same byte of a
    // word.
    constexpr int kRowWords = U == 4 ? T * PB / 4 : T * PB / 4 + 1, kLaneWords = (kRowWords + 31) / 32;
    const size_t pitch = (size_t)w * PB;
    const size_t offset = tile.sy0 * pitch + (size_t)tile.sx0 * PB;
    const uint8_t *first = src + offset;
    // (units of whole words start and end on their boundaries)
    const bool by_word = U == 4 || jxr::words_inside(reinterpret_cast<uintptr_t>(src), h * pitch, offset, pitch, sw * PB, sh);
    const int a = (int)(reinterpret_cast<uintptr_t>(first) & 3);
    const int S = T * PB + 4 + (int)(pitch & 3);
    {
        const int mis = (a + warp * S) & 3, n = mis + sw * PB;
        const uint8_t *row = first + warp * pitch - mis;
        uint32_t held[T / 8][kLaneWords];
        if (by_word) {
#pragma unroll
            for (int j = 0; j < T / 8; j++, row += 8 * pitch)
#pragma unroll
                for (int q = 0; q < kLaneWords; q++)
                    if (warp + 8 * j < sh && 4 * (lane + 32 * q) < n)
                        held[j][q] = __ldg(reinterpret_cast<const uint32_t *>(row) + lane + 32 * q);
        } else {
            for (int j = 0; j < T / 8; j++, row += 8 * pitch) {
                if (warp + 8 * j >= sh) break;
                for (int q = 0; q < kLaneWords; q++) {
                    const int k = 4 * (lane + 32 * q);
                    for (int b = max(k, mis); b < min(k + 4, n); b++) in[a + (warp + 8 * j) * S - mis + b] = __ldg(row + b);
                }
            }
        }
        if (by_word) {
            uint32_t *to = in_words + ((a + warp * S) >> 2) + lane;
#pragma unroll
            for (int j = 0; j < T / 8; j++, to += 2 * S)
#pragma unroll
                for (int q = 0; q < kLaneWords; q++)
                    if (warp + 8 * j < sh && 4 * (lane + 32 * q) < n) to[32 * q] = held[j][q];
        }
    }
    __syncthreads();
    // pass 2: destination pixel (p, r) is at corner + p * step_p + r * step_r.
    // A thread's groups are a multiple of four rows apart, at the same byte of
    // a word.
    const bool flip_p = o == JXRB_ORIENT_MIRROR_HORIZONTAL || o == JXRB_ORIENT_ROTATE180 ||
                        o == JXRB_ORIENT_ROTATE90 || o == JXRB_ORIENT_TRANSVERSE;
    const bool flip_r = o == JXRB_ORIENT_ROTATE180 || o == JXRB_ORIENT_MIRROR_VERTICAL ||
                        o == JXRB_ORIENT_TRANSVERSE || o == JXRB_ORIENT_ROTATE270;
    const int unit_p = swap ? S : PB, unit_r = swap ? PB : S;
    const int step_p = flip_p ? -unit_p : unit_p, step_r = flip_r ? -unit_r : unit_r;
    const uint8_t *corner = in + a + (flip_p ? (dw - 1) * unit_p : 0) + (flip_r ? (dh - 1) * unit_r : 0);
    uint8_t *out = dst + ((size_t)dy0 * ow + dx0) * PB;
    const size_t opitch = (size_t)ow * PB;
    const int out0 = (int)(reinterpret_cast<uintptr_t>(out) & 3), om = (int)(opitch & 3);
    // the first pixel of a row whose first byte starts a word, in a row whose
    // first byte is byte d of one: PB * p = -d (mod 4)
    auto head = [&](int d) { return G == 1 ? 0 : PB % 4 == 1 ? (-d & 3) : PB % 4 == 3 ? (d & 3) : (d >> 1) & 1; };
    {
        constexpr int kRows = 256 / (T / G);
        static_assert(kRows % 4 == 0, "a thread's rows share their alignment");
        const int r0 = threadIdx.x / (T / G), g = threadIdx.x % (T / G);
        const int d = (out0 + r0 * om) & 3, p0 = head(d) + g * G;
        const uint8_t *q = corner + r0 * step_r + p0 * step_p;
        uint32_t *to = out_words + r0 * (Sh::kOutPitch / 4) + ((d + p0 * PB) >> 2);
        if (p0 + G <= dw) {
#pragma unroll 4
            for (int r = r0; r < dh; r += kRows) {
                uint32_t v[NW];
#pragma unroll
                for (int k = 0; k < NW; k++) v[k] = 0;
#pragma unroll
                for (int b = 0; b < NW * 4; b += U) {
                    const uint8_t *e = q + (b / PB) * step_p + b % PB;
                    const uint32_t x = U == 4 ? *reinterpret_cast<const uint32_t *>(e)
                                     : U == 2 ? *reinterpret_cast<const uint16_t *>(e) : *e;
                    v[b / 4] |= x << (8 * (b % 4));
                }
#pragma unroll
                for (int k = 0; k < NW; k++) to[k] = v[k];
                q += kRows * step_r;
                to += kRows * (Sh::kOutPitch / 4);
            }
        }
    }
    if (G > 1 && ((out0 | om) != 0 || dw % G != 0)) {
        // the pixels before a row's first group and after its last
        for (int i = threadIdx.x; i < dh * 2 * G; i += 256) {
            const int r = i / (2 * G), k = i % (2 * G);
            const int d = (out0 + r * om) & 3, p0 = min(head(d), dw), tail = (dw - p0) % G;
            if (k >= p0 + tail) continue;
            const int p = k < p0 ? k : dw - (p0 + tail) + k;
            const uint8_t *q = corner + r * step_r + p * step_p;
            uint8_t *to = outb + r * Sh::kOutPitch + d + p * PB;
#pragma unroll
            for (int b = 0; b < PB; b++) to[b] = q[b];
        }
    }
    __syncthreads();
    // pass 3: whole words, then the bytes of the rows' ends
    {
        const int mis = (out0 + warp * om) & 3, words = (mis + dw * PB) >> 2;
        uint32_t *row = reinterpret_cast<uint32_t *>(out + warp * opitch - mis) + lane;
        const uint32_t *from = out_words + warp * (Sh::kOutPitch / 4) + lane;
#pragma unroll 4
        for (int r = warp; r < dh; r += 8) {
#pragma unroll
            for (int q = 0; q < kLaneWords; q++)
                if (lane + 32 * q < words && (q > 0 || lane > 0 || mis == 0)) row[32 * q] = from[32 * q];
            row += 2 * opitch;
            from += 2 * Sh::kOutPitch;
        }
    }
    if (U < 4 && ((out0 | om) != 0 || (dw * PB) % 4 != 0)) {
        for (int i = threadIdx.x; i < dh * 8; i += 256) {
            const int r = i >> 3, mis = (out0 + r * om) & 3, n = mis + dw * PB, tail = max(n & ~3, mis ? 4 : 0);
            const int b = (i & 4) ? tail + (i & 3) : (i & 3);
            if (b < mis || b >= n || (!(i & 4) && mis == 0)) continue;
            out[(size_t)r * opitch + b - mis] = outb[r * Sh::kOutPitch + b];
        }
    }
}

// One-bit luma: one destination byte a thread (orient_bitpacked,
// orientation.rs:93-162).
__global__ void __launch_bounds__(256) jxrb_orient_bits(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst,
                                                       uint32_t w, uint32_t h, int o) {
    const bool swap = swaps_axes(o);
    const uint32_t ow = swap ? h : w, oh = swap ? w : h;
    const uint32_t in_stride = (w + 7) / 8, out_stride = (ow + 7) / 8;
    const size_t n = (size_t)out_stride * oh;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t y = (uint32_t)(i / out_stride), xb = (uint32_t)(i % out_stride);
        uint32_t byte = 0;
        for (uint32_t b = 0; b < 8; b++) {
            const uint32_t x = xb * 8 + b;
            if (x >= ow) break;
            uint32_t sx, sy;
            source_of(o, w, h, x, y, sx, sy);
            if (src[(size_t)sy * in_stride + sx / 8] & (0x80u >> (sx % 8))) byte |= 0x80u >> b;
        }
        dst[i] = (uint8_t)byte;
    }
}

template <typename W>
cudaError_t launch_tiles(const void *src, void *dst, uint32_t w, uint32_t h, uint32_t words, int o,
                         cudaStream_t stream) {
    const bool swap = o >= JXRB_ORIENT_TRANSPOSE;
    const uint32_t ow = swap ? h : w, oh = swap ? w : h;
    const dim3 grid((ow + kTile - 1) / kTile, (oh + kTile - 1) / kTile);
    const size_t smem = (size_t)kTile * kTile * words * sizeof(W);
    jxrb_orient_tiles<W><<<grid, 256, smem, stream>>>(static_cast<const W *>(src), static_cast<W *>(dst), w, h, words,
                                                      o);
    return cudaGetLastError();
}

template <int PB>
cudaError_t launch_pixels(const void *src, void *dst, uint32_t w, uint32_t h, int o, cudaStream_t stream) {
    constexpr int T = OrientShape<PB>::kSide;
    const bool swap = o >= JXRB_ORIENT_TRANSPOSE;
    const uint32_t ow = swap ? h : w, oh = swap ? w : h;
    const dim3 grid((ow + T - 1) / T, (oh + T - 1) / T);
    jxrb_orient_pixels<PB><<<grid, 256, 0, stream>>>(static_cast<const uint8_t *>(src), static_cast<uint8_t *>(dst), w,
                                                     h, o);
    return cudaGetLastError();
}

}  // namespace

extern "C" uint64_t jxrb_oriented_bytes(uint32_t width, uint32_t height, uint32_t pixel_bytes, int orientation) {
    const bool swap = orientation >= JXRB_ORIENT_TRANSPOSE;
    const uint64_t ow = swap ? height : width, oh = swap ? width : height;
    return pixel_bytes ? ow * oh * pixel_bytes : (ow + 7) / 8 * oh;
}

extern "C" jxrb_status jxrb_orient(const void *device_source, void *device_destination, uint32_t width,
                                   uint32_t height, uint32_t pixel_bytes, int orientation, void *cuda_stream) {
    if (orientation < JXRB_ORIENT_IDENTITY || orientation > JXRB_ORIENT_ROTATE270)
        return jxr::report_error(JXRB_INVALID_PLAN, "orientation code");
    if (!device_source || !device_destination) return jxr::report_error(JXRB_INVALID_DESTINATION, "null surface");
    if (device_source == device_destination)
        return jxr::report_error(JXRB_INVALID_DESTINATION, "orientation needs a destination apart from its source");
    if (pixel_bytes > kMaxPixelBytes)
        return jxr::report_error(JXRB_UNSUPPORTED_OUTPUT, "orientation of pixels above 48 bytes");
    if (width == 0 || height == 0) return JXRB_OK;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    cudaError_t e;
    if (pixel_bytes == 0) {
        const uint64_t n = jxrb_oriented_bytes(width, height, 0, orientation);
        const unsigned blocks = (unsigned)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
        jxrb_orient_bits<<<blocks, 256, 0, stream>>>(static_cast<const uint8_t *>(device_source),
                                                    static_cast<uint8_t *>(device_destination), width, height,
                                                    orientation);
        e = cudaGetLastError();
    } else {
        // the widest word that divides the pixel and both surfaces' alignment
        const uintptr_t a = reinterpret_cast<uintptr_t>(device_source) | reinterpret_cast<uintptr_t>(device_destination);
        const uint32_t n = pixel_bytes;
        if (jxr::takes_pixel_kernel(n, a, width, height))
            e = n == 1 ? launch_pixels<1>(device_source, device_destination, width, height, orientation, stream)
              : n == 2 ? launch_pixels<2>(device_source, device_destination, width, height, orientation, stream)
              : n == 3 ? launch_pixels<3>(device_source, device_destination, width, height, orientation, stream)
              : n == 4 ? launch_pixels<4>(device_source, device_destination, width, height, orientation, stream)
              : n == 6 ? launch_pixels<6>(device_source, device_destination, width, height, orientation, stream)
              : n == 8 ? launch_pixels<8>(device_source, device_destination, width, height, orientation, stream)
              : n == 12 ? launch_pixels<12>(device_source, device_destination, width, height, orientation, stream)
                        : launch_pixels<16>(device_source, device_destination, width, height, orientation, stream);
        else if (pixel_bytes % 4 == 0 && a % 4 == 0)
            e = launch_tiles<uint32_t>(device_source, device_destination, width, height, pixel_bytes / 4, orientation,
                                       stream);
        else if (pixel_bytes % 2 == 0 && a % 2 == 0)
            e = launch_tiles<uint16_t>(device_source, device_destination, width, height, pixel_bytes / 2, orientation,
                                       stream);
        else
            e = launch_tiles<uint8_t>(device_source, device_destination, width, height, pixel_bytes, orientation,
                                      stream);
    }
    if (e != cudaSuccess) return jxr::report_cuda(e, "orientation launch");
    return JXRB_OK;
}
