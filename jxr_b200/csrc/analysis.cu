// analysis.cu -- the forward half of the codec on the GPU: the mirror of the
// reconstruction path, from sample planes to quantized coefficients.
//
// The reference analyses on the CPU only (analyze_component,
// crates/jxr-native/src/analyze.rs:56-131): the second-level prefilter (the
// forward overlap operators over the sample plane, overlap modes 1 and 2),
// the forward core transform of every 4x4 block, the first-level prefilter
// over the plane of block DCs (overlap mode 2; the ordered subsampled
// schedule for 4:2:0 / 4:2:2 chroma), the forward transform of each
// macroblock's block DCs (halved first where the plane is scaled), and the
// quantization of the DC, low-pass and high-pass bands (Quantizer::quantize,
// crates/jxr-math/src/quantization.rs:28-50).  Here a plane takes two passes:
// the second-level prefilter in place, then everything from the block
// transforms to the quantized bands; overlap mode 2 takes the first-level
// prefilter and the low-pass bands in kernels of their own after that.  The
// overlap operators of one level are disjoint (the subsampled corners aside,
// which run in three ordered phases as in the decoder), so every operator,
// block and macroblock is its own work item.  The results equal the CPU
// analysis bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/jxr_b200.h"
#include "forward.h"

namespace jxr {
jxrb_status report_error(jxrb_status s, const char *why);
jxrb_status report_cuda(cudaError_t e, const char *what);
}  // namespace jxr

namespace {

using namespace jxr::fwd;

// Division by a step that does not change, as a multiplication and shifts
// exact for every 32-bit dividend (Granlund and Montgomery, "Division by
// invariant integers using multiplication", 1994, figure 4.1).
struct Divider {
    uint32_t mul, offset;      // multiplier; the rounding offset added before the division
    uint32_t shift1, shift2;
};

// One plane on the device.  `starts` maps mark the macroblock columns / rows
// where a hard tile begins (planes with soft tiles have none).  Maps and
// region lists are at byte offsets of the set's blob.
struct APlane {
    int32_t *samples;          // W x H, prefiltered in place
    int32_t *low;              // block DCs, (W/4) x (H/4): overlap mode 2
    int32_t *low_q;            // 16 a macroblock
    int32_t *high_q;           // 256 a macroblock
    uint32_t col_at, row_at;   // tile-start maps
    uint32_t cols_at;          // column region boundaries in macroblocks (0 .. mbs_x)
    uint32_t ncols;
    uint32_t W, H, mbs_x, mbs_y;
    int32_t bc, br, scale2, overlap, hard;
    int32_t wide;              // outputs 16-byte aligned, block DCs 8-byte aligned
    Divider q[3];              // DC, low-pass, high-pass
};

// The planes of a call.  A few planes (a picture's) travel in the kernels'
// parameters; more of them, or longer tile lists, in device memory.
constexpr uint32_t kInlinePlanes = 8, kInlineBlob = 2560;
struct ASet {
    const APlane *planes_mem;  // null: the planes and the blob below
    const uint8_t *blob_mem;
    APlane planes[kInlinePlanes];
    uint32_t blob[kInlineBlob / 4];
};
static_assert(sizeof(ASet) <= 4096, "kernel parameters");

__device__ __forceinline__ const APlane &plane_of(const ASet &s) {
    return s.planes_mem ? s.planes_mem[blockIdx.y] : s.planes[blockIdx.y];
}
__device__ __forceinline__ const uint8_t *blob_of(const ASet &s) {
    return s.planes_mem ? s.blob_mem : reinterpret_cast<const uint8_t *>(s.blob);
}

// quantize() of forward.h: (|c| + offset) / step.  The offset is at most half
// the step, so the sum stays below 2^32.
__device__ __forceinline__ int32_t quantized(int32_t c, const Divider &d) {
    const uint32_t n = (c < 0 ? 0u - (uint32_t)c : (uint32_t)c) + d.offset;
    const uint32_t t = __umulhi(d.mul, n);
    const uint32_t q = (t + ((n - t) >> d.shift1)) >> d.shift2;
    return c < 0 ? (int32_t)(0u - q) : (int32_t)q;
}

__device__ __forceinline__ void store4(int32_t *p, bool wide, int32_t a, int32_t b, int32_t c, int32_t d) {
    if (wide) {
        *reinterpret_cast<int4 *>(p) = make_int4(a, b, c, d);
    } else {
        p[0] = a; p[1] = b; p[2] = c; p[3] = d;
    }
}

__device__ __forceinline__ bool boundary(int p, int extent, int lg, int hard, const uint8_t *starts) {
    if (p <= 0 || p >= extent) return true;
    return hard && (p & ((1 << lg) - 1)) == 0 && starts[p >> lg];
}

__device__ __forceinline__ int log2i(int v) { return 31 - __clz(v); }

// The full-resolution overlap schedule of a plane of W x H values whose
// macroblocks are 2^lx x 2^ly of them, run forward: one 4x4 cell a thread,
// cells at origins 2 (mod 4); a cell a region boundary crosses takes the
// edge strips or corner quarters (the decoder's window list, forward
// operators; crates/jxr-native/src/reconstruct/overlap.rs:124-323).  A window
// starts two values past a 16-byte boundary: with `pairs` (values 8-byte
// aligned, W even) its rows move as two 8-byte pieces each.
__device__ void prefilter_cells(int32_t *s, int W, int H, int lx, int ly, int hard, const uint8_t *col_start,
                                const uint8_t *row_start, bool pairs) {
    const int ncx = W / 4 + 1, ncy = H / 4 + 1;
    auto at = [&](int x, int y) -> int32_t & { return s[(size_t)y * W + x]; };
    auto inside = [&](int x, int y) { return x >= 0 && x < W && y >= 0 && y < H; };
    for (int item = blockIdx.x * blockDim.x + threadIdx.x; item < ncx * ncy; item += gridDim.x * blockDim.x) {
        const int cx = -2 + 4 * (item % ncx), cy = -2 + 4 * (item / ncx);
        const bool vs = boundary(cx + 2, W, lx, hard, col_start), hs = boundary(cy + 2, H, ly, hard, row_start);
        if (!vs && !hs) {
            int32_t v[16];
            if (pairs) {
#pragma unroll
                for (int r = 0; r < 4; r++)
#pragma unroll
                    for (int c = 0; c < 4; c += 2) {
                        const int2 q = *reinterpret_cast<const int2 *>(&at(cx + c, cy + r));
                        v[r * 4 + c] = q.x;
                        v[r * 4 + c + 1] = q.y;
                    }
                forward_pot4x4(v);
#pragma unroll
                for (int r = 0; r < 4; r++)
#pragma unroll
                    for (int c = 0; c < 4; c += 2)
                        *reinterpret_cast<int2 *>(&at(cx + c, cy + r)) = make_int2(v[r * 4 + c], v[r * 4 + c + 1]);
                continue;
            }
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) v[r * 4 + c] = at(cx + c, cy + r);
            forward_pot4x4(v);
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) at(cx + c, cy + r) = v[r * 4 + c];
        } else if (vs && !hs) {
            for (int c = 0; c < 4; c++)
                if (cx + c >= 0 && cx + c < W) forward_pot4(at(cx + c, cy), at(cx + c, cy + 1), at(cx + c, cy + 2), at(cx + c, cy + 3));
        } else if (!vs && hs) {
            for (int r = 0; r < 4; r++)
                if (cy + r >= 0 && cy + r < H) forward_pot4(at(cx, cy + r), at(cx + 1, cy + r), at(cx + 2, cy + r), at(cx + 3, cy + r));
        } else {
            for (int k = 0; k < 4; k++) {
                const int x = cx + (k & 1) * 2, y = cy + (k >> 1) * 2;
                if (inside(x, y)) forward_pot4(at(x, y), at(x + 1, y), at(x, y + 1), at(x + 1, y + 1));
            }
        }
    }
}

__global__ void __launch_bounds__(256) jxrb_analysis_prefilter(const __grid_constant__ ASet set) {
    const APlane &p = plane_of(set);
    if (p.overlap < 1) return;
    const uint8_t *blob = blob_of(set);
    prefilter_cells(p.samples, (int)p.W, (int)p.H, log2i(p.bc * 4), log2i(p.br * 4), p.hard, blob + p.col_at,
                    blob + p.row_at, true);
}

// A macroblock's block DCs (raster in l; halved where the plane is scaled)
// through the forward first-level transform, quantized, to its 16 low-pass
// places (analyze.rs:88-131).
__device__ __forceinline__ void analyze_low(const APlane &p, int32_t (&l)[16], uint32_t m) {
    const int count = p.bc * p.br;
#pragma unroll
    for (int k = 0; k < 16; k++) l[k] = k < count ? (p.scale2 ? l[k] >> 1 : l[k]) : 0;
    if (count == 16) {
        forward_pct(l);
    } else if (count == 4) {
        int32_t w[4] = {l[0], l[1], l[2], l[3]};
        forward_420(w);
#pragma unroll
        for (int k = 0; k < 4; k++) l[k] = w[k];
    } else {
        int32_t w[8] = {l[0], l[1], l[2], l[3], l[4], l[5], l[6], l[7]};
        forward_422(w);
#pragma unroll
        for (int k = 0; k < 8; k++) l[k] = w[k];
    }
    l[0] = quantized(l[0], p.q[0]);
#pragma unroll
    for (int k = 1; k < 16; k++) l[k] = k < count ? quantized(l[k], p.q[1]) : 0;
#pragma unroll
    for (int k = 0; k < 16; k += 4) store4(p.low_q + (size_t)m * 16 + k, p.wide, l[k], l[k + 1], l[k + 2], l[k + 3]);
}

// Forward core transform of every block, its fifteen coefficients quantized
// (rounding offsets of half the step for DC and low-pass, a third for
// high-pass), and, without a first-level prefilter, its macroblock's low-pass
// band; overlap mode 2 writes the block DCs for the kernels below instead.
//
// One block a thread, the 256 blocks of 16 (full resolution), 32 or 64
// macroblocks a CTA: threads take blocks along a block row, so that a warp
// reads 512-byte row pieces, and the coefficients leave through shared memory
// as the run of whole macroblocks they are in the output.  Memory traffic is
// what bounds it: the separate transform and one-macroblock-a-thread
// quantization kernels wrote 4-byte words 64 bytes and 1 KB apart (three
// planes of a 2048 x 1536 4:2:0 picture, cold caches: 32 + 89 us, 18.7 us
// here).
constexpr int kBlocks = 256;
__global__ void __launch_bounds__(kBlocks) jxrb_analysis_blocks(const __grid_constant__ ASet set) {
    __shared__ __align__(16) int32_t coded[kBlocks * 16];
    __shared__ int32_t dcs[kBlocks + 64];
    const APlane &p = plane_of(set);
    const int bc = p.bc, count = bc * p.br, lcount = log2i(count), n = kBlocks >> lcount;
    const uint32_t mbs = p.mbs_x * p.mbs_y;
    const int t = threadIdx.x;
    const int across = n * bc, r = t / across, c = t % across;   // powers of two
    const int i = c / bc, col = c % bc, s = i * count + r * bc + col;
    // piece q of slot s sits at q ^ swizzle(s): the threads of a quarter-warp
    // then write to distinct bank groups at every block shape
    auto swizzle = [](int slot) { return ((slot >> 1) ^ (slot >> 3)) & 3; };
    for (uint32_t first = blockIdx.x * n; first < mbs; first += gridDim.x * n) {
        const uint32_t m = first + i;
        if (m < mbs) {
            const uint32_t my = m / p.mbs_x, mx = m - my * p.mbs_x;
            const uint32_t by = my * p.br + r, bx = mx * bc + col;
            const int32_t *from = p.samples + (size_t)by * 4 * p.W + bx * 4;
            int32_t v[16];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int4 q = *reinterpret_cast<const int4 *>(from + (size_t)k * p.W);
                v[k * 4] = q.x; v[k * 4 + 1] = q.y; v[k * 4 + 2] = q.z; v[k * 4 + 3] = q.w;
            }
            forward_pct(v);
            if (p.overlap == 2) p.low[(size_t)by * (p.W / 4) + bx] = v[0];
            else dcs[i * (count + 1) + r * bc + col] = v[0];
            v[0] = 0;
            const Divider d = p.q[2];
#pragma unroll
            for (int k = 1; k < 16; k++) v[k] = quantized(v[k], d);
#pragma unroll
            for (int k = 0; k < 4; k++)
                *reinterpret_cast<int4 *>(&coded[s * 16 + ((k ^ swizzle(s)) << 2)]) =
                    make_int4(v[k * 4], v[k * 4 + 1], v[k * 4 + 2], v[k * 4 + 3]);
        }
        __syncthreads();
        // past the macroblock's block count its places are zero
        const uint32_t held = min((uint32_t)n, mbs - first);
        int32_t *to = p.high_q + (size_t)first * 256;
        for (uint32_t k = t; k < held * 64; k += kBlocks) {
            const int b = (k & 63) >> 2, slot = (int)(k >> 6) * count + b;
            const int4 q = b < count ? *reinterpret_cast<const int4 *>(&coded[slot * 16 + (((k & 3) ^ swizzle(slot)) << 2)])
                                     : make_int4(0, 0, 0, 0);
            store4(to + k * 4, p.wide, q.x, q.y, q.z, q.w);
        }
        if (p.overlap != 2 && t < (int)held) {
            int32_t l[16];
#pragma unroll
            for (int k = 0; k < 16; k++) l[k] = k < count ? dcs[t * (count + 1) + k] : 0;
            analyze_low(p, l, first + t);
        }
        __syncthreads();
    }
}

// First-level prefilter of full-resolution planes: the cells of the block-DC plane.
__global__ void __launch_bounds__(256) jxrb_analysis_low_full(const __grid_constant__ ASet set) {
    const APlane &p = plane_of(set);
    if (p.overlap != 2 || p.bc != 4) return;
    const uint8_t *blob = blob_of(set);
    prefilter_cells(p.low, (int)(p.W / 4), (int)(p.H / 4), 2, 2, p.hard, blob + p.col_at, blob + p.row_at, p.wide);
}

// First-level prefilter of subsampled chroma, the decoder's ordered schedule
// inverted (crates/jxr-native/src/reconstruct/subsampled_overlap.rs:244-296):
// phase 0, each boundary row's corners lose their neighbour (right corner
// first); phase 1, every two-sample pair and 2x2 square forward; phase 2, the
// corners regain their (now filtered) neighbour.  A region two samples wide
// runs its four corner steps in that order as well.
__global__ void __launch_bounds__(256) jxrb_analysis_low_subsampled(const __grid_constant__ ASet set, int phase) {
    const APlane &p = plane_of(set);
    if (p.overlap != 2 || p.bc != 2) return;
    const uint8_t *blob = blob_of(set);
    const int W = (int)(p.W / 4), H = (int)(p.H / 4);
    const int lx = log2i(p.bc), ly = log2i(p.br);
    int32_t *s = p.low;
    auto at = [&](int x, int y) -> int32_t & { return s[(size_t)y * W + x]; };
    auto vb = [&](int x) { return boundary(x, W, lx, p.hard, blob + p.col_at); };
    auto hb = [&](int y) { return boundary(y, H, ly, p.hard, blob + p.row_at); };
    if (phase == 1) {
        auto inside = [&](int x, int y) { return x >= 0 && x < W && y >= 0 && y < H; };
        const int ncx = W / 2 + 1, ncy = H / 2 + 1;
        for (int item = blockIdx.x * blockDim.x + threadIdx.x; item < ncx * ncy; item += gridDim.x * blockDim.x) {
            const int cx = -1 + 2 * (item % ncx), cy = -1 + 2 * (item / ncx);
            const bool vs = vb(cx + 1), hs = hb(cy + 1);
            if (!vs && !hs) {
                if (inside(cx, cy) && inside(cx + 1, cy + 1))
                    forward_pot2x2(at(cx, cy), at(cx + 1, cy), at(cx, cy + 1), at(cx + 1, cy + 1));
            } else if (vs && !hs) {
                for (int c = 0; c < 2; c++)
                    if (inside(cx + c, cy) && inside(cx + c, cy + 1)) forward_pot2(at(cx + c, cy), at(cx + c, cy + 1));
            } else if (!vs && hs) {
                for (int r = 0; r < 2; r++)
                    if (inside(cx, cy + r) && inside(cx + 1, cy + r)) forward_pot2(at(cx, cy + r), at(cx + 1, cy + r));
            }
        }
        return;
    }
    // phases 0 and 2: one (boundary row, column region) a thread
    const int nreg = (int)p.ncols - 1;
    const uint32_t *cols = reinterpret_cast<const uint32_t *>(blob + p.cols_at);
    for (int item = blockIdx.x * blockDim.x + threadIdx.x; item < H * nreg; item += gridDim.x * blockDim.x) {
        const int y = item / nreg, k = item % nreg;
        const bool top = hb(y), bottom = hb(y + 1);
        if (!top && !bottom) continue;
        const int l = (int)cols[k] * p.bc, r = (int)cols[k + 1] * p.bc;
        int32_t &c0 = at(l, y), &n0 = at(l + 1, y), &c1 = at(r - 1, y), &n1 = at(r - 2, y);
        if (phase == 0) {
            c1 -= n1;
            c0 -= n0;
        } else {
            c1 += n1;
            c0 += n0;
        }
    }
}

// The low-pass bands of two-level planes from their filtered block DCs, one
// macroblock a thread.
__global__ void __launch_bounds__(256) jxrb_analysis_low_bands(const __grid_constant__ ASet set) {
    const APlane &p = plane_of(set);
    if (p.overlap != 2) return;
    const uint32_t n = p.mbs_x * p.mbs_y, lw = p.W / 4;
    const int lbc = log2i(p.bc), count = p.bc * p.br;
    for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += gridDim.x * blockDim.x) {
        const uint32_t mx = m % p.mbs_x, my = m / p.mbs_x;
        const int32_t *from = p.low + (size_t)my * p.br * lw + mx * p.bc;
        int32_t l[16];
#pragma unroll
        for (int k = 0; k < 16; k++) l[k] = k < count ? from[(size_t)(k >> lbc) * lw + (k & (p.bc - 1))] : 0;
        analyze_low(p, l, m);
    }
}

Divider divider(uint32_t step, uint32_t offset) {
    if (offset >= step) offset = step - 1;
    int l = 0;
    while (l < 32 && (1ull << l) < step) l++;
    return Divider{(uint32_t)((((1ull << l) - step) << 32) / step + 1), offset, (uint32_t)std::min(l, 1),
                   (uint32_t)std::max(l - 1, 0)};
}

unsigned grid_for(uint64_t work) {
    return (unsigned)std::min<uint64_t>(std::max<uint64_t>((work + 255) / 256, 1), 2048);
}

}  // namespace

extern "C" jxrb_status jxrb_analyze_planes(const jxrb_analysis_plane *planes, uint32_t count, void *cuda_stream) {
    if (!planes || count == 0) return jxr::report_error(JXRB_INVALID_PLAN, "no planes");
    if (count > 65535) return jxr::report_error(JXRB_RESOURCE_LIMIT, "too many planes in one call");
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    // descriptors, and the blob of tile-start maps and region lists
    std::vector<APlane> dev(count);
    std::vector<uint8_t> blob;
    uint64_t max_samples = 0, max_mbs = 0, max_rows = 0, max_groups = 0;
    bool filtered = false, two_level = false, subsampled = false;
    for (uint32_t i = 0; i < count; i++) {
        const jxrb_analysis_plane &a = planes[i];
        const bool full = a.block_columns == 4 && a.block_rows == 4;
        const bool c420 = a.block_columns == 2 && a.block_rows == 2, c422 = a.block_columns == 2 && a.block_rows == 4;
        if (!full && !c420 && !c422) return jxr::report_error(JXRB_INVALID_PLAN, "block shape (4x4, 2x4 or 2x2)");
        const uint32_t mw = a.block_columns * 4, mh = a.block_rows * 4;
        if (a.width == 0 || a.height == 0 || a.width % mw || a.height % mh)
            return jxr::report_error(JXRB_INVALID_PLAN, "plane extent is not a whole number of macroblocks");
        if (a.overlap < 0 || a.overlap > 2) return jxr::report_error(JXRB_INVALID_PLAN, "overlap mode");
        if (a.steps[0] == 0 || a.steps[1] == 0 || a.steps[2] == 0) return jxr::report_error(JXRB_INVALID_PLAN, "zero quantizer");
        if (!a.samples || !a.low_scratch || !a.low_q || !a.high_q)
            return jxr::report_error(JXRB_INVALID_DESTINATION, "null device buffer");
        const uint32_t mbs_x = a.width / mw, mbs_y = a.height / mh;
        // tile starts and column regions from the boundaries (0 .. extent)
        const uint32_t *cb = a.column_boundaries, *rb = a.row_boundaries;
        if (!cb || !rb || a.column_count < 2 || a.row_count < 2 || cb[0] != 0 || rb[0] != 0 ||
            cb[a.column_count - 1] != mbs_x || rb[a.row_count - 1] != mbs_y)
            return jxr::report_error(JXRB_INVALID_PLAN, "tile boundaries must run from 0 to the macroblock extent");
        for (uint32_t k = 1; k < a.column_count; k++)
            if (cb[k] <= cb[k - 1]) return jxr::report_error(JXRB_INVALID_PLAN, "tile column boundaries");
        for (uint32_t k = 1; k < a.row_count; k++)
            if (rb[k] <= rb[k - 1]) return jxr::report_error(JXRB_INVALID_PLAN, "tile row boundaries");
        APlane &d = dev[i];
        d.samples = a.samples;
        d.low = a.low_scratch;
        d.low_q = a.low_q;
        d.high_q = a.high_q;
        d.W = a.width;
        d.H = a.height;
        d.mbs_x = mbs_x;
        d.mbs_y = mbs_y;
        d.bc = (int)a.block_columns;
        d.br = (int)a.block_rows;
        d.scale2 = a.scaled ? 1 : 0;
        d.overlap = a.overlap;
        d.hard = a.hard_tiles ? 1 : 0;
        d.ncols = a.hard_tiles ? a.column_count : 2;
        for (int b = 0; b < 3; b++) d.q[b] = divider(a.steps[b], a.steps[b] / (b < 2 ? 2 : 3));
        d.wide = ((reinterpret_cast<uintptr_t>(a.low_q) | reinterpret_cast<uintptr_t>(a.high_q)) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(a.low_scratch) & 7) == 0;
        if (a.hard_tiles) {
            d.col_at = (uint32_t)blob.size();
            d.row_at = d.col_at + mbs_x + 1;
            blob.resize(blob.size() + mbs_x + mbs_y + 2, 0);
            for (uint32_t k = 1; k + 1 < a.column_count; k++) blob[d.col_at + cb[k]] = 1;
            for (uint32_t k = 1; k + 1 < a.row_count; k++) blob[d.row_at + rb[k]] = 1;
        }
        if (a.overlap == 2 && !full) {
            const uint32_t whole[2] = {0, mbs_x};
            const uint32_t *list = a.hard_tiles ? cb : whole;
            blob.resize((blob.size() + 3) / 4 * 4, 0);
            d.cols_at = (uint32_t)blob.size();
            blob.insert(blob.end(), reinterpret_cast<const uint8_t *>(list),
                        reinterpret_cast<const uint8_t *>(list + d.ncols));
        }
        max_samples = std::max<uint64_t>(max_samples, (uint64_t)a.width * a.height);
        max_mbs = std::max<uint64_t>(max_mbs, (uint64_t)mbs_x * mbs_y);
        max_groups = std::max<uint64_t>(max_groups, ((uint64_t)a.width * a.height / 16 + kBlocks - 1) / kBlocks);
        max_rows = std::max<uint64_t>(max_rows, (uint64_t)(a.height / 4) * (d.ncols - 1));
        filtered |= a.overlap >= 1;
        two_level |= a.overlap == 2;
        subsampled |= a.overlap == 2 && !full;
    }
    // A call of a few planes needs no device memory for them: allocating,
    // copying and freeing it cost about as long as a small picture's kernels.
    ASet set;
    std::memset(&set, 0, sizeof set);
    void *mem = nullptr;
    std::vector<uint8_t> host;
    cudaError_t e = cudaSuccess;
    if (count <= kInlinePlanes && blob.size() <= kInlineBlob) {
        std::copy(dev.begin(), dev.end(), set.planes);
        if (!blob.empty()) std::memcpy(set.blob, blob.data(), blob.size());
    } else {
        const size_t blob_at = (sizeof(APlane) * count + 255) / 256 * 256;
        e = cudaMallocAsync(&mem, blob_at + blob.size(), stream);
        if (e != cudaSuccess) return jxr::report_cuda(e, "cudaMallocAsync (analysis descriptors)");
        host.assign(blob_at + blob.size(), 0);
        std::memcpy(host.data(), dev.data(), sizeof(APlane) * count);
        if (!blob.empty()) std::memcpy(host.data() + blob_at, blob.data(), blob.size());
        set.planes_mem = static_cast<const APlane *>(mem);
        set.blob_mem = static_cast<const uint8_t *>(mem) + blob_at;
        e = cudaMemcpyAsync(mem, host.data(), host.size(), cudaMemcpyHostToDevice, stream);
    }
    const dim3 g_cells(grid_for(max_samples / 16 + 64), count);
    const dim3 g_blocks((unsigned)std::min<uint64_t>(max_groups, 4096), count);
    const dim3 g_mbs(grid_for(max_mbs), count), g_rows(grid_for(max_rows), count);
    if (e == cudaSuccess) {
        if (filtered) jxrb_analysis_prefilter<<<g_cells, 256, 0, stream>>>(set);
        jxrb_analysis_blocks<<<g_blocks, kBlocks, 0, stream>>>(set);
        if (two_level) {
            jxrb_analysis_low_full<<<g_cells, 256, 0, stream>>>(set);
            if (subsampled) {
                jxrb_analysis_low_subsampled<<<g_rows, 256, 0, stream>>>(set, 0);
                jxrb_analysis_low_subsampled<<<g_cells, 256, 0, stream>>>(set, 1);
                jxrb_analysis_low_subsampled<<<g_rows, 256, 0, stream>>>(set, 2);
            }
            jxrb_analysis_low_bands<<<g_mbs, 256, 0, stream>>>(set);
        }
        e = cudaGetLastError();
    }
    // the outputs are written, and the host image of the descriptors read,
    // once the stream has come this far
    const cudaError_t s = cudaStreamSynchronize(stream);
    if (mem) cudaFreeAsync(mem, stream);
    if (e != cudaSuccess) return jxr::report_cuda(e, "analysis launch");
    if (s != cudaSuccess) return jxr::report_cuda(s, "analysis");
    return JXRB_OK;
}
