// The FP32 field's repetition loop over the streaming passes (stream_f32.cuh).
#include "passes.cuh"
#include "profiler.h"
#include "stream_f32.cuh"
#include "unrolled_impl.cuh"

namespace maxi {

int radius_bucket(int r) { return radius_bucket_impl(r); }

template cudaError_t launch_init_field<float>(const void *, int, uint32_t *, float *, int64_t, cudaStream_t);

namespace {

// Blocks a pass is cut into at least, where the axis allows it.  A block walks its segment
// of the axis alone, so few long walks leave SMs idle at the end of a launch; each further
// segment costs 2r rows read again and one un-overlapped first load.
constexpr int64_t kStreamMinBlocks = 148 * 4 * 5;

StreamShape stream_shape(int64_t outer, int64_t A, int64_t I, int tile, int chunk, int ring_multiple, int radius) {
    StreamShape s{};
    s.A = A;
    s.I = I;
    s.radius = radius;
    s.col_tiles = ceil_div(I, tile);
    int64_t segments = std::min(ceil_div(kStreamMinBlocks, outer * s.col_tiles), ceil_div(A, chunk));
    segments = std::max(segments, ceil_div(A, int64_t(1) << 30));  // positions in a segment are 32-bit
    s.seg_len = (int) round_up(ceil_div(A, segments), chunk);
    s.segments = ceil_div(A, s.seg_len);
    // The input of one chunk and, unless a segment is a single chunk, of the next one.
    s.ring = (int) round_up((s.seg_len > chunk ? 2 : 1) * chunk + 2 * radius, ring_multiple);
    return s;
}

bool aligned(const void *p, uintptr_t to) { return reinterpret_cast<uintptr_t>(p) % to == 0; }

// z (outer 1, axis z) or y (outer z, axis y) pass; `mask`: read the field from it instead.
// The passes are launched overlapped (launch.cuh) at every size; ten repetitions without / with it:
// 128^3 212 / 190 us, 301 x 517 x 333 3340 / 3375, 1024^3 75.4 ms both.
cudaError_t axis_pass(const float *in, const uint32_t *mask, float *out, int64_t outer, int64_t A, int64_t I,
                      int radius, const StreamTaps &taps, cudaStream_t st) {
    const StreamShape s = stream_shape(outer, A, I, kStreamCols, kStreamChunk, kStreamM, radius);
    const bool al = I % 4 == 0 && aligned(in, 16) && aligned(out, 16);
    auto kernel = mask ? (al ? stream_axis_pass<true, true> : stream_axis_pass<true, false>)
                       : (al ? stream_axis_pass<false, true> : stream_axis_pass<false, false>);
    return launch_pass(kernel, true, outer * s.col_tiles * s.segments, kStreamThreads, s.ring * kStreamRow, st, in, mask, out, s, taps);
}

// The tile form of the x pass (contig_pass): 16-byte copies and taps unrolled for radius R, zero
// beyond the kernel's own.
template <int R>
cudaError_t x_tile_pass(const float *in, float *out, const void *mask, int64_t rows, int64_t nx, int radius,
                        const float *kernel, cudaStream_t st) {
    const int64_t xt = ceil_div(nx, kConTX);
    return launch_pass(contig_pass<R, float, MAXI_MASK_BITPACKED, false>, true, xt * ceil_div(rows, kConTR), kConThreads,
                       contig_smem_bytes<R>(), st, in, out, mask, static_cast<uint16_t *>(nullptr),
                       static_cast<float *>(nullptr), rows, nx, xt, make_taps<R>(kernel, radius));
}

// The tile form needs rows that allow 16-byte accesses; a uint8 mask, which only the
// allocation-free call passes in, never comes with a volume large enough for it.  At large
// volumes it is the faster one for all but the last repetition where at most three taps a side
// are padding (its 16-byte copies and 40 warps per SM against 4-byte copies and 20).  1024^3, ms
// a pass, tile against stream_x_pass: r = 5 to 8 1.69 against 1.77 to 1.80, 9 to 12 1.94 to 2.00 against
// 2.06 to 2.12, 16 2.10 against 2.29 and more, 23 2.51 against 2.58, 29 2.84 against 2.89, 32 2.79
// against 3.05; r = 20 2.55 against 2.43, 28 2.84 against 2.83.  The last repetition's streaming form
// wins at every radius (r = 8 1.75 against 1.87, 32 3.05 against 3.24).  From 256^3 down the two are even
// (58 us at r = 32) and below that the streaming form's smaller blocks win (128^3: 7.7 against 8.8).
//
// That is for rows that fill the tiles.  A row ends in a tile of 256 voxels or a chunk of 128, and the form
// that computes fewer voxels beyond it gains that share: tile / stream at 2^26 voxels, r = 8, 16 and 31, at
// nx = 64 1.54 1.81 2.09, 300 1.07 1.16 1.27, 640 1.02 1.08 1.08, 896 0.97 1.04 1.01, 1100 0.95 1.00 0.98, 700
// 0.92 0.97 0.93, 1024 0.91 0.97 0.92.  Hence a limit on the tiles' voxels in per cent of the chunks', from whole
// calls of 2^24 to 2^27 voxels, and with padding taps beyond radius 8 a least row: r = 14 at nx = 132
// 1.02 times the streaming form's time, 0.98 at 200; r = 22 1.01 at 400, 0.99 at 500.
constexpr int64_t kTileMinVoxels = int64_t(1) << 24;
constexpr int kTilePadding = 3;
bool rows_fill_tiles(int64_t nx, int radius, bool padded) {
    if (padded && nx < (radius <= 8 ? 0 : radius <= 16 ? 192 : 448)) return false;
    const int limit = radius <= 8 || (radius <= 16 && !padded) ? 115 : padded ? 106 : 112;
    return 100 * round_up(nx, kConTX) <= limit * round_up(nx, kStreamChunkX);
}

template <int MASK_FMT, bool FINAL>
cudaError_t x_pass(const float *in, float *out, const void *mask, uint16_t *out_u16, float *field_out, int64_t rows,
                   int64_t nx, int radius, const StreamTaps &taps, cudaStream_t st) {
    if constexpr (MASK_FMT == MAXI_MASK_BITPACKED && !FINAL)
        if (radius > 0 && nx % 4 == 0 && rows * nx >= kTileMinVoxels && aligned(in, 16) && aligned(out, 16)) {
#define MAXI_CASE(R) \
    if (radius <= R && radius + kTilePadding >= R && rows_fill_tiles(nx, radius, radius < R)) \
        return x_tile_pass<R>(in, out, mask, rows, nx, radius, taps.k, st);
            MAXI_CASE(4) MAXI_CASE(8) MAXI_CASE(12) MAXI_CASE(16) MAXI_CASE(24) MAXI_CASE(32)
#undef MAXI_CASE
        }
    const StreamShape s = stream_shape(1, nx, rows, kStreamRowsX, kStreamChunkX, 32, radius);
    const int smem = kStreamRowsX * stream_x_pitch(s.ring) * 4 + kStreamMaskBytes;
    return launch_pass(stream_x_pass<MASK_FMT, FINAL>, true, s.col_tiles * s.segments, kStreamThreads, smem, st, in, out,
                       mask, out_u16, field_out, s, taps);
}

}  // namespace

template <>
cudaError_t dispatch_unrolled<float>(const Volume &v, const void *mask, int mask_fmt, const float *kernel, int radius,
                                     int64_t reps, float *buf0, float *buf1, uint16_t *out_u16, float *field_out,
                                     int32_t flags, cudaStream_t st, const RunOpts &o) {
    if (radius > kMaxUnrolledRadius) return cudaErrorInvalidValue;
    StreamTaps taps{};
    std::copy(kernel, kernel + 2 * radius + 1, taps.k);
    uint32_t *rebuild = (flags & MAXI_FLAG_MASK_FROM_FIELD) && mask_fmt == MAXI_MASK_BITPACKED
                            ? const_cast<uint32_t *>(static_cast<const uint32_t *>(mask))
                            : nullptr;
    cudaError_t e;
    // The first z pass reads a bit-packed mask itself; a field to continue from or a uint8
    // mask becomes the field first.
    const bool from_mask = !o.field_ready && !o.init_field && mask_fmt == MAXI_MASK_BITPACKED;
    if (!from_mask && !o.field_ready) {
        ProfScope ps(MAXI_KERNEL_INIT, st);
        if (o.init_field)
            field_from_f32<float><<<std::min<int64_t>(ceil_div(v.n(), 256), 148 * 64), 256, 0, st>>>(o.init_field, buf0, v.n());
        else if ((e = launch_init_field<float>(mask, mask_fmt, nullptr, buf0, v.n(), st)) != cudaSuccess)
            return e;
    }
    if (reps > 0) note_path(MAXI_PATH_CUDA_CORES);
    const int64_t plane = v.ny * v.nx;
    for (int64_t rep = 0; rep < reps; rep++) {
        // Plane window of this repetition (the whole volume unless shrinking).
        const int64_t lo = std::min(v.nz - 1, o.shrink_lo * rep);
        const int64_t hi = std::max(lo + 1, v.nz - o.shrink_hi * rep);
        const int64_t nzv = hi - lo, off = lo * plane, rows = nzv * v.ny;
        float *b0 = buf0 + off, *b1 = buf1 + off;
        const bool last = rep + 1 == reps;
        if (o.final_wait && last && (e = cudaStreamWaitEvent(st, o.final_wait, 0)) != cudaSuccess) return e;
        // The rebuilt-mask semantics: before every repetition after the first of
        // the whole run (a continued run's first repetition is not the first).
        if (rebuild && (rep > 0 || o.init_field)) {
            ProfScope ps(MAXI_KERNEL_OTHER, st);
            const int64_t blocks = std::min<int64_t>(ceil_div(ceil_div(nzv * plane, 32), 256), 148 * 16);
            mask_from_field<float><<<blocks, 256, 0, st>>>(b0, rebuild + off / 32, nzv * plane);
        }
        const void *mv = mask_fmt == MAXI_MASK_U8 ? static_cast<const void *>(static_cast<const uint8_t *>(mask) + off)
                                                  : static_cast<const void *>(static_cast<const uint32_t *>(mask) + off / 32);
        {
            ProfScope ps(MAXI_KERNEL_Z, st);
            e = axis_pass(b0, from_mask && rep == 0 ? static_cast<const uint32_t *>(mv) : nullptr, b1, 1, nzv, plane,
                          radius, taps, st);
        }
        if (e != cudaSuccess) return e;
        {
            ProfScope ps(MAXI_KERNEL_Y, st);
            e = axis_pass(b1, nullptr, b0, nzv, v.ny, v.nx, radius, taps, st);
        }
        if (e != cudaSuccess) return e;
        {
            ProfScope ps(last ? MAXI_KERNEL_X_FINAL : MAXI_KERNEL_X, st);
            uint16_t *ou = last && out_u16 ? out_u16 + off : nullptr;
            float *fo = last && field_out ? field_out + off : nullptr;
            const bool u8 = mask_fmt == MAXI_MASK_U8;
            auto pass = last ? (u8 ? x_pass<MAXI_MASK_U8, true> : x_pass<MAXI_MASK_BITPACKED, true>)
                             : (u8 ? x_pass<MAXI_MASK_U8, false> : x_pass<MAXI_MASK_BITPACKED, false>);
            e = pass(b0, b1, mv, ou, fo, rows, v.nx, radius, taps, st);
        }
        if (e != cudaSuccess) return e;
        std::swap(buf0, buf1);
    }
    return cudaGetLastError();
}

}  // namespace maxi
