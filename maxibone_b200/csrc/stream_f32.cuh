// FP32 convolution passes of the diffusion step, any radius up to kMaxUnrolledRadius.
//
// What bounds them: one pass reads and writes 8 bytes and does 2r + 1 FMAs per voxel, so
// up to about r = 20 HBM sets the time and above it the FP32 pipe does (65 taps per
// 1024^3 voxels: 1.33 ms of HBM against 1.9 ms of FMAs).  Both have to run at once, so a
// CTA streams along the convolution axis instead of staging one tile and then
// computing it: the input passes through a ring in shared memory, and while one chunk of
// outputs is computed the input of the next one arrives by cp.async.  Every input is read
// once per segment of the axis, not once per tile plus halo.
//
// Every output is summed over the taps in increasing order with one FMA each -- the
// reference's summation order (src/lib/cpp/cpu/diffusion.cc:41-54) -- with the inputs of
// the current tap in a register window that rotates as the taps advance, so any radius
// runs without padding taps.
//
//   * stream_axis_pass: the z and y passes; the volume as [outer][axis][inner].  A CTA has
//     64 columns, a thread two of them (packed FMAs) and 16 consecutive outputs.
//   * stream_x_pass: the x pass with re-illumination and, in the last repetition,
//     quantisation.  A CTA has 32 rows, a lane one of them and a thread 32 consecutive
//     outputs as packed pairs (x, x + 16), which leave through the ring a row at a time.
//
// Per pass on a B200 at 1965 MHz, against the tiled passes with unrolled taps before them
// (which took 4-byte loads wherever rows are not 16-byte aligned):
//   1024^3, r = 32: z and y 2.34 ms (59.5 TFLOP/s), before 2.59 and 2.56
//   1024^3, r = 12: z and y 1.33 ms (6.4 TB/s), before 1.55 and 1.44
//   1024^3, r = 40: before 9.7 (the unrolled taps overflowed the instruction cache)
//   301 x 517 x 333, r = 10: z 108, y 113, x 103 us, before 220, 208 and 384
//   128^3, r = 12: z and y 5.2, x 7.7 us, before 8.6 and 8.8
// The packed FMAs alone reach 66 TFLOP/s from a window like this one (73 with every operand
// but the accumulator constant); the rest goes to the copies, stores and barriers.
#pragma once

#include "common.cuh"

namespace maxi {

constexpr int kStreamWarps = 4;
constexpr int kStreamThreads = 32 * kStreamWarps;
// z and y passes
constexpr int kStreamM = 16;                           // outputs per thread along the axis
constexpr int kStreamChunk = kStreamM * kStreamWarps;  // outputs per CTA and step
constexpr int kStreamCols = 64;
constexpr int kStreamRow = kStreamCols * 4;            // bytes of a ring row
// x pass
constexpr int kStreamMX = 2 * kStreamM;  // a thread's outputs: 16 pairs (x, x + 16)
constexpr int kStreamChunkX = kStreamMX * kStreamWarps;
constexpr int kStreamRowsX = 32;
// Words of a ring row: odd, so the 32 lanes' reads of one x (a row each) fall into 32 banks.
// That rules out copies of more than 4 bytes, and rows and radii then need no alignment.
__host__ __device__ constexpr int stream_x_pitch(int ring) { return ring + 1; }
// Mask words kept per row and chunk: those that it may touch.
constexpr int kStreamMaskWords = kStreamChunkX / 32 + 1;
constexpr int kStreamMaskBytes = 2 * kStreamRowsX * kStreamMaskWords * 4;

struct StreamTaps {
    float k[2 * kMaxUnrolledRadius + 1];
};

// One pass's view of the volume, cut into segments of the axis (a CTA walks one).
struct StreamShape {
    int64_t A, I;         // axis length; columns (z, y) or rows (x)
    int64_t col_tiles;    // tiles of the columns
    int64_t segments;
    int seg_len;          // a multiple of the chunk, except that it may exceed A
    int radius, ring;     // ring: axis positions in shared memory
};

__device__ __forceinline__ uint32_t shared_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
template <int BYTES>
__device__ __forceinline__ void async_copy(uint32_t dst, const float *src, bool ok = true) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(dst), "l"(src), "n"(BYTES), "r"(ok ? BYTES : 0) : "memory");
}
__device__ __forceinline__ float2 load_pair(uint32_t p) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(p));
    return v;
}
__device__ __forceinline__ float load_one(uint32_t p) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_pair(uint32_t p, float a, float b) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(p), "f"(a), "f"(b) : "memory");
}

// Positions of a ring along the axis, relative to the segment's start: input up to `mark` is
// loaded or on its way; `mark` itself goes to `slot`.
struct StreamRing {
    int size, mark, slot;
    __device__ __forceinline__ int slot_of(int q) const {  // q in [mark, mark + size)
        const int s = slot + (q - mark);
        return s >= size ? s - size : s;
    }
    __device__ __forceinline__ void advance(int to) {
        slot = slot_of(to - 1) + 1;
        if (slot >= size) slot -= size;
        mark = to;
    }
};

// The walk both passes share.  `load(to)` starts the copies up to position `to`;
// `chunk(q0, slot, ahead)` computes the outputs from q0 on, whose first input is in `slot`.
template <int CHUNK, typename Load, typename Compute>
__device__ __forceinline__ void stream_walk(const StreamShape &s, int len, StreamRing &ring, Load &&load, Compute &&chunk) {
    const int last = len + s.radius;  // no output needs input from here on
    int first = 0;                    // slot of the chunk's first input
    load(min(CHUNK + s.radius, last));
    for (int q0 = 0; q0 < len; q0 += CHUNK) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();  // the chunk's input is here, and the previous chunk's is free
        const int next = min(q0 + 2 * CHUNK + s.radius, last);
        if (next > ring.mark) load(next);
        chunk(q0, first);
        first += CHUNK;
        if (first >= s.ring) first -= s.ring;
    }
}

// One tap of a thread's 16 pairs; `u` is the tap's place modulo 16 (the window's rotation).
__device__ __forceinline__ void stream_tap(float k, int u, const float2 (&w)[kStreamM], float2 (&acc)[kStreamM]) {
    const float2 kk = make_float2(k, k);
#pragma unroll
    for (int i = 0; i < kStreamM; i++) acc[i] = __ffma2_rn(w[(u + i) % kStreamM], kk, acc[i]);
}

// acc[i] = sum over t of taps[t] * input(i + t), the taps in increasing order.  `load(u)`
// reads the input pair u places after the reader's, `step()` moves the reader on by 16
// places.  The load after the last tap reads a pair that no output uses.
template <typename Load, typename Step>
__device__ __forceinline__ void stream_conv(int n_taps, const StreamTaps &taps, float2 (&acc)[kStreamM], Load &&load,
                                            Step &&step) {
    float2 w[kStreamM];
#pragma unroll
    for (int i = 0; i < kStreamM; i++) {
        acc[i] = make_float2(0.0f, 0.0f);
        w[i] = load(i);
    }
    step();
    int t = 0;
#pragma unroll 1
    for (; t + kStreamM <= n_taps; t += kStreamM) {
#pragma unroll
        for (int u = 0; u < kStreamM; u++) {
            stream_tap(taps.k[t + u], u, w, acc);
            w[u] = load(u);
        }
        step();
    }
#pragma unroll
    for (int u = 0; u < kStreamM; u++) {
        if (t + u >= n_taps) break;
        stream_tap(taps.k[t + u], u, w, acc);
        w[u] = load(u);
    }
}

// FROM_MASK: the first repetition's z pass, which reads the {0, 1} field out of the
// bit-packed mask (32 times fewer bytes, and no pass to write that field).
template <bool FROM_MASK, bool ALIGNED>
__global__ void __launch_bounds__(kStreamThreads)
stream_axis_pass(const float *__restrict__ in, const uint32_t *__restrict__ mask, float *__restrict__ out,
                 const StreamShape s, const __grid_constant__ StreamTaps taps) {
    extern __shared__ __align__(16) float s_ring[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t b = blockIdx.x;
    const int64_t seg = b % s.segments;
    b /= s.segments;
    const int64_t i0 = (b % s.col_tiles) * kStreamCols, o = b / s.col_tiles;
    const int64_t a0 = seg * s.seg_len;
    const int len = (int) min((int64_t) s.seg_len, s.A - a0);
    // Rows [q_lo, q_hi) relative to a0 lie inside the volume; the others read as zero.
    const int q_lo = (int) max(-a0, (int64_t) -kMaxUnrolledRadius);
    const int q_hi = (int) min(s.A - a0, (int64_t) s.seg_len + kMaxUnrolledRadius);
    const int64_t origin = (o * s.A + a0) * s.I + i0;
    const int cols = (int) min((int64_t) kStreamCols, s.I - i0);  // ALIGNED: a multiple of 4
    StreamRing ring{s.ring, -s.radius, 0};
    const uint32_t base = shared_addr(s_ring);
    pass_begin();

    // A thread copies the columns c (and c + 32, one at a time) of every kStep-th row.
    constexpr int kPerCopy = ALIGNED ? 4 : 1;
    constexpr int kStep = ALIGNED ? kStreamThreads * 4 / kStreamCols : kStreamWarps;
    const int row0 = ALIGNED ? threadIdx.x / (kStreamCols / 4) : warp;
    const int c = ALIGNED ? threadIdx.x % (kStreamCols / 4) * 4 : lane;
    const bool c_ok = c < cols, c2_ok = !ALIGNED && c + 32 < cols;
    auto load = [&](int to) {
        if constexpr (FROM_MASK) {
            // 64 rows at a time: a thread fetches the 32 mask bits of half a row, and its
            // warp then writes 16 rows, a lane the columns 2 lane and 2 lane + 1.
            const int64_t words = (s.A * s.I + 31) >> 5;
            for (int qb = ring.mark; qb < to; qb += kStreamChunk) {
                const int q = qb + (threadIdx.x >> 1), half = (threadIdx.x & 1) * 32;
                uint32_t bits = 0;
                if (q >= q_lo && q < q_hi && q < to && half < cols) {
                    const int64_t first = origin + q * s.I + half, word = first >> 5;
                    const uint32_t next = word + 1 < words ? __ldg(mask + word + 1) : 0u;
                    bits = __funnelshift_l(next, __ldg(mask + word), (int) (first & 31));
                }
#pragma unroll
                for (int i = 0; i < kStreamM; i++) {
                    const uint32_t w = __shfl_sync(0xffffffffu, bits, 2 * i + (lane >> 4)) << (2 * (lane & 15));
                    const int row = qb + warp * kStreamM + i;
                    if (row < to)
                        store_pair(base + ring.slot_of(row) * kStreamRow + lane * 8, w >> 31 ? 1.0f : 0.0f,
                                   w & 0x40000000u ? 1.0f : 0.0f);
                }
            }
            ring.advance(to);
            return;
        }
        int q = ring.mark + row0, slot = ring.slot_of(q);
        const float *src = in + origin + q * s.I + c;
        const bool inside = ring.mark >= q_lo && to <= q_hi;
        for (; q < to; q += kStep, src += kStep * s.I) {
            const uint32_t dst = base + slot * kStreamRow + c * 4;
            const bool ok = inside || (q >= q_lo && q < q_hi);
            if (c_ok) async_copy<kPerCopy * 4>(dst, ok ? src : in, ok);
            if (c2_ok) async_copy<4>(dst + 128, ok ? src + 32 : in, ok);
            slot += kStep;
            if (slot >= s.ring) slot -= s.ring;
        }
        ring.advance(to);
    };
    stream_walk<kStreamChunk>(s, len, ring, load, [&](int q0, int slot) {
        const int q1 = q0 + warp * kStreamM;
        if (q1 >= len) return;
        slot += warp * kStreamM;
        if (slot >= s.ring) slot -= s.ring;
        float2 acc[kStreamM];
        uint32_t p = base + slot * kStreamRow + lane * 8;
        const uint32_t end = base + s.ring * kStreamRow;
        stream_conv(2 * s.radius + 1, taps, acc, [&](int u) { return load_pair(p + u * kStreamRow); },
                    [&]() {
                        p += kStreamM * kStreamRow;
                        if (p >= end) p -= s.ring * kStreamRow;
                    });
        float *dst = out + origin + q1 * s.I + 2 * lane;
        const bool ok0 = 2 * lane < cols, ok1 = 2 * lane + 1 < cols;
        if (!ok0) return;
#pragma unroll
        for (int i = 0; i < kStreamM; i++, dst += s.I) {
            if (q1 + i >= len) break;
            if (ALIGNED) {
                *reinterpret_cast<float2 *>(dst) = acc[i];
            } else {
                dst[0] = acc[i].x;
                if (ok1) dst[1] = acc[i].y;
            }
        }
    });
}

// `rows` = s.I rows of s.A voxels.  FINAL: the last repetition, which writes the uint16
// output and/or the FP32 field instead of the next repetition's field.
template <int MASK_FMT, bool FINAL>
__global__ void __launch_bounds__(kStreamThreads, 5)
stream_x_pass(const float *__restrict__ in, float *__restrict__ out, const void *__restrict__ mask,
              uint16_t *__restrict__ out_u16, float *__restrict__ field_out, const StreamShape s,
              const __grid_constant__ StreamTaps taps) {
    extern __shared__ __align__(16) float s_ring[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t seg = blockIdx.x % s.segments, r0 = (blockIdx.x / s.segments) * kStreamRowsX;
    const int64_t x0 = seg * s.seg_len;
    const int len = (int) min((int64_t) s.seg_len, s.A - x0);
    const int q_lo = (int) max(-x0, (int64_t) -kMaxUnrolledRadius);
    const int q_hi = (int) min(s.A - x0, (int64_t) s.seg_len + kMaxUnrolledRadius);
    const int rows = (int) min((int64_t) kStreamRowsX, s.I - r0);
    const int64_t origin = r0 * s.A + x0;
    const int pitch = stream_x_pitch(s.ring);
    StreamRing ring{s.ring, -s.radius, 0};
    const uint32_t base = shared_addr(s_ring);
    uint32_t *s_mask = reinterpret_cast<uint32_t *>(s_ring + kStreamRowsX * pitch);  // [2][rows][kStreamMaskWords]
    pass_begin();

    // A warp copies (and stores) rows warp, warp + 4, ..., 128 voxels of each at a time.
    constexpr int kPer = kStreamChunkX / 32;
    auto load = [&](int to) {
        for (int qb = ring.mark; qb < to; qb += kStreamChunkX) {
            uint32_t dst[kPer];
            bool want[kPer], ok[kPer];
#pragma unroll
            for (int j = 0; j < kPer; j++) {
                const int q = qb + 32 * j + lane;
                want[j] = q < to;
                ok[j] = q >= q_lo && q < q_hi;
                dst[j] = base + (warp * pitch + ring.slot_of(q)) * 4;
            }
            const bool inside = qb + kStreamChunkX <= to && qb >= q_lo && qb + kStreamChunkX <= q_hi;
            const float *src = in + origin + warp * s.A + qb + lane;
            const uint32_t row_bytes = kStreamWarps * pitch * 4;
            if (inside && rows == kStreamRowsX) {
#pragma unroll
                for (int r = 0; r < kStreamRowsX / kStreamWarps; r++, src += kStreamWarps * s.A) {
#pragma unroll
                    for (int j = 0; j < kPer; j++) async_copy<4>(dst[j] + r * row_bytes, src + 32 * j);
                }
            } else {
                const float *at[kPer];
                int64_t step[kPer];
#pragma unroll
                for (int j = 0; j < kPer; j++) {
                    at[j] = ok[j] ? src + 32 * j : in;
                    step[j] = ok[j] ? kStreamWarps * s.A : 0;
                }
#pragma unroll
                for (int r = 0; r < kStreamRowsX / kStreamWarps; r++) {
                    if (warp + r * kStreamWarps >= rows) break;
#pragma unroll
                    for (int j = 0; j < kPer; j++, at[j - 1] += step[j - 1])
                        if (want[j]) async_copy<4>(dst[j] + r * row_bytes, at[j], ok[j]);
                }
            }
        }
        ring.advance(to);
    };
    // The bit-packed mask words of the chunk at q0.
    auto load_mask = [&](int q0) {
        if (MASK_FMT == MAXI_MASK_U8) return;
        const int64_t words = (s.A * s.I + 31) >> 5;
        for (int i = threadIdx.x; i < kStreamRowsX * kStreamMaskWords; i += kStreamThreads) {
            const int row = i / kStreamMaskWords, j = i % kStreamMaskWords;
            const int64_t word = ((origin + row * s.A + q0) >> 5) + j;
            if (row < rows && word < words)
                async_copy<4>(shared_addr(s_mask + (q0 / kStreamChunkX & 1) * kStreamRowsX * kStreamMaskWords + i),
                              reinterpret_cast<const float *>(static_cast<const uint32_t *>(mask) + word));
        }
    };
    load_mask(0);
    stream_walk<kStreamChunkX>(s, len, ring, load, [&](int q0, int slot) {
        const int q1 = q0 + warp * kStreamMX;
        if (q0 + kStreamChunkX < len) load_mask(q0 + kStreamChunkX);
        float2 acc[kStreamM];
        int at = slot + warp * kStreamMX;
        if (at >= s.ring) at -= s.ring;
        if (q1 < len) {
            // The pair (x, x + 16): the second reader is one step ahead of the first.
            const uint32_t row = base + lane * pitch * 4, end = row + s.ring * 4;
            uint32_t p = row + at * 4, p16 = p + kStreamM * 4;
            if (p16 >= end) p16 = row;
            stream_conv(2 * s.radius + 1, taps, acc,
                        [&](int u) { return make_float2(load_one(p + u * 4), load_one(p16 + u * 4)); },
                        [&]() {
                            p = p16;
                            p16 += kStreamM * 4;
                            if (p16 >= end) p16 = row;
                        });
        }
        // Re-illuminated, the outputs take the places of the chunk's first inputs, which no
        // warp needs any more, and leave from there in whole rows.
        __syncthreads();
        if (q1 < len) {
            uint32_t lit = 0;  // bit i: voxel i
            if (MASK_FMT == MAXI_MASK_U8) {
                // A row's 32 bytes at a time, a lane per voxel (a row per lane, byte by byte, takes 32
                // sectors a load: 128 x 128 x 256, r = 8, four repetitions 167 us, 112 now).
                const uint8_t *m = static_cast<const uint8_t *>(mask) + origin + q1 + lane;
                const bool in_row = q1 + lane < len;
#pragma unroll 16
                for (int r = 0; r < kStreamRowsX; r++) {
                    const uint32_t row = __ballot_sync(0xffffffffu, in_row && r < rows && __ldg(m + r * s.A) != 0);
                    if (lane == r) lit = row;
                }
            } else if (lane < rows) {
                const uint32_t *m = s_mask + ((q0 / kStreamChunkX & 1) * kStreamRowsX + lane) * kStreamMaskWords + warp;
                lit = __brev(__funnelshift_l(m[1], m[0], (int) ((origin + lane * s.A + q1) & 31)));
            }
            float *dst = s_ring + lane * pitch + at;
#pragma unroll
            for (int i = 0; i < kStreamM; i++) {
                dst[i] = (lit >> i) & 1u ? 1.0f : acc[i].x;
                dst[i + kStreamM] = (lit >> (i + kStreamM)) & 1u ? 1.0f : acc[i].y;
            }
        }
        __syncthreads();
        const int count = min(kStreamChunkX, len - q0);
        uint32_t src[kPer];
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            int from = slot + 32 * j;
            if (from >= s.ring) from -= s.ring;
            src[j] = base + (warp * pitch + from + lane) * 4;
        }
        const int64_t idx = origin + warp * s.A + q0 + lane, step = kStreamWarps * s.A;
        auto put = [&](int64_t at_, int r, int j) {
            const float v = load_one(src[j] + r * kStreamWarps * pitch * 4);
            if (!FINAL) {
                out[at_ + 32 * j] = v;
            } else {
                if (out_u16) out_u16[at_ + 32 * j] = quantise_u16(v);
                if (field_out) field_out[at_ + 32 * j] = v;
            }
        };
        if (count == kStreamChunkX && rows == kStreamRowsX) {
#pragma unroll
            for (int r = 0; r < kStreamRowsX / kStreamWarps; r++)
#pragma unroll
                for (int j = 0; j < kPer; j++) put(idx + r * step, r, j);
        } else {
#pragma unroll 1
            for (int r = 0; r < kStreamRowsX / kStreamWarps && warp + r * kStreamWarps < rows; r++)
#pragma unroll
                for (int j = 0; j < kPer; j++)
                    if (32 * j + lane < count) put(idx + r * step, r, j);
        }
    });
}

}  // namespace maxi
