// Combination of the Gaussian (diffusion) field with the implant EDT field:
// the step after the diffusion in maxibone's pipeline,
// src/processing_steps/0975_combine_fields.py:38-62.  On uint16 fields G, E
// [nz][ny][nx] and the cylinder mask C[y][x] of generate_cylinder_mask
// (src/lib/py/helpers.py:411-434, here over ny and nx):
//
//   c   = G / max(G) - E / max(E)                     (FP32, as numpy does it)
//   c'  = (c + |min c|) / max(c + |min c|)
//   c'' = c' * C
//   out = to_int(c'') * C,  to_int = normalized_convert<float, uint16_t>
//         (src/lib/cpp/include/general.hh:78-118): (x - vmin) / (vmax - vmin) * 65535, truncated
//
// Every step after c is monotone non-decreasing in c (rounding included), so
// the extremes the later steps need follow from the extremes of c over all
// voxels and over the voxels inside the cylinder: two reduction passes (the
// field maxima, then those extremes) and one conversion pass, each a read of
// both fields -- HBM-bound: 14 bytes per voxel.  The scalar steps between the passes are
// done by every thread of the next pass, in FP32 in numpy's order, so the host reads back
// once, at the end.  The cylinder is convex along x for every row, so each row's
// inside voxels are one x interval, found on the host with numpy's own FP64
// arithmetic (linspace(-1, 1, n)[i] = i * (2 / (n - 1)) - 1, last point 1).
//
// Divisions.  Two per voxel of the second pass and four of the third, all by per-call
// scalars, bound those passes as divide sequences (803 and 1205 us at 384 x 1000 x 1000,
// against 376 for the maxima).  They are done with the scalar's correctly rounded
// reciprocal y instead: q = a y, then q + (a - q b) y with two FMAs, which is the
// correctly rounded quotient (P. Markstein, Computation of elementary functions on the
// IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990, theorem 8.2) away from
// over- and underflow; scalars that could bring one about keep the division.  Conversions
// between uint16 and FP32 go through the bits of 2^23 + v rather than the quarter-rate
// conversion instructions.
// Every integer quotient of two uint16 values was compared with the division, and 2^31
// random ones: all equal.
// 384 x 1000 x 1000 on a B200, before and now: maxima 376 and 222 us (6.9 TB/s from DRAM and
// L2), extremes 803 and 276, conversion 1205 and 385 (6.0 TB/s).
#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "host_copy.h"
#include "host_util.h"
#include "scratch.h"

namespace maxi {
namespace {

// All-zero to start with: minima are kept as maxima of the complemented keys.
struct CombineStats {
    unsigned int gmax, emax;          // field maxima
    unsigned int ncmin, cmax;         // extremes of c over all voxels (order-preserving keys)
    unsigned int ncmin_in, cmax_in;   // the same inside the cylinder
    unsigned int pad[2];
};

// Float <-> unsigned key with the same order (for atomicMax).
__device__ __forceinline__ unsigned int fkey(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned int k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Correctly rounded division by a scalar (see the top of the file).
struct Divisor {
    float b, y;
    bool plain;  // over- or underflow possible: divide
    template <bool PLAIN = false>
    __device__ __forceinline__ float2 quotient(float2 a) const {
        if (PLAIN) return make_float2(__fdiv_rn(a.x, b), __fdiv_rn(a.y, b));
        const float2 yy = make_float2(y, y), q = __fmul2_rn(a, yy);
        return __ffma2_rn(__ffma2_rn(q, make_float2(-b, -b), a), yy, q);
    }
};
__device__ __forceinline__ Divisor divisor(float b) {
    return {b, __fdiv_rn(1.0f, b), !(b >= 0x1p-60f && b <= 0x1p60f)};
}
// c = G / gm - E / em, in numpy's FP32 operations.
__device__ __forceinline__ float2 combined(const Divisor &by_g, const Divisor &by_e, float2 g, float2 e) {
    return __ffma2_rn(by_e.quotient(e), make_float2(-1.0f, -1.0f), by_g.quotient(g));
}

// Both halves of w as floats.
__device__ __forceinline__ float2 halves(uint32_t w) {
    const float2 v = make_float2(__uint_as_float(__byte_perm(w, 0x4b000000u, 0x7610)),
                                 __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7632)));
    return __fadd2_rn(v, make_float2(-8388608.0f, -8388608.0f));
}

// The maxima of both fields over the flat volume, in packed 16-bit lanes.
__global__ void __launch_bounds__(256) field_maxima(const uint16_t *__restrict__ g, const uint16_t *__restrict__ e,
                                                    int64_t n, bool vec, CombineStats *st) {
    const int64_t stride = (int64_t) gridDim.x * blockDim.x, thread = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
    unsigned int gm = 0, em = 0;
    int64_t done = 0;
    if (vec) {
        constexpr int kAtOnce = 4;
        const uint4 *gp = reinterpret_cast<const uint4 *>(g), *ep = reinterpret_cast<const uint4 *>(e);
        const int64_t groups = n / 8;
        for (int64_t i = (int64_t) blockIdx.x * kAtOnce * blockDim.x + threadIdx.x; i < groups; i += kAtOnce * stride) {
            uint4 a[kAtOnce], b[kAtOnce];
#pragma unroll
            for (int k = 0; k < kAtOnce; k++) {
                const int64_t j = min(i + k * blockDim.x, groups - 1);  // past the end: the last group again
                a[k] = __ldg(gp + j), b[k] = __ldg(ep + j);
            }
#pragma unroll
            for (int k = 0; k < kAtOnce; k++) {
                gm = __vmaxu2(gm, __vmaxu2(__vmaxu2(a[k].x, a[k].y), __vmaxu2(a[k].z, a[k].w)));
                em = __vmaxu2(em, __vmaxu2(__vmaxu2(b[k].x, b[k].y), __vmaxu2(b[k].z, b[k].w)));
            }
        }
        done = groups * 8;
    }
    for (int64_t i = done + thread; i < n; i += stride) {
        gm = __vmaxu2(gm, __ldg(g + i));
        em = __vmaxu2(em, __ldg(e + i));
    }
    gm = __reduce_max_sync(0xffffffffu, max(gm >> 16, gm & 0xffffu));
    em = __reduce_max_sync(0xffffffffu, max(em >> 16, em & 0xffffu));
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&st->gmax, gm);
        atomicMax(&st->emax, em);
    }
}

// The walk of the other two passes: `lanes` (a power of two; of all the launch's threads in order)
// threads per row, 8 voxels each at a time (VEC: rows are 16-byte aligned) or one; row(r) for
// every row, then voxels(r, x, a, b) with the two fields' voxels from x on.  Row indices stay
// below 2^32 (the host checks), so their division is 32-bit.  A warp to a row, or more threads where
// there are too few rows for the chip (1 x 4 x 4194304: the two passes 11.7 ms with a warp, 0.04 now).
template <bool VEC, typename Row, typename Voxels>
__device__ __forceinline__ void for_rows(const uint16_t *__restrict__ g, const uint16_t *__restrict__ e, int64_t rows,
                                         uint32_t nx, int lanes, Row &&row, Voxels &&voxels) {
    constexpr int V = VEC ? 8 : 1, kAtOnce = VEC ? 2 : 4;
    const int thread = blockIdx.x * blockDim.x + threadIdx.x, lane = thread & (lanes - 1);
    const int64_t first = thread / lanes;
    const int64_t step = (int64_t) gridDim.x * blockDim.x / lanes;
    for (int64_t r = first; r < rows; r += step) {
        row(r);
        const uint16_t *gr = g + r * nx, *er = e + r * nx;
        for (uint32_t x0 = lane * V; x0 < nx; x0 += kAtOnce * lanes * V) {
            uint4 a[kAtOnce], b[kAtOnce];
#pragma unroll
            for (int k = 0; k < kAtOnce; k++) {
                const uint32_t x = x0 + k * lanes * V;
                if (x < nx) {
                    if (VEC) {
                        a[k] = __ldg(reinterpret_cast<const uint4 *>(gr + x));
                        b[k] = __ldg(reinterpret_cast<const uint4 *>(er + x));
                    } else {
                        a[k].x = __ldg(gr + x);
                        b[k].x = __ldg(er + x);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kAtOnce; k++) {
                const uint32_t x = x0 + k * lanes * V;
                if (x < nx) voxels(r, x, a[k], b[k]);
            }
            if (nx - x0 <= (uint32_t) (kAtOnce * lanes * V)) break;  // (x0 may be about to wrap around)
        }
    }
}
// Extremes of c = G / gm - E / em with numpy's FP32 operations (no contraction).
template <bool VEC>
__global__ void __launch_bounds__(256) combined_extremes(const uint16_t *__restrict__ g, const uint16_t *__restrict__ e,
                                                         int64_t rows, uint32_t ny, uint32_t nx, int lanes,
                                                         const uint2 *__restrict__ inside, CombineStats *st) {
    constexpr int V = VEC ? 8 : 1;
    if (st->gmax == 0 || st->emax == 0) return;  // the host reports it
    const Divisor by_g = divisor((float) st->gmax), by_e = divisor((float) st->emax);
    const float inf = __int_as_float(0x7f800000);
    float lo = inf, hi = -inf, lo_in = inf, hi_in = -inf;
    uint2 iv = make_uint2(0, 0);
    for_rows<VEC>(g, e, rows, nx, lanes, [&](int64_t r) { iv = __ldg(inside + (uint32_t) r % ny); },
                  [&](int64_t, uint32_t x, const uint4 &wa, const uint4 &wb) {
                      const uint32_t a[4] = {wa.x, wa.y, wa.z, wa.w}, b[4] = {wb.x, wb.y, wb.z, wb.w};
                      float c[V + 1], l = inf, h = -inf;
#pragma unroll
                      for (int i = 0; i < V; i += 2) {
                          const float2 p = combined(by_g, by_e, halves(a[i / 2]), halves(b[i / 2]));
                          c[i] = p.x;
                          c[i + 1] = p.y;  // (one voxel at a time: of no voxel)
                      }
#pragma unroll
                      for (int i = 0; i < V; i++) {
                          l = fminf(l, c[i]);
                          h = fmaxf(h, c[i]);
                      }
                      lo = fminf(lo, l);
                      hi = fmaxf(hi, h);
                      if (x >= iv.x && x + V <= iv.y) {
                          lo_in = fminf(lo_in, l);
                          hi_in = fmaxf(hi_in, h);
                      } else if (x + V > iv.x && x < iv.y) {
#pragma unroll
                          for (int i = 0; i < V; i++)
                              if (x + i >= iv.x && x + i < iv.y) {
                                  lo_in = fminf(lo_in, c[i]);
                                  hi_in = fmaxf(hi_in, c[i]);
                              }
                      }
                  });
    const unsigned int k[4] = {lo <= hi ? ~fkey(lo) : 0u, lo <= hi ? fkey(hi) : 0u, lo_in <= hi_in ? ~fkey(lo_in) : 0u,
                               lo_in <= hi_in ? fkey(hi_in) : 0u};
    unsigned int *to = &st->ncmin;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const unsigned int m = __reduce_max_sync(0xffffffffu, k[i]);
        if ((threadIdx.x & 31) == 0 && m) atomicMax(to + i, m);
    }
}

// any_inside / any_outside: whether the cylinder has voxels, and whether some are outside it.
template <bool VEC>
__global__ void __launch_bounds__(256) combined_convert(const uint16_t *__restrict__ g, const uint16_t *__restrict__ e,
                                                        uint16_t *__restrict__ out, int64_t rows, uint32_t ny,
                                                        uint32_t nx, int lanes, const uint2 *__restrict__ inside,
                                                        bool any_inside,
                                                        bool any_outside, const CombineStats *__restrict__ st) {
    constexpr int V = VEC ? 8 : 1;
    if (st->gmax == 0 || st->emax == 0) return;
    // The scalar steps in FP32, in numpy's order.
    const Divisor by_g = divisor((float) st->gmax), by_e = divisor((float) st->emax);
    const float shift = fabsf(key_float(~st->ncmin));
    const Divisor by_denom = divisor(__fadd_rn(key_float(st->cmax), shift));
    float vmin = 0.0f, vmax = 0.0f;
    if (any_inside) {
        const float lo = __fdiv_rn(__fadd_rn(key_float(~st->ncmin_in), shift), by_denom.b);
        const float hi = __fdiv_rn(__fadd_rn(key_float(st->cmax_in), shift), by_denom.b);
        // the host's std::min and std::max, which give the first argument for a NaN
        vmin = any_outside ? (lo < 0.0f ? lo : 0.0f) : lo;
        vmax = any_outside ? (0.0f < hi ? hi : 0.0f) : hi;
    }
    const Divisor by_range = divisor(__fsub_rn(vmax, vmin));
    const bool some = by_range.b > 0.0f;
    auto walk = [&](auto plain) {
        constexpr bool PLAIN = decltype(plain)::value;
        uint2 iv = make_uint2(0, 0);
        for_rows<VEC>(
            g, e, rows, nx, lanes, [&](int64_t r) { iv = __ldg(inside + (uint32_t) r % ny); },
            [&](int64_t r, uint32_t x, const uint4 &wa, const uint4 &wb) {
                const uint32_t a[4] = {wa.x, wa.y, wa.z, wa.w}, b[4] = {wb.x, wb.y, wb.z, wb.w};
                uint32_t q[4] = {0u, 0u, 0u, 0u};
                if (some && x + V > iv.x && x < iv.y) {
#pragma unroll
                    for (int i = 0; i < (V + 1) / 2; i++) {
                        const float2 c = combined(by_g, by_e, halves(a[i]), halves(b[i]));
                        const float2 c1 = by_denom.quotient<PLAIN>(__fadd2_rn(c, make_float2(shift, shift)));
                        const float2 u = by_range.quotient<PLAIN>(__fadd2_rn(c1, make_float2(-vmin, -vmin)));
                        float2 t = __fmul2_rn(u, make_float2(65535.0f, 65535.0f));
                        // Inside the cylinder t lies in [0, 65535] (or is a NaN, taken as 0): the low bits of its
                        // sum with 2^23 are its integer part.
                        if (PLAIN) t = make_float2(fmaxf(t.x, 0.0f), fmaxf(t.y, 0.0f));
                        t = __fadd2_rz(t, make_float2(8388608.0f, 8388608.0f));
                        q[i] = __byte_perm(__float_as_uint(t.x), __float_as_uint(t.y), 0x5410);
                    }
                    if (x < iv.x || x + V > iv.y) {  // the cylinder's edge
#pragma unroll
                        for (int i = 0; i < V; i++)
                            if (x + i < iv.x || x + i >= iv.y) q[i / 2] &= i % 2 ? 0x0000ffffu : 0xffff0000u;
                    }
                }
                if constexpr (VEC) *reinterpret_cast<uint4 *>(out + r * nx + x) = make_uint4(q[0], q[1], q[2], q[3]);
                else out[r * nx + x] = (uint16_t) q[0];
            });
    };
    if (by_denom.plain || by_range.plain) walk(std::true_type{});
    else walk(std::false_type{});
}

// numpy.linspace(-1, 1, n)[i] in FP64 (numpy: arange * step + start, last point = stop).
double linspace_pm1(int64_t i, int64_t n) {
    if (n == 1) return -1.0;
    if (i == n - 1) return 1.0;
    const double step = 2.0 / (double) (n - 1);
    volatile double t = (double) i * step;  // two roundings, as numpy (no fused multiply-add)
    return t + -1.0;
}

// Inside interval [x0, x1) of each row y of generate_cylinder_mask(ny, nx):
// xs[x]^2 + ys[y]^2 < 1 in FP64.  xs^2 falls then rises along x and fl(a + c) is
// monotone in a, so a row's inside voxels run from a first to a last index around
// the argmin of xs^2: two binary searches per row, exact.
void cylinder_intervals(int64_t ny, int64_t nx, std::vector<uint2> &inside, bool &any_outside, bool &any_inside) {
    std::vector<double> xs2(nx);
    int64_t xm = 0;
    for (int64_t x = 0; x < nx; x++) {
        const double v = linspace_pm1(x, nx);
        volatile double sq = v * v;
        xs2[x] = sq;
        if (xs2[x] < xs2[xm]) xm = x;
    }
    inside.assign(ny, make_uint2(0, 0));
    any_outside = any_inside = false;
    for (int64_t y = 0; y < ny; y++) {
        const double v = linspace_pm1(y, ny);
        volatile double ys2 = v * v;
        auto in = [&](int64_t x) {
            volatile double s = xs2[x] + ys2;
            return s < 1.0;
        };
        int64_t x0 = 0, x1 = 0;
        if (in(xm)) {
            int64_t lo = 0, hi = xm;  // first inside index in [0, xm]
            while (lo < hi) {
                const int64_t mid = (lo + hi) / 2;
                if (in(mid)) hi = mid;
                else lo = mid + 1;
            }
            x0 = lo;
            lo = xm + 1, hi = nx;  // first outside index in [xm + 1, nx]
            while (lo < hi) {
                const int64_t mid = (lo + hi) / 2;
                if (in(mid)) lo = mid + 1;
                else hi = mid;
            }
            x1 = lo;
        }
        inside[y] = make_uint2((uint32_t) x0, (uint32_t) x1);
        any_outside |= x0 > 0 || x1 < nx;
        any_inside |= x1 > x0;
    }
}

// Zeroes the voxels of each row outside its cylinder interval (one block per row
// at a time; the inside voxels are neither read nor written).
__global__ void cylinder_zero(uint16_t *__restrict__ f, int64_t rows, int64_t ny, int nx,
                              const uint2 *__restrict__ iv) {
    for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
        const uint2 in = __ldg(iv + row % ny);
        uint16_t *r = f + row * nx;
        for (int x = threadIdx.x; x < (int) in.x; x += blockDim.x) r[x] = 0;
        for (int x = (int) in.y + threadIdx.x; x < nx; x += blockDim.x) r[x] = 0;
    }
}

}  // namespace
}  // namespace maxi

using namespace maxi;

extern "C" int maxi_combine_fields(const uint16_t *gauss, const uint16_t *edt, int64_t nz, int64_t ny, int64_t nx,
                                   uint16_t *output, void *stream) {
    clear_error();
    if (!gauss || !edt || !output) return set_error(MAXI_ERR_INVALID_ARGUMENT, "NULL pointer");
    if (nz <= 0 || ny <= 0 || nx <= 0)
        return set_error(MAXI_ERR_INVALID_ARGUMENT, "shape (%lld, %lld, %lld) has an empty axis", (long long) nz,
                         (long long) ny, (long long) nx);
    int rc = require_device();
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t rows = nz * ny;
    if (rows * nx >= (int64_t(1) << 32))
        return set_error(MAXI_ERR_UNSUPPORTED, "volumes of 2^32 voxels or more are not served by this step");

    std::vector<uint2> inside;
    bool any_outside = false, any_inside = false;
    cylinder_intervals(ny, nx, inside, any_outside, any_inside);

    const size_t iv_bytes = (size_t) ny * sizeof(uint2);
    SpareBuffer scratch;
    if ((rc = scratch.take(256 + iv_bytes, st, "field combination"))) return rc;
    CombineStats *d_st = reinterpret_cast<CombineStats *>(scratch.data());
    uint2 *d_iv = reinterpret_cast<uint2 *>(scratch.data() + 256);
    const bool aligned = ((reinterpret_cast<uintptr_t>(gauss) | reinterpret_cast<uintptr_t>(edt) |
                           reinterpret_cast<uintptr_t>(output)) & 15) == 0;
    const bool vec = nx % 8 == 0 && aligned;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int threads = 256;
    int lanes = 1;
    // (At least 64 voxels a thread: every warp ends in four additions to the same words.)
    const int64_t wanted = std::min<int64_t>((int64_t) sms * 1024, rows * nx / 64);
    while (lanes * (vec ? 8 : 1) < nx && (lanes < 32 || rows * lanes < wanted)) lanes *= 2;
    const unsigned grid_flat = (unsigned) std::min<int64_t>(ceil_div(ceil_div(rows * nx, 8), threads), (int64_t) sms * 16);
    // (Of more lanes than a block has threads, whole rows: the grid is a multiple of lanes / threads.)
    const int64_t blocks = std::min<int64_t>(ceil_div(rows * lanes, threads), (int64_t) sms * 16);
    const unsigned grid = (unsigned) (lanes > threads ? round_up(blocks, lanes / threads) : blocks);
    CombineStats pageable{};
    const StagingBuffer staging;
    CombineStats &h = staging.data() ? *static_cast<CombineStats *>(staging.data()) : pageable;
    cudaError_t e = cudaMemsetAsync(d_st, 0, sizeof(CombineStats), st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_iv, inside.data(), iv_bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        field_maxima<<<grid_flat, threads, 0, st>>>(gauss, edt, rows * nx, aligned, d_st);
        auto extremes = vec ? combined_extremes<true> : combined_extremes<false>;
        extremes<<<grid, threads, 0, st>>>(gauss, edt, rows, (uint32_t) ny, (uint32_t) nx, lanes, d_iv, d_st);
        auto convert = vec ? combined_convert<true> : combined_convert<false>;
        convert<<<grid, threads, 0, st>>>(gauss, edt, output, rows, (uint32_t) ny, (uint32_t) nx, lanes, d_iv,
                                          any_inside, any_outside, d_st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d_st, sizeof(h), cudaMemcpyDeviceToHost, st);
    cudaError_t e2 = scratch.give_back();  // waits for the stream: the host intervals are free after it
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) return set_cuda_error(e, "combine_fields");
    if (h.gmax == 0 || h.emax == 0)
        return set_error(MAXI_ERR_INVALID_ARGUMENT, "the %s field is all zero (the combination divides by its maximum)",
                         h.gmax == 0 ? "Gaussian" : "EDT");
    return MAXI_OK;
}

extern "C" int maxi_mask_cylinder(uint16_t *field, int64_t nz, int64_t ny, int64_t nx, void *stream) {
    clear_error();
    if (!field) return set_error(MAXI_ERR_INVALID_ARGUMENT, "NULL pointer");
    if (nz <= 0 || ny <= 0 || nx <= 0)
        return set_error(MAXI_ERR_INVALID_ARGUMENT, "shape (%lld, %lld, %lld) has an empty axis", (long long) nz,
                         (long long) ny, (long long) nx);
    if (nx >= (int64_t(1) << 31)) return set_error(MAXI_ERR_UNSUPPORTED, "rows of 2^31 voxels or more are not served");
    int rc = require_device();
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    std::vector<uint2> inside;
    bool any_outside = false, any_inside = false;
    cylinder_intervals(ny, nx, inside, any_outside, any_inside);
    if (!any_outside) return MAXI_OK;
    uint2 *d_iv = nullptr;
    const size_t bytes = inside.size() * sizeof(uint2);
    if (cudaMallocAsync(reinterpret_cast<void **>(&d_iv), bytes, st) != cudaSuccess) {
        cudaGetLastError();
        return set_error(MAXI_ERR_OUT_OF_MEMORY, "could not allocate %zu bytes of intervals", bytes);
    }
    cudaError_t e = cudaMemcpyAsync(d_iv, inside.data(), bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const int64_t rows = nz * ny;
        const unsigned grid = (unsigned) std::min<int64_t>(rows, (int64_t) sms * 16);
        cylinder_zero<<<grid, 128, 0, st>>>(field, rows, ny, (int) nx, d_iv);
        e = cudaGetLastError();
    }
    cudaError_t e2 = cudaStreamSynchronize(st);  // the host intervals must outlive the copy
    cudaFreeAsync(d_iv, st);
    if (e == cudaSuccess) e = e2;
    return e == cudaSuccess ? MAXI_OK : set_cuda_error(e, "cylinder mask");
}
