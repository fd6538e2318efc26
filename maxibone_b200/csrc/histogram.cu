// The reference's histograms module on the GPU.
//
// field_histogram (src/lib/cpp/cpu/histograms.cc:231-305, via
// src/pybind/histograms-pybind.cc:81-107; the consumer of the diffusion field in
// src/processing_steps/1000_compute_histograms.py:470-472): for every voxel (Z, Y, X)
// with Y >= y_start and X >= x_start, the uint16 voxel value v counts as 0 outside
// [vmin, vmax] and is binned as floor((voxel_bins - 1) * ((v - vmin) / (vmax - vmin)))
// in FP64; the field is read at (min(nz - 1, floor(Z * nz/nZ)), floor(Y * ny/nY),
// floor(X * nx/nX)) and binned the same way over [fmin, fmax]; pairs with a zero
// voxel or a zero field value are skipped; bins[field_bin][voxel_bin] += 1.  Field
// bins outside [0, field_bins) -- out-of-bounds writes in the reference -- are skipped.
//
// axis_histograms (histograms.cc:14-80, via histograms-pybind.cc:30-66): each
// counted voxel of a z-block adds to x_bins[x], y_bins[y], z_bins[z] and
// r_bins[floor(sqrt((x-cx)^2 + (y-cy)^2))] at its voxel bin.
//
// Exact binning without FP64 in the kernels.  Each bin expression is a monotone, very
// nearly linear function of an integer value, so the host evaluates it with the reference's
// own FP64 arithmetic for all 65536 values and fits a fixed-point line whose floor is the
// reference's bin for every counted one (checked value by value): two integer instructions per
// bin and no table.  Where no line fits, thresholds T[b] (the smallest counted value whose
// bin is >= b) settle the fixed-point bin by one comparison each way.
//
// Counting, field_histogram.  One thread takes 8 consecutive voxels of a row (one 16-byte load
// when rows are 16-byte aligned), adds runs of equal keys once and issues one 64-bit
// reduction per run into the histogram (L2-resident at the pipeline's 2048 x 4096); each
// block walks one contiguous range of rows.
//
// Counting, axis_histograms.  L2 takes about 150 to 190 G reductions per second on random
// cells, shared memory 2300 G (measured), and a voxel counts in four histograms.  So each
// histogram has a kernel of its own whose blocks own a part of it in shared memory and read
// the voxels that belong there: a y (or z) the rows of that y (or z), a strip of 8 x its
// columns, a ring of radii its pixels.  Voxels are read four times and reductions go out once
// per block and counted cell.  A 128 x 1024 x 1024 block at 4096 bins on a B200: z and y 98 us
// each, x 155 (half of each 32-byte sector is another strip's), r 251 (a ring's row interval
// fills about 40% of its sectors); before, one kernel with two reductions per voxel and a
// shared histogram per row, 1611 us.
#include <cmath>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "host_util.h"

namespace maxi {
namespace {

constexpr int kVec = 8;  // voxels per thread (one 16-byte load)

// A counted value range [lo, lo + span] and the bin of each value in it.
struct BinMap {
    const uint32_t *T;  // thresholds T[0 .. bins], or NULL where the fixed-point bin is exact
    int lo, span, bins;
    uint32_t mul_lo, mul_hi;  // the bin's slope and offset in 1/2^32
    uint64_t offset;
};

// The bin of v, or -1 if v is not counted.  EXACT: the map has no thresholds.
template <bool EXACT = false>
__device__ __forceinline__ int bin_of(const BinMap &m, int v) {
    const uint32_t d = (uint32_t) (v - m.lo);
    int b = (int) (((uint64_t) d * m.mul_lo + m.offset) >> 32) + (int) (d * m.mul_hi);
    if (!EXACT && m.T && d <= (uint32_t) m.span) {
        b = min(max(b, 0), m.bins - 1);
        if ((uint32_t) v < __ldg(m.T + b)) b--;
        else if ((uint32_t) v >= __ldg(m.T + b + 1)) b++;
    }
    return d <= (uint32_t) m.span ? b : -1;
}

// Voxels are read once: loaded evict-first, so the L2-resident bins stay in L2.
__device__ __forceinline__ void load_row8(const uint16_t *p, int (&v)[kVec]) {
    const uint4 w = __ldcs(reinterpret_cast<const uint4 *>(p));
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        v[2 * k] = (int) (u[k] & 0xffffu);
        v[2 * k + 1] = (int) (u[k] >> 16);
    }
}

// VEC8: rows are 16-byte aligned (nX % 8 == 0, aligned base); otherwise one voxel at a time.
template <bool VEC8>
__global__ void field_histogram_kernel(const uint16_t *__restrict__ voxels, const uint16_t *__restrict__ field,
                                       int64_t nZ, int64_t nY, int nX, int64_t ny, int64_t nx, int64_t y_start,
                                       int x_start, BinMap vm, BinMap fm, const int32_t *__restrict__ zmap,
                                       const int32_t *__restrict__ ymap, const int32_t *__restrict__ xmap,
                                       unsigned long long *__restrict__ bins, int64_t voxel_bins) {
    constexpr int V = VEC8 ? kVec : 1;
    const int x_first = x_start / V * V;
    // Each block takes one contiguous range of rows, so the blocks at work at any time
    // sit far apart in the volume: a smooth field gives neighbouring rows the same
    // keys, and same-address reductions from many blocks at once serialise in L2.
    const int64_t rows = nZ * nY, per = (rows + gridDim.x - 1) / gridDim.x;
    const int64_t row_end = min(rows, (int64_t) (blockIdx.x + 1) * per);
    for (int64_t row = (int64_t) blockIdx.x * per; row < row_end; row++) {
        const int64_t Z = row / nY, Y = row - Z * nY;
        if (Y < y_start) continue;
        const uint16_t *vrow = voxels + row * nX;
        const uint16_t *frow = field + ((int64_t) __ldg(zmap + Z) * ny + __ldg(ymap + Y)) * nx;
        for (int X = x_first + threadIdx.x * V; X < nX; X += blockDim.x * V) {
            int v[V];
            if constexpr (VEC8) load_row8(vrow + X, v);
            else v[0] = __ldcs(vrow + X);
            long long run_key = -1;
            unsigned run = 0;
#pragma unroll
            for (int j = 0; j < V; j++) {
                const int x = X + j;
                long long key = -1;
                const int vb = x >= x_start ? bin_of(vm, v[j]) : -1;
                if (vb >= 0) {
                    const int fb = bin_of(fm, __ldg(frow + __ldg(xmap + x)));
                    if (fb >= 0) key = (long long) fb * voxel_bins + vb;
                }
                if (key == run_key) {
                    run++;
                } else {
                    if (run_key >= 0) atomicAdd(bins + run_key, (unsigned long long) run);
                    run_key = key;
                    run = 1;
                }
            }
            if (run_key >= 0) atomicAdd(bins + run_key, (unsigned long long) run);
        }
    }
}

// floor(sqrt(n)) for 0 <= n < 2^50: a float estimate corrected in integers.  In that
// range it equals floor of the correctly rounded double sqrt of n, the reference's
// std::floor(std::sqrt(uint64)), since (k + 1)^2 - 1 and (k + 1)^2 stay apart in double.
__device__ __forceinline__ int64_t isqrt64(int64_t n) {
    int64_t r = (int64_t) sqrtf((float) n);
    while (r * r > n) r--;
    while ((r + 1) * (r + 1) <= n) r++;
    return r;
}

// axis_histograms where the shared-memory forms below do not apply: every voxel adds to the
// global bins, runs of equal keys once (x: every voxel).
template <bool VEC8>
__global__ void axis_histograms_direct(const uint16_t *__restrict__ voxels, int64_t nzl, int64_t Ny, int Nx,
                                       int64_t z_start, int64_t y_start, int x_start, BinMap vm, int64_t cy,
                                       int64_t cx, unsigned long long *__restrict__ x_bins,
                                       unsigned long long *__restrict__ y_bins,
                                       unsigned long long *__restrict__ z_bins,
                                       unsigned long long *__restrict__ r_bins, int voxel_bins, int64_t n_r) {
    constexpr int V = VEC8 ? kVec : 1;
    const int x_first = x_start / V * V;
    for (int64_t row = blockIdx.x; row < nzl * Ny; row += gridDim.x) {
        const int64_t zl = row / Ny, y = row - zl * Ny;
        if (y < y_start) continue;
        const uint16_t *vrow = voxels + row * Nx;
        const int64_t dy2 = (y - cy) * (y - cy);
        unsigned long long *yrow = y_bins + y * voxel_bins, *zrow = z_bins + (z_start + zl) * voxel_bins;
        for (int X = x_first + threadIdx.x * V; X < Nx; X += blockDim.x * V) {
            int v[V];
            if constexpr (VEC8) load_row8(vrow + X, v);
            else v[0] = __ldcs(vrow + X);
            long long r_key = -1;
            unsigned r_run = 0;
            int b_key = -1;
            unsigned b_run = 0;
#pragma unroll
            for (int j = 0; j < V; j++) {
                const int x = X + j;
                const int vb = x >= x_start ? bin_of(vm, v[j]) : -1;
                long long rk = -1;
                if (vb >= 0) {
                    atomicAdd(x_bins + (int64_t) x * voxel_bins + vb, 1ull);
                    const int64_t r = isqrt64(dy2 + (x - cx) * (x - cx));
                    if (r < n_r) rk = r * voxel_bins + vb;
                }
                if (rk == r_key) {
                    r_run++;
                } else {
                    if (r_key >= 0) atomicAdd(r_bins + r_key, (unsigned long long) r_run);
                    r_key = rk;
                    r_run = 1;
                }
                if (vb == b_key) {
                    b_run++;
                } else {
                    if (b_key >= 0) {
                        atomicAdd(yrow + b_key, (unsigned long long) b_run);
                        atomicAdd(zrow + b_key, (unsigned long long) b_run);
                    }
                    b_key = vb;
                    b_run = 1;
                }
            }
            if (r_key >= 0) atomicAdd(r_bins + r_key, (unsigned long long) r_run);
            if (b_key >= 0) {
                atomicAdd(yrow + b_key, (unsigned long long) b_run);
                atomicAdd(zrow + b_key, (unsigned long long) b_run);
            }
        }
    }
}

// The block's counters, zeroed before and added to `bins` (the counted cells alone) after.
__device__ __forceinline__ void counters_clear(uint32_t *c, int n) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) c[i] = 0;
    __syncthreads();
}
__device__ __forceinline__ void counters_flush(const uint32_t *c, int n, unsigned long long *bins) {
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (const uint32_t k = c[i]) atomicAdd(bins + i, (unsigned long long) k);
}

// y_bins or z_bins: block (p, chunk) counts the rows row0(p), row0(p) + row_step, .. of one y
// (or z), from row chunk * per on, in one shared histogram.  A warp per row.
struct RowSets {
    int64_t sets, set_step, row_step, rows, first_row, per;  // per: rows of a chunk
    int64_t first_set;                                      // sets below are not counted
    unsigned long long *bins;                               // of set 0
};
template <bool VEC8, bool EXACT>
__global__ void __launch_bounds__(256) row_set_histograms(const uint16_t *__restrict__ voxels, int Nx, int x_start,
                                                          BinMap vm, RowSets s, int voxel_bins) {
    extern __shared__ uint32_t counters[];
    const int64_t set = s.first_set + blockIdx.x % (s.sets - s.first_set), chunk = blockIdx.x / (s.sets - s.first_set);
    const int64_t end = min(s.rows, s.first_row + (chunk + 1) * s.per);
    const int lane = threadIdx.x & 31;
    counters_clear(counters, voxel_bins);
    auto count = [&](int v) {
        const int b = bin_of<EXACT>(vm, v);
        if (b >= 0) atomicAdd(counters + b, 1u);
    };
    for (int64_t i = s.first_row + chunk * s.per + (threadIdx.x >> 5); i < end; i += blockDim.x >> 5) {
        const uint16_t *row = voxels + (set * s.set_step + i * s.row_step) * Nx;
        if (VEC8) {
            // Up to x_first one voxel per lane, then two loads of 8 ahead of their counting.
            const int x_first = (x_start + kVec - 1) / kVec * kVec;
            if (x_start + lane < x_first) count(__ldcs(row + x_start + lane));
            for (int x = x_first + lane * kVec; x < Nx; x += 64 * kVec) {
                int v[kVec], w[kVec];
                const bool second = x + 32 * kVec < Nx;
                load_row8(row + x, v);
                if (second) load_row8(row + x + 32 * kVec, w);
#pragma unroll
                for (int j = 0; j < kVec; j++) count(v[j]);
                if (second)
#pragma unroll
                    for (int j = 0; j < kVec; j++) count(w[j]);
            }
        } else {
            for (int x = x_start + lane; x < Nx; x += 32 * kVec) {
                int v[kVec];
#pragma unroll
                for (int j = 0; j < kVec; j++) v[j] = x + 32 * j < Nx ? __ldcs(row + x + 32 * j) : -1;
#pragma unroll
                for (int j = 0; j < kVec; j++)
                    if (v[j] >= 0) count(v[j]);
            }
        }
    }
    counters_flush(counters, voxel_bins, s.bins + set * voxel_bins);
}

// x_bins: block (strip, chunk) counts `strip` neighbouring x over the rows of the chunk, a
// row per thread, two rows loaded ahead of their counting.
template <bool VEC8, bool EXACT>
__global__ void __launch_bounds__(1024) strip_histograms(const uint16_t *__restrict__ voxels, int64_t rows, int64_t Ny,
                                                         int Nx, int64_t y_start, int x_start, BinMap vm, int strips,
                                                         int strip, int64_t per, unsigned long long *__restrict__ x_bins,
                                                         int voxel_bins) {
    extern __shared__ uint32_t counters[];
    const int x0 = blockIdx.x % strips * strip, width = min(strip, Nx - x0), skip = max(0, x_start - x0);
    const int64_t begin = blockIdx.x / strips * per, end = min(rows, begin + per);
    counters_clear(counters, width * voxel_bins);
    auto count = [&](int v, int j) {
        const int b = bin_of<EXACT>(vm, v);
        if (b >= 0 && j >= skip) atomicAdd(counters + j * voxel_bins + b, 1u);
    };
    for (int64_t row = begin + threadIdx.x; row < end; row += 2 * blockDim.x) {
        const int64_t next = row + blockDim.x;
        bool first = true, second = next < end;
        if (y_start > 0) {
            first = row % Ny >= y_start;
            second = second && next % Ny >= y_start;
        }
        const uint16_t *p = voxels + row * Nx + x0, *q = voxels + next * Nx + x0;
        int v[kVec], w[kVec];
        if (VEC8) {  // strips of 8
            if (first) load_row8(p, v);
            if (second) load_row8(q, w);
        } else {
#pragma unroll
            for (int j = 0; j < kVec; j++) {
                v[j] = first && j < width ? __ldg(p + j) : -1;
                w[j] = second && j < width ? __ldg(q + j) : -1;
            }
        }
        if (first)
#pragma unroll
            for (int j = 0; j < kVec; j++)
                if (VEC8 || v[j] >= 0) count(v[j], j);
        if (second)
#pragma unroll
            for (int j = 0; j < kVec; j++)
                if (VEC8 || w[j] >= 0) count(w[j], j);
    }
    counters_flush(counters, width * voxel_bins, x_bins + (int64_t) x0 * voxel_bins);
}

// floor(sqrt(n)), 0 <= n < 2^31: the float estimate is within one.
__device__ __forceinline__ int isqrt32(int n) {
    int r = (int) sqrtf((float) n);
    if ((uint32_t) r * (uint32_t) r > (uint32_t) n) r--;
    if ((uint32_t) (r + 1) * (uint32_t) (r + 1) <= (uint32_t) n) r++;
    return r;
}

// r_bins: block (ring, chunk) counts the pixels with ring * width <= r < (ring + 1) * width
// over the planes of the chunk.  Eight lanes take a row: its pixels of the ring are at most
// two x intervals (of about `width` each for most rows, hence eight), a lane per pixel, which
// reads that pixel of every plane, eight ahead of their counting.  The outer, larger rings
// start first.  Distances stay below 2^31 (the host checks).
template <bool EXACT>
__global__ void __launch_bounds__(1024) ring_histograms(const uint16_t *__restrict__ voxels, int64_t nzl, int Ny,
                                                        int Nx, int y_start, int x_start, BinMap vm, int cy, int cx,
                                                        int rings, int width, int64_t per,
                                                        unsigned long long *__restrict__ r_bins, int voxel_bins,
                                                        int n_r) {
    extern __shared__ uint32_t counters[];
    const int64_t chunks = (nzl + per - 1) / per;
    const int ring = rings - 1 - (int) (blockIdx.x / chunks);
    const int64_t z0 = blockIdx.x % chunks * per;
    const int planes = (int) min(per, nzl - z0);
    const int r0 = ring * width, r1 = min(r0 + width, n_r);
    counters_clear(counters, (r1 - r0) * voxel_bins);
    const int64_t plane = (int64_t) Ny * Nx;
    const int inner = r0 * r0, outer = r1 * r1 - 1;  // squared distances inner .. outer
    const int y_end = min(Ny - 1, cy + r1 - 1), lane = threadIdx.x & 7;
    for (int y = max(y_start, cy - r1 + 1) + (threadIdx.x >> 3); y <= y_end; y += blockDim.x >> 3) {
        const int dy2 = (y - cy) * (y - cy);
        const int far = isqrt32(outer - dy2), near = dy2 >= inner ? 0 : isqrt32(inner - dy2 - 1) + 1;
        // right: cx + near .. cx + far; left: cx - far .. cx - max(near, 1)
        const int right = max(cx + near, x_start), n_right = max(0, min(cx + far, Nx - 1) - right + 1);
        const int left = max(cx - far, x_start), n_left = max(0, min(cx - max(near, 1), Nx - 1) - left + 1);
        const uint16_t *row = voxels + z0 * plane + (int64_t) y * Nx;
        for (int k = lane; k < n_right + n_left; k += 8) {
            const int x = k < n_right ? right + k : left + (k - n_right);
            uint32_t *c = counters + (isqrt32(dy2 + (x - cx) * (x - cx)) - r0) * voxel_bins;
            const uint16_t *p = row + x;
            for (int z = 0; z < planes; z += 8, p += 8 * plane) {
                int v[8];
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = z + j < planes ? __ldg(p + j * plane) : -1;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int b = bin_of<EXACT>(vm, v[j]);
                    if (b >= 0 && v[j] >= 0) atomicAdd(c + b, 1u);
                }
            }
        }
    }
    counters_flush(counters, (r1 - r0) * voxel_bins, r_bins + (int64_t) r0 * voxel_bins);
}

// floor((bins - 1) * ((v - lo) / (hi - lo))) in FP64, as the reference writes it.
int64_t ref_bin(double v, double lo, double hi, int64_t bins) {
    volatile double t = (v - lo) / (hi - lo);
    volatile double u = (double) (bins - 1) * t;
    return (int64_t) std::floor((double) u);
}

// The map of an exact bin table (-1: not counted) whose counted values form one contiguous
// range with bins non-decreasing in the value.  `scale` and `origin` are the FP64 slope and
// zero of the bin expression.  The fixed-point bin floor((d * slope + offset) / 2^32) is
// evaluated here for every counted value, with the offset raised in steps until all of them
// are right (values that fall on a bin's edge need it above the rounding of the slope); where
// no offset is, which takes an expression whose own FP64 rounding is uneven, the thresholds
// settle it, provided that the bin is within one.  Leaves T empty if they are not needed.
int make_bin_map(const std::vector<int32_t> &tab, int64_t bins, double scale, double origin,
                 std::vector<uint32_t> &T, BinMap &m, const char *what) {
    int lo = -1, hi = -1;
    for (int v = 0; v < 65536; v++)
        if (tab[v] >= 0) {
            if (lo < 0) lo = v;
            hi = v;
        }
    T.clear();
    m = BinMap{};
    m.bins = (int) bins;
    if (lo < 0) {  // nothing counted: a range no uint16 reaches
        m.lo = 65536 + 1;
        return MAXI_OK;
    }
    for (int v = lo; v <= hi; v++)
        if (tab[v] < 0 || (v > lo && tab[v] < tab[v - 1]))
            return set_error(MAXI_ERR_UNSUPPORTED, "%s bins are not monotone in the value", what);
    m.lo = lo;
    m.span = hi - lo;
    if (m.span == 0) {  // one counted value
        m.offset = (uint64_t) tab[lo] << 32;
        return MAXI_OK;
    }
    const double one = 4294967296.0;
    const uint64_t slope = (uint64_t) std::llround(scale * one);  // scale < 2^20: two values are counted
    m.mul_lo = (uint32_t) slope;
    m.mul_hi = (uint32_t) (slope >> 32);
    const double base = std::max(0.0, ((double) lo - origin) * scale);
    auto bin = [&](int v) {
        const uint64_t d = (uint64_t) (v - lo);
        return (int64_t) ((d * m.mul_lo + m.offset) >> 32) + (int64_t) (uint32_t) (d * m.mul_hi);
    };
    int64_t off_by = 0;
    for (int step = 0; step <= 20; step++) {
        m.offset = (uint64_t) std::floor(base * one) + (uint64_t(1) << step);
        off_by = 0;
        for (int v = lo; v <= hi && off_by <= 1; v++) off_by = std::max(off_by, std::abs(bin(v) - (int64_t) tab[v]));
        if (off_by == 0) return MAXI_OK;
    }
    if (off_by > 1) return set_error(MAXI_ERR_UNSUPPORTED, "%s bin estimate off by more than one", what);
    T.assign(bins + 1, 0);
    int64_t b = 0;
    for (int v = lo; v <= hi; v++)
        while (b <= tab[v]) T[b++] = (uint32_t) v;
    while (b <= bins) T[b++] = (uint32_t) hi + 1;
    return MAXI_OK;
}

// Bin of every uint16 value, -1 where the reference does not count it.  Voxels:
// values outside [lo, hi] count as 0 and zero voxels are skipped.  Field values:
// zero values and bins outside [0, bins) are skipped.
void value_table(std::vector<int32_t> &tab, bool voxel, double lo, double hi, int64_t bins) {
    tab.assign(65536, -1);
    for (int v = 1; v < 65536; v++) {
        const double vv = (double) v;
        if (voxel && !(vv >= lo && vv <= hi)) continue;
        const int64_t b = ref_bin(vv, lo, hi, bins);
        if (b >= 0 && b < bins) tab[v] = (int32_t) b;
    }
}

// The bin map of (kind, lo, hi, bins), built once and kept: the pipeline calls the
// histograms block by block with the same ranges.  A few recent maps are kept.
struct CachedMap {
    bool voxel;
    double lo, hi;
    int64_t bins;
    std::vector<uint32_t> T;
    BinMap m;
};

int cached_bin_map(bool voxel, double lo, double hi, int64_t bins, std::vector<uint32_t> &T, BinMap &m) {
    static std::mutex mu;
    static std::vector<CachedMap> cache;
    std::lock_guard<std::mutex> lock(mu);
    for (const CachedMap &c : cache)
        if (c.voxel == voxel && c.lo == lo && c.hi == hi && c.bins == bins) {
            T = c.T;
            m = c.m;
            return MAXI_OK;
        }
    std::vector<int32_t> tab;
    value_table(tab, voxel, lo, hi, bins);
    const int rc = make_bin_map(tab, bins, (double) (bins - 1) / (hi - lo), lo, T, m, voxel ? "voxel" : "field");
    if (rc) return rc;
    if (cache.size() >= 4) cache.erase(cache.begin());
    cache.push_back({voxel, lo, hi, bins, T, m});
    return MAXI_OK;
}

int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Device copy of host words laid out in 16-byte aligned segments.
struct DeviceTables {
    std::vector<uint32_t> host;
    uint32_t *dev = nullptr;
    size_t add(const uint32_t *p, size_t n) {
        const size_t at = host.size();
        host.insert(host.end(), p, p + n);
        host.resize((host.size() + 3) / 4 * 4, 0);
        return at;
    }
};

int upload(DeviceTables &t, cudaStream_t st) {
    const size_t bytes = t.host.size() * sizeof(uint32_t);
    if (bytes == 0) return MAXI_OK;
    if (cudaMallocAsync(reinterpret_cast<void **>(&t.dev), bytes, st) != cudaSuccess) {
        cudaGetLastError();
        t.dev = nullptr;
        return set_error(MAXI_ERR_OUT_OF_MEMORY, "could not allocate %zu bytes of tables", bytes);
    }
    cudaError_t e = cudaMemcpyAsync(t.dev, t.host.data(), bytes, cudaMemcpyHostToDevice, st);
    return e == cudaSuccess ? MAXI_OK : set_cuda_error(e, "histogram tables");
}

// Waits for the launch (the host tables must outlive their copy) and frees the device copy.
int finish(DeviceTables &t, cudaStream_t st, int rc, const char *what) {
    cudaError_t e = rc == MAXI_OK ? cudaGetLastError() : cudaSuccess;
    cudaError_t e2 = cudaStreamSynchronize(st);
    if (t.dev) cudaFreeAsync(t.dev, st);
    if (rc != MAXI_OK) return rc;
    if (e == cudaSuccess) e = e2;
    return e == cudaSuccess ? MAXI_OK : set_cuda_error(e, what);
}

// Shared counters of one block of the strip and ring forms (128 KB).
constexpr int kBlockCells = 32768;
constexpr int kMaxSharedBins = 8192;
// Voxels below which the direct form's single launch is the faster one.
constexpr int64_t kAxisMinVoxels = int64_t(1) << 17;

int axis_launches(const uint16_t *voxels, int64_t nzl, int64_t Ny, int Nx, int64_t z_start, int64_t y_start, int x_start,
                  const BinMap &vm, int64_t cy, int64_t cx, unsigned long long *xb, unsigned long long *yb,
                  unsigned long long *zb, unsigned long long *rb, int voxel_bins, int64_t n_r, bool vec,
                  int64_t farthest, cudaStream_t st) {
    const int64_t sms = sm_count(), rows = nzl * Ny;
    if (voxel_bins > kMaxSharedBins || rows * Nx < kAxisMinVoxels || farthest >= (1 << 15) || n_r >= (1 << 15)) {
        const unsigned grid = (unsigned) std::min<int64_t>(rows, sms * 16);
        auto direct = vec ? axis_histograms_direct<true> : axis_histograms_direct<false>;
        direct<<<grid, vec ? 128 : 256, 0, st>>>(voxels, nzl, Ny, Nx, z_start, y_start, x_start, vm, cy, cx, xb, yb, zb,
                                                 rb, voxel_bins, n_r);
        return MAXI_OK;
    }
    const bool exact = !vm.T;
    auto launch = [&](auto kernel, int64_t grid, int threads, int cells, auto... args) {
        const int smem = cells * (int) sizeof(uint32_t);
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return set_cuda_error(e, "axis histograms set-up");
        kernel<<<(unsigned) grid, threads, smem, st>>>(args...);
        return (int) MAXI_OK;
    };
    // z and y: several chunks per plane (or y) where there are few of them, of 16 rows at least.
    auto row_sets = [&](int64_t sets, int64_t first_set, int64_t set_step, int64_t row_step, int64_t row_count,
                        int64_t first_row, unsigned long long *bins) {
        const int64_t n = row_count - first_row, counted = sets - first_set;
        const int64_t chunks = std::max<int64_t>(1, std::min(ceil_div(sms * 8, counted), n / 16));
        const int64_t per = ceil_div(n, chunks);
        const RowSets s{sets, set_step, row_step, row_count, first_row, per, first_set, bins};
        return launch(vec ? (exact ? row_set_histograms<true, true> : row_set_histograms<true, false>)
                          : (exact ? row_set_histograms<false, true> : row_set_histograms<false, false>), counted * ceil_div(n, per), 256,
                      voxel_bins, voxels, Nx, x_start, vm, s, voxel_bins);
    };
    int rc = row_sets(nzl, 0, Ny, 1, Ny, y_start, zb + z_start * voxel_bins);
    if (rc == MAXI_OK) rc = row_sets(Ny, y_start, 1, Ny, nzl, 0, yb);
    if (rc) return rc;
    // x: strips of 8, or as many as the counters allow; chunks of at least 2048 rows.
    const int strip = std::min(kVec, kBlockCells / voxel_bins), strips = (int) ceil_div(Nx, strip);
    const int64_t x_chunks = std::max<int64_t>(1, std::min(ceil_div(sms * 4, strips), rows / 2048));
    const int64_t x_per = ceil_div(rows, x_chunks);
    const bool wide = vec && strip == kVec;
    rc = launch(wide ? (exact ? strip_histograms<true, true> : strip_histograms<true, false>)
                     : (exact ? strip_histograms<false, true> : strip_histograms<false, false>), strips * ceil_div(rows, x_per),
                1024, strip * voxel_bins, voxels, rows, Ny, Nx, y_start, x_start, vm, strips, strip, x_per, xb, voxel_bins);
    if (rc) return rc;
    // r: rings of as many radii as the counters allow; 16 planes per block.
    const int64_t radii = std::min<int64_t>(n_r, (int64_t) (1.4142136 * (double) farthest) + 2);
    const int width = (int) std::min<int64_t>(radii, std::max(1, kBlockCells / voxel_bins));
    const int rings = (int) ceil_div(radii, width);
    const int64_t per = std::min<int64_t>(nzl, 16);
    return launch(exact ? ring_histograms<true> : ring_histograms<false>, rings * ceil_div(nzl, per), 1024,
                  width * voxel_bins, voxels, nzl, (int) Ny, Nx, (int) y_start, x_start, vm, (int) cy, (int) cx, rings,
                  width, per, rb, voxel_bins, (int) n_r);
}

}  // namespace
}  // namespace maxi

using namespace maxi;

extern "C" int maxi_field_histogram(const uint16_t *voxels, int64_t nZ, int64_t nY, int64_t nX, const uint16_t *field,
                                    int64_t nz, int64_t ny, int64_t nx, int64_t y_start, int64_t x_start,
                                    uint64_t *bins, int64_t field_bins, int64_t voxel_bins, double vmin, double vmax,
                                    double fmin, double fmax, void *stream) {
    clear_error();
    if (!voxels || !field || !bins) return set_error(MAXI_ERR_INVALID_ARGUMENT, "NULL pointer");
    if (nZ <= 0 || nY <= 0 || nX <= 0 || nz <= 0 || ny <= 0 || nx <= 0)
        return set_error(MAXI_ERR_INVALID_ARGUMENT, "empty voxel or field volume");
    if (field_bins <= 0 || voxel_bins <= 0 || field_bins > (1 << 20) || voxel_bins > (1 << 20))
        return set_error(MAXI_ERR_INVALID_ARGUMENT, "bad histogram size %lld x %lld", (long long) field_bins,
                         (long long) voxel_bins);
    if (!(vmax > vmin) || !(fmax > fmin)) return set_error(MAXI_ERR_INVALID_ARGUMENT, "empty value range");
    if (y_start < 0 || x_start < 0) return set_error(MAXI_ERR_INVALID_ARGUMENT, "negative offset");
    if (nX >= (int64_t(1) << 30) || nx >= (int64_t(1) << 31))
        return set_error(MAXI_ERR_UNSUPPORTED, "rows of 2^30 voxels or more are not served");
    if (x_start >= nX || y_start >= nY) return MAXI_OK;  // nothing to count
    int rc = require_device();
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    std::vector<uint32_t> vT, fT;
    BinMap vm{}, fm{};
    if ((rc = cached_bin_map(true, vmin, vmax, voxel_bins, vT, vm))) return rc;
    if ((rc = cached_bin_map(false, fmin, fmax, field_bins, fT, fm))) return rc;
    std::vector<uint32_t> zmap(nZ), ymap(nY), xmap(nX);
    const double dz = (double) nz / (double) nZ, dy = (double) ny / (double) nY, dx = (double) nx / (double) nX;
    for (int64_t Z = 0; Z < nZ; Z++) {
        volatile double t = (double) Z * dz;
        zmap[Z] = (uint32_t) std::min<int64_t>(nz - 1, (int64_t) std::floor((double) t));
    }
    for (int64_t Y = 0; Y < nY; Y++) {
        volatile double t = (double) Y * dy;
        ymap[Y] = (uint32_t) std::min<int64_t>(ny - 1, (int64_t) std::floor((double) t));
    }
    for (int64_t X = 0; X < nX; X++) {
        volatile double t = (double) X * dx;
        xmap[X] = (uint32_t) std::min<int64_t>(nx - 1, (int64_t) std::floor((double) t));
    }
    DeviceTables t;
    const size_t o_vT = t.add(vT.data(), vT.size()), o_fT = t.add(fT.data(), fT.size());
    const size_t o_z = t.add(zmap.data(), zmap.size()), o_y = t.add(ymap.data(), ymap.size());
    const size_t o_x = t.add(xmap.data(), xmap.size());
    rc = upload(t, st);
    if (rc == MAXI_OK) {
        if (!vT.empty()) vm.T = t.dev + o_vT;
        if (!fT.empty()) fm.T = t.dev + o_fT;
        const int32_t *zm = reinterpret_cast<const int32_t *>(t.dev + o_z);
        const int32_t *ym = reinterpret_cast<const int32_t *>(t.dev + o_y);
        const int32_t *xm = reinterpret_cast<const int32_t *>(t.dev + o_x);
        auto *b = reinterpret_cast<unsigned long long *>(bins);
        const bool vec = nX % kVec == 0 && reinterpret_cast<uintptr_t>(voxels) % 16 == 0;
        const unsigned grid = (unsigned) std::min<int64_t>(nZ * nY, (int64_t) sm_count() * 16);
        if (vec)
            field_histogram_kernel<true><<<grid, 128, 0, st>>>(voxels, field, nZ, nY, (int) nX, ny, nx, y_start,
                                                               (int) x_start, vm, fm, zm, ym, xm, b, voxel_bins);
        else
            field_histogram_kernel<false><<<grid, 256, 0, st>>>(voxels, field, nZ, nY, (int) nX, ny, nx, y_start,
                                                                (int) x_start, vm, fm, zm, ym, xm, b, voxel_bins);
    }
    return finish(t, st, rc, "field histogram");
}

extern "C" int maxi_axis_histograms(const uint16_t *voxels, int64_t nz_block, int64_t Nz, int64_t Ny, int64_t Nx,
                                    int64_t z_start, int64_t y_start, int64_t x_start, uint64_t *x_bins,
                                    uint64_t *y_bins, uint64_t *z_bins, uint64_t *r_bins, int64_t voxel_bins,
                                    int64_t n_r, int64_t cy, int64_t cx, double vmin, double vmax, void *stream) {
    clear_error();
    if (!voxels || !x_bins || !y_bins || !z_bins || !r_bins) return set_error(MAXI_ERR_INVALID_ARGUMENT, "NULL pointer");
    if (nz_block <= 0 || Nz <= 0 || Ny <= 0 || Nx <= 0) return set_error(MAXI_ERR_INVALID_ARGUMENT, "empty volume");
    if (voxel_bins <= 0 || voxel_bins > (1 << 20) || n_r <= 0)
        return set_error(MAXI_ERR_INVALID_ARGUMENT, "bad histogram size");
    if (!(vmax > vmin)) return set_error(MAXI_ERR_INVALID_ARGUMENT, "empty value range");
    if (z_start < 0 || y_start < 0 || x_start < 0 || cy < 0 || cx < 0)
        return set_error(MAXI_ERR_INVALID_ARGUMENT, "negative offset or centre");
    if (Nx >= (int64_t(1) << 30)) return set_error(MAXI_ERR_UNSUPPORTED, "rows of 2^30 voxels or more are not served");
    // Largest distance from the centre; the integer square root equals the reference's double one below 2^50.
    const int64_t ry = std::max(cy, Ny - 1 - cy), rx = std::max(cx, Nx - 1 - cx);
    if (ry >= (int64_t(1) << 24) || rx >= (int64_t(1) << 24))
        return set_error(MAXI_ERR_UNSUPPORTED, "distances of 2^24 voxels or more from the centre are not served");
    const int64_t nzl = std::min(z_start + nz_block, Nz) - z_start;
    if (nzl <= 0 || y_start >= Ny || x_start >= Nx) return MAXI_OK;  // nothing to count
    int rc = require_device();
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    std::vector<uint32_t> vT;
    BinMap vm{};
    if ((rc = cached_bin_map(true, vmin, vmax, voxel_bins, vT, vm))) return rc;
    DeviceTables t;
    const size_t o_vT = t.add(vT.data(), vT.size());
    rc = upload(t, st);
    if (rc == MAXI_OK) {
        if (!vT.empty()) vm.T = t.dev + o_vT;
        auto *xb = reinterpret_cast<unsigned long long *>(x_bins), *yb = reinterpret_cast<unsigned long long *>(y_bins);
        auto *zb = reinterpret_cast<unsigned long long *>(z_bins), *rb = reinterpret_cast<unsigned long long *>(r_bins);
        const bool vec = Nx % kVec == 0 && reinterpret_cast<uintptr_t>(voxels) % 16 == 0;
        rc = axis_launches(voxels, nzl, Ny, (int) Nx, z_start, y_start, (int) x_start, vm, cy, cx, xb, yb, zb, rb,
                           (int) voxel_bins, n_r, vec, std::max(rx, ry), st);
    }
    return finish(t, st, rc, "axis histograms");
}
