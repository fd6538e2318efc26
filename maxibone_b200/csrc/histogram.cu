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
// Counting, field_histogram.  Large volumes: sorted by parts of the histogram, which are then
// counted in shared memory (below).  The others, and bins too many for that: one thread takes 8
// consecutive voxels of a row (one 16-byte load when rows are 16-byte aligned), adds runs of
// equal keys once and issues one 64-bit reduction per run into the histogram (L2-resident at
// the pipeline's 2048 x 4096); each block walks one contiguous range of rows.
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
#include <atomic>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "host_util.h"
#include "launch.cuh"
#include "scratch.h"

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

// The same for a value within the range; anything outside it.
template <bool EXACT = false>
__device__ __forceinline__ int bin_in_range(const BinMap &m, int v) {
    if (!EXACT) return bin_of(m, v);
    const uint32_t d = (uint32_t) (v - m.lo);
    return (int) (((uint64_t) d * m.mul_lo + m.offset) >> 32) + (int) (d * m.mul_hi);
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

// ---- field_histogram through partitioned keys ----------------------------------------
//
// The reductions of field_histogram_kernel hit random 64-bit cells of a histogram far larger
// than any shared memory, 95 to 148 G a second whatever the launch (L2's rate), while shared
// memory adds 2300 G a second.  So the cells are split into partitions of `group` field bins
// that fit one SM's shared memory, and the voxels' cells are sorted by partition on the way:
// partition_keys takes tiles of 16384 voxels, ranks each tile's 16-bit keys (the cell within
// its partition) by partition with counters in shared memory, lines them up there and writes
// them out in one run; count_partitions reads them back, partition after partition.  That moves
// the voxels once and 2 bytes a voxel each way (158 partitions of a tile: about 70 keys in a
// row).  54 instructions a voxel fill 59% of the issue slots: at 64 registers a scheduler has 7.5 warps,
// which wait for the field's values, at the tile's barriers and in fixed latencies alike.  A
// branch around tiles of air made the others slower (1.90 -> 1.97 ms: it ends the overlap of
// one vector's loads with another's counting).
// 512 x 1024 x 1024 against half resolution, 2048 x 4096 bins: 2.85 -> 1.90 ms (partition_keys
// 1.36, count_partitions 0.50).
constexpr int kKeyThreads = 512;
constexpr int kKeyVecs = 4;                                // 8-voxel vectors per thread and tile
constexpr int kTileVecs = kKeyThreads * kKeyVecs;
constexpr int kTileKeys = kTileVecs * kVec;                // 16384
constexpr int kMaxParts = 256;
constexpr int kPartCells = 53248;                          // 208 KB of 32-bit counters
constexpr int kGroupTiles = 4096;                          // whose runs a block lines up at a time
constexpr int kMaxGroup = 4096;                            // fb / group below is exact up to here

// n / d by a multiplication: exact for n * d < 2^32.
struct SmallDiv {
    uint32_t d, magic, one;
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const { return __umulhi(n, magic) + n * one; }
};

struct PartitionArgs {
    const uint16_t *voxels, *field;
    int64_t ny, nx;                     // the field's rows
    int nX, x_start;
    uint32_t nY, y_start, first_row, rows;  // this batch's rows of the volume
    SmallDiv per_row, group;            // vectors per row, field bins per partition
    BinMap vm, fm;
    const int32_t *zmap, *ymap, *xmap;  // xmap: padded to whole vectors
    int voxel_bins, field_bins, parts, tiles;
    int pitch;                          // of starts: the tiles of a full batch, a multiple of 4
    uint16_t *keys;                     // [tiles][kTileKeys], each tile's keys by partition
    uint16_t *starts;                   // [parts + 1][pitch]: where a partition starts in a tile
    uint32_t *totals;                   // [parts]: keys of a partition, all tiles
    unsigned long long *bins;
};

// VEC8: rows of whole aligned vectors.
template <bool VEC8, bool EXACT>
__global__ void __launch_bounds__(kKeyThreads, 2) partition_keys(const PartitionArgs a) {
    __shared__ __align__(16) uint16_t sorted[kTileKeys];
    __shared__ uint32_t counts[kMaxParts], place[kMaxParts], sums[kMaxParts / 32];
    constexpr uint32_t none = ~0u;  // part << 16 | rank of a voxel that is not counted
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < kMaxParts) counts[tid] = 0;
    // VEC8: the batch's vectors lie one after another.
    const uint4 *first = reinterpret_cast<const uint4 *>(a.voxels + (int64_t) a.first_row * a.nX);
    const uint32_t vecs = a.rows * a.per_row.d;
    uint32_t total = 0;  // of partition tid, over this block's tiles
    __syncthreads();
    for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
        // Every load of the tile's voxels first, then the field's rows and values.
        uint32_t key[kKeyVecs][kVec / 2], rank[kKeyVecs][kVec];  // two keys a word; part << 16 | rank
        uint4 w[kKeyVecs];
        int zi[kKeyVecs], yi[kKeyVecs], X[kKeyVecs];
        const uint32_t vec0 = (uint32_t) tile * kTileVecs;
#pragma unroll
        for (int k = 0; k < kKeyVecs; k++) {
            const uint32_t vec = vec0 + tid + kKeyThreads * k;
            w[k] = make_uint4(0, 0, 0, 0);  // zero voxels are not counted
            if (VEC8 && vec < vecs) w[k] = __ldcs(first + vec);
        }
        const uint32_t row0 = vec0 / a.per_row.d, col0 = vec0 - row0 * a.per_row.d;
        const uint32_t Z0 = (a.first_row + row0) / a.nY, Y0 = a.first_row + row0 - Z0 * a.nY;
#pragma unroll
        for (int k = 0; k < kKeyVecs; k++) {
            const uint32_t o = col0 + tid + kKeyThreads * k, r = a.per_row(o);
            X[k] = (int) (o - r * a.per_row.d) * kVec;
            uint32_t Z = Z0, Y = Y0 + r;
            if (Y >= a.nY) Z += Y / a.nY, Y %= a.nY;
            const bool live = row0 + r < a.rows && Y >= a.y_start;
            zi[k] = live ? __ldg(a.zmap + Z) : 0;
            yi[k] = live ? __ldg(a.ymap + Y) : 0;
            if (!VEC8 && live) {
                const uint16_t *vrow = a.voxels + ((int64_t) a.first_row + row0 + r) * a.nX + X[k];
                uint32_t u[kVec];
#pragma unroll
                for (int j = 0; j < kVec; j++) u[j] = X[k] + j < a.nX ? __ldcs(vrow + j) : 0;
                w[k] = make_uint4(u[0] | u[1] << 16, u[2] | u[3] << 16, u[4] | u[5] << 16, u[6] | u[7] << 16);
            }
            if (!live || X[k] < a.x_start) {  // voxels before the offset: zero
                uint32_t u[4] = {w[k].x, w[k].y, w[k].z, w[k].w};
                const int skip = live ? a.x_start - X[k] : kVec;
#pragma unroll
                for (int j = 0; j < kVec; j++)
                    if (j < skip) u[j / 2] &= j & 1 ? 0x0000ffffu : 0xffff0000u;
                w[k] = make_uint4(u[0], u[1], u[2], u[3]);
            }
        }
#pragma unroll
        for (int k = 0; k < kKeyVecs; k++) {
            const int4 m0 = __ldg(reinterpret_cast<const int4 *>(a.xmap + X[k])),
                       m1 = __ldg(reinterpret_cast<const int4 *>(a.xmap + X[k]) + 1);
            const int at[kVec] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
            const uint32_t u[4] = {w[k].x, w[k].y, w[k].z, w[k].w};
            const uint16_t *frow = a.field + ((int64_t) zi[k] * a.ny + yi[k]) * a.nx;
            // G voxels to a field value: two where every pair of the warp's voxels reads one
            // (a field at half resolution or less), whose bin and addition they then share.
            auto rank_vector = [&](auto voxels_per_value) {
                constexpr int G = decltype(voxels_per_value)::value;
                uint32_t part[kVec / G], base[kVec / G], below[kVec / G], differ = 0;
                int f[kVec / G];
#pragma unroll
                for (int i = 0; i < kVec / G; i++) f[i] = (int) __ldg(frow + at[G * i]);
#pragma unroll
                for (int i = 0; i < kVec / G; i++) {
                    const int fb = bin_of<EXACT>(a.fm, f[i]);
                    part[i] = fb >= 0 ? a.group((uint32_t) fb) : (uint32_t) kMaxParts;
                    base[i] = ((uint32_t) fb - part[i] * a.group.d) * (uint32_t) a.voxel_bins;
                    below[i] = fb >= 0 ? (uint32_t) a.vm.span + 1 : 0;
                    differ |= part[i] ^ part[0];
                }
                bool counted[kVec];
#pragma unroll
                for (int j = 0; j < kVec; j += 2) {
                    uint32_t q[2];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int v = (int) (h ? u[j / 2] >> 16 : u[j / 2] & 0xffffu);
                        q[h] = base[(j + h) / G] + (uint32_t) bin_in_range<EXACT>(a.vm, v);
                        counted[j + h] = (uint32_t) (v - a.vm.lo) < below[(j + h) / G];
                    }
                    key[k][j / 2] = __byte_perm(q[0], q[1], 0x5410);
                }
                // A warp whose 256 voxels all belong to one partition (a plateau's, or a smooth
                // field's) ranks its own voxels and adds once; additions of many lanes to one
                // counter would be taken one at a time.
                const uint32_t p0 = __shfl_sync(0xffffffffu, part[0], 0);
                if (__all_sync(0xffffffffu, (differ | (part[0] ^ p0)) == 0)) {
                    uint32_t n = 0, m[kVec];
#pragma unroll
                    for (int j = 0; j < kVec; j++) {
                        m[j] = __ballot_sync(0xffffffffu, counted[j]);
                        n += __popc(m[j]);
                    }
                    uint32_t from = 0;
                    if (lane == 0 && n) from = atomicAdd(&counts[p0], n);
                    from = (p0 << 16) + __shfl_sync(0xffffffffu, from, 0);
#pragma unroll
                    for (int j = 0; j < kVec; j++) {
                        rank[k][j] = counted[j] ? from + __popc(m[j] & ((1u << lane) - 1)) : none;
                        from += __popc(m[j]);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < kVec / G; i++) {
                        uint32_t n = 0;
#pragma unroll
                        for (int h = 0; h < G; h++) n += counted[G * i + h];
                        uint32_t r = part[i] << 16;
                        if (n) r += atomicAdd(&counts[part[i]], n);
#pragma unroll
                        for (int h = 0; h < G; h++) {
                            rank[k][G * i + h] = counted[G * i + h] ? r : none;
                            r += counted[G * i + h];
                        }
                    }
                }
            };
            if (__all_sync(0xffffffffu, at[0] == at[1] && at[2] == at[3] && at[4] == at[5] && at[6] == at[7]))
                rank_vector(std::integral_constant<int, 2>{});
            else
                rank_vector(std::integral_constant<int, 1>{});
        }
        __syncthreads();
        // Partition starts: exclusive sums over the counts.
        uint32_t count = 0, sum = 0;
        if (warp < kMaxParts / 32) {
            count = counts[tid];
            counts[tid] = 0;
            sum = count;
#pragma unroll
            for (int d = 1; d < 32; d *= 2) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += y;
            }
            if (lane == 31) sums[warp] = sum;
            total += count;
        }
        __syncthreads();
        uint32_t all = 0, before = 0;
#pragma unroll
        for (int i = 0; i < kMaxParts / 32; i++) {
            if (i < warp) before += sums[i];
            all += sums[i];
        }
        if (tid < a.parts) {
            place[tid] = before + sum - count;
            a.starts[(int64_t) tid * a.pitch + tile] = (uint16_t) (before + sum - count);
        }
        if (tid == 0) a.starts[(int64_t) a.parts * a.pitch + tile] = (uint16_t) all;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kKeyVecs; k++)
#pragma unroll
            for (int j = 0; j < kVec; j++)
                if (rank[k][j] != none)
                    sorted[place[rank[k][j] >> 16] + (rank[k][j] & 0xffffu)] =
                        (uint16_t) (j & 1 ? key[k][j / 2] >> 16 : key[k][j / 2]);
        __syncthreads();
        // (The next tile's counts and sums change what this tile read before the barrier above;
        // its keys go out before the next tile's scatter, two barriers on.)
        uint4 *out = reinterpret_cast<uint4 *>(a.keys + (int64_t) tile * kTileKeys);
        for (uint32_t i = tid; i * 8 < all; i += kKeyThreads) out[i] = reinterpret_cast<const uint4 *>(sorted)[i];
    }
    if (tid < a.parts && total) atomicAdd(a.totals + tid, total);
}

// Inclusive sum over the block's 1024 threads.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += y;
    }
    __syncthreads();
    if (lane == 31) sums[warp] = v;
    __syncthreads();
    uint32_t s = sums[lane];
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, s, d);
        if (lane >= d) s += y;
    }
    const uint32_t before = __shfl_sync(0xffffffffu, s, (warp + 31) & 31);
    return warp ? v + before : v;
}

// Counts the keys.  The (partition, tile) runs in order are split into one range of about equal
// cost per block, cut between tiles, so that a partition that holds most keys (a field's
// plateau) is shared by many blocks, and each block adds its counters to the bins once per
// partition it meets.  Costs in keys: a run's look-up and partly filled loads, and a partition's
// counters.
constexpr uint32_t kRunCost = 16, kPartCost = 8192;

__global__ void __launch_bounds__(1024) count_partitions(const PartitionArgs a) {
    extern __shared__ uint32_t counters[];
    __shared__ uint32_t upto[kMaxParts + 1], sums[32], cut[2];
    __shared__ __align__(16) uint32_t chunks[kGroupTiles];
    const int tid = threadIdx.x, lane = tid & 31;
    for (int i = tid; i < kPartCells; i += 1024) counters[i] = 0;
    {
        const uint32_t keys = tid < a.parts ? __ldg(a.totals + tid) : 0;
        const uint32_t s = block_sum(keys ? keys + kPartCost + kRunCost * a.tiles : 0, sums);
        if (tid < a.parts) upto[tid + 1] = s;
        if (tid == 0) upto[0] = 0;
    }
    __syncthreads();
    const uint32_t n = upto[a.parts];
    // The first run with a cost of `target` or more before it: partition part, tile cut[which]
    // (up to `tiles`: the partition's end).
    const int per = (a.tiles + 1023) / 1024;
    auto find = [&](uint32_t target, int which, int &part) {
        part = 0;
        if (target > 0) part = __syncthreads_count(tid < a.parts && upto[tid + 1] < target);
        const uint32_t into = target - upto[part], rest = into > kPartCost ? into - kPartCost : 0;
        const uint16_t *lo = a.starts + (int64_t) part * a.pitch, *hi = lo + a.pitch;
        const int t0 = min(a.tiles, tid * per), t1 = min(a.tiles, t0 + per);
        auto cost = [&](int t) { return (uint32_t) __ldg(hi + t) - __ldg(lo + t) + kRunCost; };
        uint32_t mine = 0;
        for (int t = t0; t < t1; t++) mine += cost(t);
        const uint32_t s = block_sum(mine, sums);
        if (rest == 0) {
            if (tid == 0) cut[which] = 0;
        } else if (s >= rest && s - mine < rest) {
            uint32_t c = s - mine;
            int t = t0;
            while (c < rest) c += cost(t++);
            cut[which] = t;
        }
        __syncthreads();
    };
    if (n == 0) return;
    int p0, p1;
    find((uint32_t) ((uint64_t) n * blockIdx.x / gridDim.x), 0, p0);
    find((uint32_t) ((uint64_t) n * (blockIdx.x + 1) / gridDim.x), 1, p1);
    for (int p = p0; p <= p1; p++) {
        const int tb = p == p0 ? (int) cut[0] : 0, te = p == p1 ? (int) cut[1] : a.tiles;
        if (tb >= te || upto[p] == upto[p + 1]) continue;  // the same for every thread
        const uint16_t *starts = a.starts + (int64_t) p * a.pitch;
        for (int t0 = tb & ~3; t0 < te; t0 += kGroupTiles) {
            // The next 4096 tiles' runs in chunks of 32 keys (a load of 8 lanes); a warp takes 32
            // chunks in order at a time.
            const int t = t0 + 4 * tid;
            uint32_t mine[4], sum = 0;
            const bool any = t < te;
            const ushort4 l4 = any ? __ldg(reinterpret_cast<const ushort4 *>(starts + t)) : ushort4{},
                          h4 = any ? __ldg(reinterpret_cast<const ushort4 *>(starts + a.pitch + t)) : ushort4{};
            const uint32_t lo[4] = {l4.x, l4.y, l4.z, l4.w}, hi[4] = {h4.x, h4.y, h4.z, h4.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                mine[i] = t + i >= tb && t + i < te && hi[i] > lo[i] ? (hi[i] - (lo[i] & ~3u) + 31) / 32 : 0;
                sum += mine[i];
            }
            uint32_t upper = block_sum(sum, sums) - sum;
            uint4 c4;
            c4.x = upper += mine[0];
            c4.y = upper += mine[1];
            c4.z = upper += mine[2];
            c4.w = upper += mine[3];
            reinterpret_cast<uint4 *>(chunks)[tid] = c4;
            __syncthreads();
            const uint32_t all = chunks[kGroupTiles - 1];
            for (uint32_t c0 = (uint32_t) tid & ~31u; c0 < all; c0 += 1024) {
                // Lane q looks up chunk c0 + q: the first tile whose sum is above it.
                const uint32_t c = c0 + lane;
                int at = 0;
#pragma unroll
                for (int d = kGroupTiles / 2; d > 0; d /= 2)
                    if (chunks[at + d - 1] <= c) at += d;
                uint32_t e = 0, base = 0;
                if (c < all) {
                    e = (uint32_t) __ldg(starts + t0 + at) | (uint32_t) __ldg(starts + a.pitch + t0 + at) << 16;
                    base = ((e & 0xffffu) & ~3u) + (c - (at ? chunks[at - 1] : 0)) * 32;
                }
                uint2 w[8];
                uint32_t i[8], run[8];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int src = 4 * q + lane / 8;
                    const int tq = t0 + __shfl_sync(0xffffffffu, at, src);
                    run[q] = __shfl_sync(0xffffffffu, e, src);
                    i[q] = __shfl_sync(0xffffffffu, base, src) + 4 * (lane & 7);
                    if (i[q] < run[q] >> 16)
                        w[q] = __ldcs(reinterpret_cast<const uint2 *>(a.keys + (int64_t) tq * kTileKeys + i[q]));
                }
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const uint32_t from = run[q] & 0xffffu, to = run[q] >> 16;
                    if (i[q] >= from && i[q] < to) atomicAdd(counters + (w[q].x & 0xffffu), 1u);
                    if (i[q] + 1 >= from && i[q] + 1 < to) atomicAdd(counters + (w[q].x >> 16), 1u);
                    if (i[q] + 2 >= from && i[q] + 2 < to) atomicAdd(counters + (w[q].y & 0xffffu), 1u);
                    if (i[q] + 3 >= from && i[q] + 3 < to) atomicAdd(counters + (w[q].y >> 16), 1u);
                }
            }
            __syncthreads();
        }
        __syncthreads();
        const int64_t first = (int64_t) p * a.group.d;
        const int cells = (int) min((int64_t) a.group.d, a.field_bins - first) * a.voxel_bins;
        unsigned long long *bins = a.bins + first * a.voxel_bins;
        for (int i = tid; i < cells; i += 1024)
            if (const uint32_t c = counters[i]) {
                atomicAdd(bins + i, (unsigned long long) c);
                counters[i] = 0;
            }
        __syncthreads();
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
// global bins, runs of equal keys once (x: every voxel).  RADIAL: the radial histogram alone, for
// distances beyond ring_histograms.
template <bool VEC8, bool RADIAL>
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
                    if (!RADIAL) atomicAdd(x_bins + (int64_t) x * voxel_bins + vb, 1ull);
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
                if (RADIAL) continue;
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
// Whether a block of voxels holds any that is counted: the z histogram, which comes first and counts
// every voxel that the others do, then writes `call` to the word (NULL: not kept), and otherwise the
// other kernels have nothing to do.  The word needs no clearing, as `call` differs from call to call
// (an old value that happened to equal it would cost those kernels' time).  A block of air,
// 128 x 1024 x 1024 at 4096 bins: 515 us with four kernels that read it, 109 now.
struct Counted {
    uint32_t *word;
    uint32_t call;
    __device__ __forceinline__ bool none() const { return word && *word != call; }
};
__device__ __forceinline__ void counters_flush(const uint32_t *c, int n, unsigned long long *bins,
                                               Counted counted = Counted{}) {
    __syncthreads();
    bool any = false;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (const uint32_t k = c[i]) {
            atomicAdd(bins + i, (unsigned long long) k);
            any = true;
        }
    if (counted.word && any) *counted.word = counted.call;
}

// y_bins or z_bins: block (p, chunk) counts the rows row0(p), row0(p) + row_step, .. of one y
// (or z), from row chunk * per on, in one shared histogram.  A warp per row; SPLIT: several of them
// per row, where the chunk has fewer rows than the block has warps.
struct RowSets {
    int64_t sets, set_step, row_step, rows, first_row, per;  // per: rows of a chunk
    int64_t first_set;                                      // sets below are not counted
    unsigned long long *bins;                               // of set 0
    Counted mark, counted;                                  // z: written; y: read
};
template <bool VEC8, bool EXACT, bool SPLIT>
__global__ void __launch_bounds__(256) row_set_histograms(const uint16_t *__restrict__ voxels, int Nx, int x_start,
                                                          BinMap vm, RowSets s, int voxel_bins) {
    extern __shared__ uint32_t counters[];
    if (s.counted.none()) return;
    const int64_t set = s.first_set + blockIdx.x % (s.sets - s.first_set), chunk = blockIdx.x / (s.sets - s.first_set);
    const int64_t end = min(s.rows, s.first_row + (chunk + 1) * s.per);
    const int lane = threadIdx.x & 31;
    counters_clear(counters, voxel_bins);
    auto count = [&](int v) {
        const int b = bin_of<EXACT>(vm, v);
        if (b >= 0) atomicAdd(counters + b, 1u);
    };
    const int64_t begin = s.first_row + chunk * s.per;
    int split = 0;  // 2^split warps to a row
    while (SPLIT && split < 3 && (end - begin) << (split + 1) <= 8) split++;
    const int warp = threadIdx.x >> 5, share = SPLIT ? warp & ((1 << split) - 1) : 0, shares = 1 << split;
    for (int64_t i = begin + (warp >> split); i < end; i += 8 >> split) {
        const uint16_t *row = voxels + (set * s.set_step + i * s.row_step) * Nx;
        if (VEC8) {
            // Up to x_first one voxel per lane, then two loads of 8 ahead of their counting.
            const int x_first = (x_start + kVec - 1) / kVec * kVec;
            if (share == 0 && x_start + lane < x_first) count(__ldcs(row + x_start + lane));
            for (int x = x_first + (lane + 32 * share) * kVec; x < Nx; x += 64 * shares * kVec) {
                int v[kVec], w[kVec];
                const bool second = x + 32 * shares * kVec < Nx;
                load_row8(row + x, v);
                if (second) load_row8(row + x + 32 * shares * kVec, w);
#pragma unroll
                for (int j = 0; j < kVec; j++) count(v[j]);
                if (second)
#pragma unroll
                    for (int j = 0; j < kVec; j++) count(w[j]);
            }
        } else {
            for (int x = x_start + lane + 32 * kVec * share; x < Nx; x += 32 * kVec * shares) {
                int v[kVec];
#pragma unroll
                for (int j = 0; j < kVec; j++) v[j] = x + 32 * j < Nx ? __ldcs(row + x + 32 * j) : -1;
#pragma unroll
                for (int j = 0; j < kVec; j++)
                    if (v[j] >= 0) count(v[j]);
            }
        }
    }
    counters_flush(counters, voxel_bins, s.bins + set * voxel_bins, s.mark);
}

// x_bins: block (strip, chunk) counts `strip` neighbouring x over the rows of the chunk, a
// row per thread, two rows loaded ahead of their counting.
template <bool VEC8, bool EXACT>
__global__ void __launch_bounds__(1024) strip_histograms(const uint16_t *__restrict__ voxels, int64_t rows, int64_t Ny,
                                                         int Nx, int64_t y_start, int x_start, BinMap vm, int strips,
                                                         int strip, int64_t per, unsigned long long *__restrict__ x_bins,
                                                         int voxel_bins, Counted counted) {
    extern __shared__ uint32_t counters[];
    if (counted.none()) return;
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

// r_bins: block (ring, chunk, part) counts the pixels with ring * width <= r < (ring + 1) * width
// over the planes of the chunk and, `parts` to a ring, every so many of its rows.  Eight lanes take
// a row: its pixels of the ring are at most two x intervals (of about `width` each for most
// rows, hence eight), a lane per pixel, which reads that pixel of every plane, eight ahead of
// their counting.  SPLIT: where the ring's rows do not fill the block, eights of planes and then
// more lanes go to a row, and of one or two planes a lane loads four pixels ahead.  Rows that the
// ring meets only outside the volume are left out (a 2 x 40000 x 1000 block, 4096 bins: a ring's
// blocks would walk 40000 rows for about 40; the call 790 us with both, 2450 without).  The outer,
// larger rings start first.  Squared distances stay below 2^31 (the host checks).
template <bool EXACT, bool SPLIT>
__global__ void __launch_bounds__(1024) ring_histograms(const uint16_t *__restrict__ voxels, int64_t nzl, int Ny,
                                                        int Nx, int y_start, int x_start, BinMap vm, int cy, int cx,
                                                        int rings, int width, int64_t per, int chunks,
                                                        int parts,
                                                        unsigned long long *__restrict__ r_bins, int voxel_bins,
                                                        int n_r, Counted counted) {
    extern __shared__ uint32_t counters[];
    if (counted.none()) return;
    const int b = (int) blockIdx.x, part = b % parts, chunk = b / parts % chunks, ring = rings - 1 - b / parts / chunks;
    const int64_t z0 = chunk * per;
    const int planes = (int) min(per, nzl - z0);
    const int r0 = ring * width, r1 = min(r0 + width, n_r);
    counters_clear(counters, (r1 - r0) * voxel_bins);
    const int64_t plane = (int64_t) Ny * Nx;
    const int inner = r0 * r0, outer = r1 * r1 - 1;  // squared distances inner .. outer
    // The rows' distances low .. reach from the centre: those at which the ring meets a column.
    const int64_t widest = max(abs(x_start - cx), abs(Nx - 1 - cx)), nearest = max(0, max(x_start - cx, cx - (Nx - 1)));
    const int low = inner > widest * widest ? isqrt32((int) (inner - widest * widest) - 1) + 1 : 0;
    const int reach = outer >= nearest * nearest ? isqrt32((int) (outer - nearest * nearest)) : -1;
    const int above = max(y_start, cy - reach), n_above = max(0, min(Ny - 1, cy - max(low, 1)) - above + 1);
    const int below = max(y_start, cy + low), n_rows = n_above + max(0, min(Ny - 1, cy + reach) - below + 1);
    // 2^lane_bits lanes to a row and an eighth of planes, 2^z_bits of these to a row.
    const int rows = (n_rows + parts - 1) / parts;
    int lane_bits = 3, z_bits = 0;
    while (SPLIT && (8 << z_bits) < planes && rows << (lane_bits + z_bits + 1) <= 1024) z_bits++;
    while (SPLIT && lane_bits < 8 && rows << (lane_bits + z_bits + 1) <= 1024) lane_bits++;
    const int lane = threadIdx.x & ((1 << lane_bits) - 1), lanes = 1 << lane_bits;
    const int z_first = SPLIT ? 8 * ((threadIdx.x >> lane_bits) & ((1 << z_bits) - 1)) : 0, z_step = 8 << z_bits;
    const int slot = threadIdx.x >> (lane_bits + z_bits), step = 1024 >> (lane_bits + z_bits);
    auto count = [&](uint32_t *c, int v) {
        const int b = bin_of<EXACT>(vm, v);
        if (b >= 0 && v >= 0) atomicAdd(c + b, 1u);
    };
    for (int i = part * step + slot; i < n_rows; i += parts * step) {
        const int y = i < n_above ? above + i : below + (i - n_above);
        const int dy2 = (y - cy) * (y - cy);
        const int far = isqrt32(outer - dy2), near = dy2 >= inner ? 0 : isqrt32(inner - dy2 - 1) + 1;
        // right: cx + near .. cx + far; left: cx - far .. cx - max(near, 1)
        const int right = max(cx + near, x_start), n_right = max(0, min(cx + far, Nx - 1) - right + 1);
        const int left = max(cx - far, x_start), n_left = max(0, min(cx - max(near, 1), Nx - 1) - left + 1);
        const uint16_t *row = voxels + z0 * plane + (int64_t) y * Nx;
        const int n = n_right + n_left;
        auto x_of = [&](int k) { return k < n_right ? right + k : left + (k - n_right); };
        auto counters_of = [&](int x) { return counters + (isqrt32(dy2 + (x - cx) * (x - cx)) - r0) * voxel_bins; };
        if (SPLIT && planes <= 2) {
            for (int z = 0; z < planes; z++, row += plane) {
                for (int k = lane; k < n; k += 4 * lanes) {
                    int v[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) v[j] = k + j * lanes < n ? __ldg(row + x_of(k + j * lanes)) : -1;
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (v[j] >= 0) count(counters_of(x_of(k + j * lanes)), v[j]);
                }
            }
            continue;
        }
        for (int k = lane; k < n; k += lanes) {
            const int x = x_of(k);
            uint32_t *c = counters_of(x);
            const uint16_t *p = row + x + z_first * plane;
            for (int z = z_first; z < planes; z += z_step, p += z_step * plane) {
                int v[8];
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = z + j < planes ? __ldg(p + j * plane) : -1;
#pragma unroll
                for (int j = 0; j < 8; j++) count(c, v[j]);
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

// Host words laid out in 16-byte aligned segments, for one copy to the device.
struct HostTables {
    std::vector<uint32_t> words;
    size_t add(const uint32_t *p, size_t n) {
        const size_t at = words.size();
        words.insert(words.end(), p, p + n);
        words.resize((words.size() + 3) / 4 * 4, 0);
        return at;
    }
    size_t bytes() const { return words.size() * sizeof(uint32_t); }
    cudaError_t copy_to(void *dev, cudaStream_t st) const {
        return cudaMemcpyAsync(dev, words.data(), bytes(), cudaMemcpyHostToDevice, st);
    }
};

// The status of a call whose launches gave `rc`; waits for `st`, as the host tables must outlive
// their copy.
int finish(SpareBuffer &scratch, cudaStream_t st, int rc, const char *what) {
    cudaError_t e = rc == MAXI_OK ? cudaGetLastError() : cudaSuccess;
    const cudaError_t e2 = scratch.data() ? scratch.give_back() : cudaStreamSynchronize(st);
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
                  int64_t farthest, Counted counted, cudaStream_t st) {
    const int64_t sms = sm_count(), rows = nzl * Ny;
    auto direct = [&](auto kernel) {
        const unsigned grid = (unsigned) std::min<int64_t>(rows, sms * 16);
        kernel<<<grid, vec ? 128 : 256, 0, st>>>(voxels, nzl, Ny, Nx, z_start, y_start, x_start, vm, cy, cx, xb, yb, zb,
                                                 rb, voxel_bins, n_r);
        return (int) MAXI_OK;
    };
    if (voxel_bins > kMaxSharedBins || rows * Nx < kAxisMinVoxels)
        return direct(vec ? axis_histograms_direct<true, false> : axis_histograms_direct<false, false>);
    const bool exact = !vm.T;
    auto launch = [&](auto kernel, int64_t grid, int threads, int cells, auto... args) {
        const int smem = cells * (int) sizeof(uint32_t);
        cudaError_t e = allow_dynamic_smem(kernel, smem);
        if (e != cudaSuccess) return set_cuda_error(e, "axis histograms set-up");
        kernel<<<(unsigned) grid, threads, smem, st>>>(args...);
        return (int) MAXI_OK;
    };
    // z and y: several chunks per plane (or y) where there are few of them, of 16 rows at least.
    auto row_sets = [&](int64_t sets, int64_t first_set, int64_t set_step, int64_t row_step, int64_t row_count,
                        int64_t first_row, unsigned long long *bins, Counted mark, Counted read) {
        const int64_t n = row_count - first_row, n_sets = sets - first_set;
        const int64_t chunks = std::max<int64_t>(1, std::min(ceil_div(sms * 8, n_sets), n / 16));
        const int64_t per = ceil_div(n, chunks);
        const RowSets s{sets, set_step, row_step, row_count, first_row, per, first_set, bins, mark, read};
        auto kernel = [&](auto split) {
            constexpr bool S = decltype(split)::value;
            return vec ? (exact ? row_set_histograms<true, true, S> : row_set_histograms<true, false, S>)
                       : (exact ? row_set_histograms<false, true, S> : row_set_histograms<false, false, S>);
        };
        return launch(per < 8 ? kernel(std::true_type{}) : kernel(std::false_type{}), n_sets * ceil_div(n, per), 256,
                      voxel_bins, voxels, Nx, x_start, vm, s, voxel_bins);
    };
    int rc = row_sets(nzl, 0, Ny, 1, Ny, y_start, zb + z_start * voxel_bins, counted, Counted{});
    if (rc == MAXI_OK) rc = row_sets(Ny, y_start, 1, Ny, nzl, 0, yb, Counted{}, counted);
    if (rc) return rc;
    // x: strips of 8, or as many as the counters allow; chunks of at least 2048 rows, and beyond a
    // block per SM of two rows per bin, for which a block clears and flushes `strip` counters (64 x 512 x
    // 512, 4096 bins: 167 -> 148 us a call).
    const int strip = std::min(kVec, kBlockCells / voxel_bins), strips = (int) ceil_div(Nx, strip);
    const int64_t x_chunks = std::max<int64_t>(
        1, std::min({ceil_div(sms * 4, strips), rows / 2048, std::max(rows / (2 * voxel_bins), sms / strips)}));
    const int64_t x_per = ceil_div(rows, x_chunks);
    const bool wide = vec && strip == kVec;
    rc = launch(wide ? (exact ? strip_histograms<true, true> : strip_histograms<true, false>)
                     : (exact ? strip_histograms<false, true> : strip_histograms<false, false>), strips * ceil_div(rows, x_per),
                1024, strip * voxel_bins, voxels, rows, Ny, Nx, y_start, x_start, vm, strips, strip, x_per, xb, voxel_bins,
                counted);
    if (rc) return rc;
    // r: rings of as many radii as the counters allow, up to 64 (a wider row interval reads no
    // fewer sectors), in chunks of 16 planes or more.  Few rings, of a volume with few bins or
    // planes, are shared by several blocks, as long as a block has 8 pixels per counter that
    // it clears and adds to the bins; if that leaves SMs idle, the rings get narrower.
    // (1 x 4096 x 4096, 64 bins: 5510 us with 6 blocks of 512 radii, 169 now.)
    const int64_t radii = std::min<int64_t>(n_r, (int64_t) (1.4142136 * (double) farthest) + 2);
    if (radii > 46340 - 64)  // squared distances of 2^31 in the last ring
        return direct(vec ? axis_histograms_direct<true, true> : axis_histograms_direct<false, true>);
    int64_t width = std::min<int64_t>({radii, 64, std::max(1, kBlockCells / voxel_bins)});
    // Volumes of some extent both ways take two blocks per SM, as the rows of narrow rings are of
    // more even length: 64 x 301 x 333, 512 bins 111 -> 102 us a call, 32 x 1024 x 1024, 512 bins 344 -> 224; of less,
    // 1024 x 64 x 64, 64 bins 84 -> 89.
    const int64_t enough = std::min<int64_t>(Ny, Nx) >= 128 ? sms * 2 : sms * 3 / 4, least = kVec / 2;
    int64_t rings, chunks, parts;
    for (;; width /= 2) {
        rings = ceil_div(radii, width);
        chunks = std::min(ceil_div(sms * 6, rings), ceil_div(nzl, 16));
        const int64_t pixels = rows * Nx / (rings * chunks);
        parts = std::max<int64_t>(1, std::min({ceil_div(sms * 6, rings * chunks), ceil_div(std::min(Ny, 2 * radii), 128),
                                               pixels / (8 * width * voxel_bins)}));
        if (rings * chunks * parts >= enough || width <= least) break;
    }
    const int64_t per = ceil_div(nzl, chunks);
    chunks = ceil_div(nzl, per);
    // Rows that a ring of half the largest radius meets.
    const double half = 0.5 * (double) radii, widest = (double) std::max(std::abs(x_start - cx), std::abs(Nx - 1 - cx));
    const double low = std::sqrt(std::max(0.0, half * half - widest * widest));
    const bool split = per <= 2 || 2.0 * (half + (double) width - low) < 64.0 || Ny < 64;
    auto kernel = split ? (exact ? ring_histograms<true, true> : ring_histograms<false, true>)
                        : (exact ? ring_histograms<true, false> : ring_histograms<false, false>);
    return launch(kernel, rings * chunks * parts, 1024, (int) width * voxel_bins, voxels, nzl, (int) Ny, Nx,
                  (int) y_start, x_start, vm, (int) cy, (int) cx, (int) rings, (int) width, per, (int) chunks, (int) parts, rb,
                  voxel_bins, (int) n_r, counted);
}

// Voxels from which the partitioned form is the faster one, with at most kFewParts partitions
// and with more.  Direct against partitioned, with torch's call, us: 3 partitions (256 x 512
// bins) 59 / 53 at 2^20 voxels, 86 / 71 at 2^22, 154 / 88 at 2^23; 158 partitions (2048 x 4096)
// 63 / 58 at 2^21, 63 / 78 at 2^22, 145 / 87 at 2^23.
constexpr int kFewParts = 8;
constexpr int64_t kFieldMinVoxelsFew = int64_t(1) << 20, kFieldMinVoxels = int64_t(3) << 21;
// Vectors of one batch: the keys of 2^25 vectors take 512 MB.
constexpr int64_t kBatchVecs = int64_t(1) << 25;

SmallDiv small_div(uint32_t d) {
    if (d == 1) return SmallDiv{1, 0, 1};
    return SmallDiv{d, (uint32_t) (((uint64_t(1) << 32) + d - 1) / d), 0};
}

// field_histogram_kernel's call, partitioned, in batches of whole rows.
struct FieldPlan {
    bool partitioned;
    int group, parts;
    int64_t per_row, batch_rows, tiles;  // vectors per row; rows and tiles of a (full) batch
    size_t o_totals, o_starts, o_keys, bytes;
};

FieldPlan field_plan(int64_t nZ, int64_t nY, int64_t nX, int64_t field_bins, int64_t voxel_bins, size_t tables) {
    FieldPlan f{};
    f.bytes = tables;
    f.group = (int) std::min<int64_t>(std::min<int64_t>(kPartCells / voxel_bins, kMaxGroup), field_bins);
    if (f.group < 1 || ceil_div(field_bins, f.group) > kMaxParts || nX > (1 << 18) || nZ * nY >= (int64_t(1) << 31) ||
        nZ * nY * nX < (ceil_div(field_bins, f.group) <= kFewParts ? kFieldMinVoxelsFew : kFieldMinVoxels))
        return f;
    f.partitioned = true;
    f.parts = (int) ceil_div(field_bins, f.group);
    f.per_row = ceil_div(nX, kVec);
    f.batch_rows = std::min(nZ * nY, kBatchVecs / f.per_row);
    f.tiles = ceil_div(f.batch_rows * f.per_row, kTileVecs);
    auto place = [&](size_t n) {
        const size_t at = f.bytes;
        f.bytes += (n + 255) / 256 * 256;
        return at;
    };
    f.o_totals = place((size_t) f.parts * sizeof(uint32_t));
    f.o_starts = place((size_t) (f.parts + 1) * round_up(f.tiles, 4) * sizeof(uint16_t));
    f.o_keys = place((size_t) f.tiles * kTileKeys * sizeof(uint16_t));
    return f;
}

int field_launches(const FieldPlan &f, PartitionArgs a, uint8_t *scratch, int64_t rows, bool vec, cudaStream_t st) {
    const bool exact = !a.vm.T && !a.fm.T;
    auto sort = vec ? (exact ? partition_keys<true, true> : partition_keys<true, false>)
                    : (exact ? partition_keys<false, true> : partition_keys<false, false>);
    const int smem = kPartCells * (int) sizeof(uint32_t), sms = sm_count();
    cudaError_t e = cudaFuncSetAttribute(count_partitions, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    a.totals = reinterpret_cast<uint32_t *>(scratch + f.o_totals);
    a.starts = reinterpret_cast<uint16_t *>(scratch + f.o_starts);
    a.keys = reinterpret_cast<uint16_t *>(scratch + f.o_keys);
    a.parts = f.parts;
    a.pitch = (int) round_up(f.tiles, 4);
    a.group = small_div((uint32_t) f.group);
    a.per_row = small_div((uint32_t) f.per_row);
    for (int64_t row = 0; row < rows && e == cudaSuccess; row += f.batch_rows) {
        a.first_row = (uint32_t) row;
        a.rows = (uint32_t) std::min(f.batch_rows, rows - row);
        a.tiles = (int) ceil_div(a.rows * f.per_row, kTileVecs);
        e = cudaMemsetAsync(a.totals, 0, f.parts * sizeof(uint32_t), st);
        if (e != cudaSuccess) break;
        sort<<<(unsigned) std::min(a.tiles, 2 * sms), kKeyThreads, 0, st>>>(a);
        count_partitions<<<(unsigned) sms, 1024, smem, st>>>(a);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? (int) MAXI_OK : set_cuda_error(e, "field histogram");
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
    xmap.resize(round_up(nX, kVec), 0);
    HostTables t;
    const size_t o_vT = t.add(vT.data(), vT.size()), o_fT = t.add(fT.data(), fT.size());
    const size_t o_z = t.add(zmap.data(), zmap.size()), o_y = t.add(ymap.data(), ymap.size());
    const size_t o_x = t.add(xmap.data(), xmap.size());
    const size_t tables = (t.bytes() + 255) / 256 * 256;
    FieldPlan f = field_plan(nZ, nY, nX, field_bins, voxel_bins, tables);
    SpareBuffer scratch;
    rc = scratch.take(f.bytes, st, "histogram");
    if (rc == MAXI_ERR_OUT_OF_MEMORY && f.partitioned) {  // the direct form needs the tables alone
        clear_error();
        f.partitioned = false;
        rc = scratch.take(tables, st, "histogram");
    }
    if (rc) return rc;
    const cudaError_t e = t.copy_to(scratch.data(), st);
    if (e != cudaSuccess) return set_cuda_error(e, "histogram tables");
    const uint32_t *dev = reinterpret_cast<const uint32_t *>(scratch.data());
    if (!vT.empty()) vm.T = dev + o_vT;
    if (!fT.empty()) fm.T = dev + o_fT;
    const int32_t *zm = reinterpret_cast<const int32_t *>(dev + o_z);
    const int32_t *ym = reinterpret_cast<const int32_t *>(dev + o_y);
    const int32_t *xm = reinterpret_cast<const int32_t *>(dev + o_x);
    auto *b = reinterpret_cast<unsigned long long *>(bins);
    const bool vec = nX % kVec == 0 && reinterpret_cast<uintptr_t>(voxels) % 16 == 0;
    if (f.partitioned) {
        PartitionArgs a{};
        a.voxels = voxels;
        a.field = field;
        a.ny = ny;
        a.nx = nx;
        a.nX = (int) nX;
        a.x_start = (int) x_start;
        a.nY = (uint32_t) nY;
        a.y_start = (uint32_t) y_start;
        a.vm = vm;
        a.fm = fm;
        a.zmap = zm;
        a.ymap = ym;
        a.xmap = xm;
        a.voxel_bins = (int) voxel_bins;
        a.field_bins = (int) field_bins;
        a.bins = b;
        rc = field_launches(f, a, scratch.data(), nZ * nY, vec, st);
    } else {
        const unsigned grid = (unsigned) std::min<int64_t>(nZ * nY, (int64_t) sm_count() * 16);
        if (vec)
            field_histogram_kernel<true><<<grid, 128, 0, st>>>(voxels, field, nZ, nY, (int) nX, ny, nx, y_start,
                                                               (int) x_start, vm, fm, zm, ym, xm, b, voxel_bins);
        else
            field_histogram_kernel<false><<<grid, 256, 0, st>>>(voxels, field, nZ, nY, (int) nX, ny, nx, y_start,
                                                                (int) x_start, vm, fm, zm, ym, xm, b, voxel_bins);
    }
    return finish(scratch, st, rc, "field histogram");
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
    HostTables t;
    t.add(vT.data(), vT.size());
    SpareBuffer scratch;
    static std::atomic<uint32_t> calls{0};
    constexpr size_t kCounted = 256;  // for Counted::word
    rc = scratch.take(kCounted + t.bytes(), st, "histogram");
    if (rc == MAXI_ERR_OUT_OF_MEMORY && vT.empty()) {
        clear_error();
        rc = MAXI_OK;
    }
    if (rc) return rc;
    if (!vT.empty()) {
        const cudaError_t e = t.copy_to(scratch.data() + kCounted, st);
        if (e != cudaSuccess) return set_cuda_error(e, "histogram tables");
        vm.T = reinterpret_cast<const uint32_t *>(scratch.data() + kCounted);
    }
    auto *xb = reinterpret_cast<unsigned long long *>(x_bins), *yb = reinterpret_cast<unsigned long long *>(y_bins);
    auto *zb = reinterpret_cast<unsigned long long *>(z_bins), *rb = reinterpret_cast<unsigned long long *>(r_bins);
    const bool vec = Nx % kVec == 0 && reinterpret_cast<uintptr_t>(voxels) % 16 == 0;
    rc = axis_launches(voxels, nzl, Ny, (int) Nx, z_start, y_start, (int) x_start, vm, cy, cx, xb, yb, zb, rb,
                       (int) voxel_bins, n_r, vec, std::max(rx, ry),
                       Counted{reinterpret_cast<uint32_t *>(scratch.data()), ++calls}, st);
    return finish(scratch, st, rc, "axis histograms");
}
