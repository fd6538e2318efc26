// 3-D sphere dilation and erosion of masks: the reference's morphology module
// (src/lib/cpp/gpu/morphology.cc, cpu_seq/morphology.cc; bound by
// src/pybind/morphology-pybind.cc:24-76,147-150), the step that prepares the
// implant mask before the diffusion (src/processing_steps/0750_bone_region.py:162 via
// src/lib/py/helpers.py:326-349 and morph_3d, :805-850).
//
// uint8 form: result[z,y,x] = 1 iff, over every in-volume offset with
// pz^2 + py^2 + px^2 <= r^2, some voxel is nonzero (dilation) / every voxel has bit 0
// set (erosion: std::bit_and of a bool and a byte).  Offsets outside the volume
// take no part.
//
// Bit-packed form: uint32 words, MSB first along x.  The reference builds one 32-bit
// kernel row per (pz, py) holding x offsets -r .. 31 - r, and reads the three words
// around each output word; with the GPU build's shifts (a shift by 32 or more, or by a
// negative amount, gives 0) that is the sphere with x offsets clipped at 31 - r.
//
// Two kernels over packed words, radius <= 32 (OP is OR for dilation, AND for erosion;
// outside-volume rows and words and the padding bits of a row are the neutral element):
//   1. morph_partials walks a tile of 32 rows through a block of planes (2 to 48).  Per plane it
//      builds, in shared memory, the x-runs X_w = OP over x offsets -w .. min(w, P) (P = r
//      for the uint8 form, 31 - r for the bit-packed one), w = 0 .. r, of the tile's rows
//      +- r, one funnel shift each way per step.  The sphere's cross-section at |pz| = k is
//      D_k = OP over py of X_w(k, py)[y + py], w(k, py) = isqrt(r^2 - k^2 - py^2).  D_k
//      contains D_{k+1}, so with k falling from r only the rows whose run grew are added:
//      about 0.5 r^2 row pairs for all k together instead of (pi/4) r^2.  Each D_k goes at
//      once into the running OPs of the output planes z - k and z + k, which a thread keeps
//      in registers and shifts by one plane per step; a finished plane is written out.
//   2. morph_combine: an output plane is the OP of the blocks whose planes reach it.
// What bounds 1 is shared-memory bandwidth: two 4-byte reads per pair and word, 262 of them
// at r = 16 (0.47 ms per 512 x 1024 x 1024 voxels at 128 bytes per cycle and SM), the
// x-runs 34 writes more.  Hence several words per thread, so that a table entry and its address
// arithmetic serve all of them: four, or two above radius 8, where the 2r + 1 running
// planes fill the registers.  Blocks of planes without a recomputed halo keep scratch traffic at about two words per
// word (17 of them before, one per k) and leave enough blocks to fill the chip.
// 512 x 1024 x 1024 voxels, bit-packed, on a B200, before (all discs to global scratch) and
// now: r = 2 366 and 218 us, r = 10 1421 and 590, r = 16 3427 and 1018 (shared memory 72%
// busy, issue 57%), r = 20 7958 and 1611, r = 31 27900 and 3954; the uint8 form at r = 16
// 3686 and 1156 (pack 101, unpack and combine 148).  Two words per thread instead of four
// from radius 9 on: 1010 against 1074 us at r = 16 (twice the warps).
#include "common.cuh"
#include "host_util.h"
#include "launch.cuh"
#include "scratch.h"

namespace maxi {
namespace {

constexpr int kMorphMaxRadius = 32;

template <bool DILATE>
__device__ __forceinline__ uint32_t op(uint32_t a, uint32_t b) {
    return DILATE ? (a | b) : (a & b);
}

constexpr int kTileRows = 32;
constexpr int kMaxPlanes = 48;     // planes per block, at most
constexpr int kMorphThreads = 128;
constexpr int kMaxPairs = 512;     // row pairs over all k (495 at radius 32)

// Words per thread and per tile row, by the radius bucket that the running planes are sized for.
constexpr int words_per_thread(int rb) { return rb <= 8 ? 4 : 2; }
constexpr int tile_words(int rb) { return kMorphThreads * words_per_thread(rb) / kTileRows; }

struct MorphTile {
    int64_t pitch;  // words of a scratch row, a multiple of 4
    int nw, ny, nz, radius, pmax, planes;
    int x_tiles, y_tiles, blocks;
    int start[kMorphMaxRadius + 2];       // pairs of k: start[k] .. start[k + 1] - 1
    int2 pair[kMaxPairs];                 // byte offsets of X_w[y + py] and X_w[y - py] from X_0[y]
};

// The row pairs that D_k adds to D_{k+1} for every k, as offsets into the shared x-runs.
void fill_pairs(MorphTile &t, int r, int row_bytes) {
    auto root = [](int n) {
        int q = 0;
        while ((q + 1) * (q + 1) <= n) q++;
        return q;
    };
    const int run_bytes = (kTileRows + 2 * r) * row_bytes;
    int n = 0;
    for (int k = 0; k <= r; k++) {
        t.start[k] = n;
        for (int py = 0; py * py <= r * r - k * k; py++) {
            const int w = root(r * r - k * k - py * py), above = r * r - (k + 1) * (k + 1) - py * py;
            if (above >= 0 && root(above) == w) continue;
            t.pair[n++] = make_int2(w * run_bytes + py * row_bytes, w * run_bytes - py * row_bytes);
        }
    }
    t.start[r + 1] = n;
}

template <int V> struct Words {
    uint32_t w[V];
};
template <int V>
__device__ __forceinline__ Words<V> load_words(const char *p) {
    Words<V> v;
    if constexpr (V == 4) {
        const uint4 q = *reinterpret_cast<const uint4 *>(p);
        v.w[0] = q.x, v.w[1] = q.y, v.w[2] = q.z, v.w[3] = q.w;
    } else {
        const uint2 q = *reinterpret_cast<const uint2 *>(p);
        v.w[0] = q.x, v.w[1] = q.y;
    }
    return v;
}
template <int V>
__device__ __forceinline__ void store_words(void *p, const Words<V> &v) {
    if constexpr (V == 4) *reinterpret_cast<uint4 *>(p) = make_uint4(v.w[0], v.w[1], v.w[2], v.w[3]);
    else *reinterpret_cast<uint2 *>(p) = make_uint2(v.w[0], v.w[1]);
}

// RB: radius bucket (radius <= RB).  Bits at x offset d of word j come from the stream
// (left, word, right): d < 0 from funnelshift_rc(word, left, -d), d > 0 from
// funnelshift_lc(right, word, d).
template <bool DILATE, int RB>
__global__ void __launch_bounds__(kMorphThreads) morph_partials(const uint32_t *__restrict__ in,
                                                                uint32_t *__restrict__ partial,
                                                                const __grid_constant__ MorphTile t) {
    constexpr int V = words_per_thread(RB), W = tile_words(RB), kRowBytes = W * 4, kPer = W / V;
    constexpr uint32_t neutral = DILATE ? 0u : 0xffffffffu;
    extern __shared__ __align__(16) char runs[];  // [r + 1][kTileRows + 2r][W] words
    const int r = t.radius, rows = kTileRows + 2 * r;
    int b = blockIdx.x;
    const int64_t x0 = (int64_t) (b % t.x_tiles) * W;
    b /= t.x_tiles;
    const int block = b / t.y_tiles;
    const int64_t y0 = (int64_t) (b % t.y_tiles) * kTileRows;
    const int64_t z0 = (int64_t) block * t.planes, z1 = min(z0 + t.planes, (int64_t) t.nz);
    const int ty = threadIdx.x / kPer, tx = threadIdx.x % kPer * V;
    const char *mine = runs + (ty + r) * kRowBytes + tx * 4;  // X_0 at this thread's row and words
    const bool store_ok = y0 + ty < t.ny && x0 + tx < t.pitch;
    uint32_t *out = partial + ((int64_t) block * (t.planes + 2 * r) * t.ny + y0 + ty) * t.pitch + x0 + tx;
    const int64_t out_plane = (int64_t) t.ny * t.pitch;
    auto put = [&](int64_t zo, const Words<V> &v) {  // output plane zo, if this block reaches it
        if (store_ok && zo >= max((int64_t) 0, z0 - r) && zo < min((int64_t) t.nz, z1 + r))
             store_words<V>(out + (zo - z0 + r) * out_plane, v);
    };
    Words<V> run[2 * RB + 1];  // running OP of output planes z - RB .. z + RB
#pragma unroll
    for (int j = 0; j <= 2 * RB; j++)
#pragma unroll
        for (int v = 0; v < V; v++) run[j].w[v] = neutral;
#pragma unroll 1
    for (int64_t z = z0; z < z1; z++) {
        __syncthreads();  // the previous plane's x-runs have been read
        const uint32_t *plane = in + z * t.ny * t.nw;
        for (int i = threadIdx.x; i < rows * kPer; i += kMorphThreads) {
            const int row = i / kPer, c = i % kPer * V;
            const int64_t y = y0 - r + row;
            uint32_t m[V + 2], acc[V];
#pragma unroll
            for (int j = 0; j < V + 2; j++) {
                const int64_t x = x0 + c + j - 1;
                m[j] = y >= 0 && y < t.ny && x >= 0 && x < t.nw ? __ldg(plane + y * t.nw + x) : neutral;
            }
            char *dst = runs + row * kRowBytes + c * 4;
            Words<V> x;
#pragma unroll
            for (int j = 0; j < V; j++) x.w[j] = acc[j] = m[j + 1];
            store_words<V>(dst, x);
            for (int w = 1; w <= r; w++) {
                dst += rows * kRowBytes;
#pragma unroll
                for (int j = 0; j < V; j++) {
                    acc[j] = op<DILATE>(acc[j], __funnelshift_rc(m[j + 1], m[j], w));
                    if (w <= t.pmax) acc[j] = op<DILATE>(acc[j], __funnelshift_lc(m[j + 2], m[j + 1], w));
                    x.w[j] = acc[j];
                }
                store_words<V>(dst, x);
            }
        }
        __syncthreads();
        Words<V> d, carry;  // D_k; the running plane that moves into the place of z + k
#pragma unroll
        for (int v = 0; v < V; v++) d.w[v] = carry.w[v] = neutral;
#pragma unroll
        for (int k = RB; k >= 0; k--) {
            if (k <= r) {
                const int last = t.start[k + 1];
#pragma unroll 4
                for (int e = t.start[k]; e < last; e++) {
                    const int2 at = t.pair[e];
                    const Words<V> p = load_words<V>(mine + at.x), q = load_words<V>(mine + at.y);
#pragma unroll
                    for (int v = 0; v < V; v++) d.w[v] = op<DILATE>(d.w[v], op<DILATE>(p.w[v], q.w[v]));
                }
            }
#pragma unroll
            for (int v = 0; v < V; v++) {
                if (k > 0) {
                    run[RB - k].w[v] = op<DILATE>(run[RB - k + 1].w[v], d.w[v]);
                    const uint32_t moved = run[RB + k].w[v];
                    run[RB + k].w[v] = op<DILATE>(carry.w[v], d.w[v]);
                    carry.w[v] = moved;
                } else {
                    run[RB].w[v] = op<DILATE>(carry.w[v], d.w[v]);
                }
            }
        }
        put(z - RB, run[0]);
    }
#pragma unroll
    for (int j = 1; j <= 2 * RB; j++) put(z1 - 1 - RB + j, run[j]);
}

// Where word i of [nz][ny][nw] lies.
struct WordAt {
    int64_t row, z, y;
    int x;
    __device__ __forceinline__ WordAt(int64_t i, int64_t ny, int nw) {
        if (i < (int64_t(1) << 31) && ny < (int64_t(1) << 31)) {  // 32-bit divisions
            const uint32_t r = (uint32_t) i / (uint32_t) nw, p = r / (uint32_t) ny;
            row = r, z = p, y = r - p * (uint32_t) ny, x = (int) ((uint32_t) i - r * (uint32_t) nw);
        } else {
            row = i / nw, z = row / ny, y = row - z * ny, x = (int) (i - row * nw);
        }
    }
};

// The partial planes' layout: block b holds planes b * planes - radius .. of the result.
struct Partials {
    const uint32_t *words;
    int64_t nz, ny, pitch;
    int radius, planes;
};

// OP of the word's partial values: those of the blocks whose planes reach its plane.
template <bool DILATE>
__device__ __forceinline__ uint32_t combined_word(const Partials &p, const WordAt &at) {
    const uint32_t z = (uint32_t) at.z, r = (uint32_t) p.radius, planes = (uint32_t) p.planes;
    const uint32_t lo = (z > r ? z - r : 0u) / planes, hi = min((uint32_t) p.nz - 1u, z + r) / planes;
    uint32_t acc = DILATE ? 0u : 0xffffffffu;
    for (uint32_t b = lo; b <= hi; b++) {
        const int64_t plane = (int64_t) b * (planes + 2 * r) + (z + r - b * planes);
        acc = op<DILATE>(acc, __ldg(p.words + (plane * p.ny + at.y) * p.pitch + at.x));
    }
    return acc;
}

// Packed result.  One thread per word.
template <bool DILATE>
__global__ void morph_combine(const Partials p, uint32_t *__restrict__ out, int64_t words, int nw) {
    for (int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (int64_t) gridDim.x * blockDim.x) {
        out[i] = combined_word<DILATE>(p, WordAt(i, p.ny, nw));
    }
}

// Words that a warp takes at a time where it handles a word's 32 voxels in one step: 32, or fewer
// for volumes that would leave warps idle (16^3: packing 8.7 us with 32, 1.7 with 1).
int words_per_warp(int64_t words, int64_t warps) {
    int n = 32;
    while (n > 1 && ceil_div(words, n) < warps) n /= 2;
    return n;
}

// uint8 result.  A warp combines `per` words (32 or a smaller power of two) and writes them out
// together: 16 bytes per lane (VEC: rows are whole words and 16-byte aligned, 32 words), or a word's 32
// voxels at a time.
template <bool DILATE, bool VEC, int PER>
__global__ void morph_combine_u8(const Partials p, uint8_t *__restrict__ out, int64_t words, int nx, int nw, int few) {
    const int lane = threadIdx.x & 31, per = PER ? PER : few;
    const int64_t stride = (int64_t) gridDim.x * blockDim.x / 32 * per;
    for (int64_t first = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) / 32 * per; first < words; first += stride) {
        const WordAt at(min(first + (VEC ? lane : min(lane, per - 1)), words - 1), p.ny, nw);
        const uint32_t word = combined_word<DILATE>(p, at);
        const uint32_t bits = __brev(word);  // bit q: voxel q
        if (VEC) {
#pragma unroll
            for (int half = 0; half < 2; half++) {
                const int c = half * 32 + lane;  // 16-byte chunk of the warp's 1024 voxels
                const uint32_t h = __shfl_sync(0xffffffffu, bits, c >> 1) >> (16 * (c & 1));
                uint4 v;
                v.x = ((h & 15u) * 0x00204081u) & 0x01010101u;
                v.y = ((h >> 4 & 15u) * 0x00204081u) & 0x01010101u;
                v.z = ((h >> 8 & 15u) * 0x00204081u) & 0x01010101u;
                v.w = ((h >> 12 & 15u) * 0x00204081u) & 0x01010101u;
                if (first + (c >> 1) < words) __stcs(reinterpret_cast<uint4 *>(out + first * 32) + c, v);
            }
        } else {
            const int x = at.x * 32;
            for (int k = 0; k < per && first + k < words; k++) {
                const uint32_t b = __shfl_sync(0xffffffffu, bits, k);
                const int64_t r = __shfl_sync(0xffffffffu, at.row, k);
                const int xk = __shfl_sync(0xffffffffu, x, k) + lane;
                if (xk < nx) out[r * nx + xk] = (uint8_t) (b >> lane & 1u);
            }
        }
    }
}

// uint8 rows -> packed words (MSB first), padding bits neutral.  VEC: rows are whole words
// (nx % 32 == 0) and 16-byte aligned, one thread per word with two 16-byte loads; otherwise
// a warp takes `per` words, a word's 32 voxels at a time.
template <bool DILATE, bool VEC, int PER>
__global__ void morph_pack(const uint8_t *__restrict__ in, uint32_t *__restrict__ packed, int64_t words, int nx,
                           int nw, int few) {
    const int per = PER ? PER : few;
    const int64_t stride = (int64_t) gridDim.x * blockDim.x, thread = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (VEC) {
        for (int64_t idx = thread; idx < words; idx += stride) {
            const uint4 *p = reinterpret_cast<const uint4 *>(in + idx * 32);
            const uint4 q0 = __ldcs(p), q1 = __ldcs(p + 1);
            const uint32_t u[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            uint32_t w = 0;
#pragma unroll
            for (int b = 0; b < 32; b++) {
                const uint32_t byte = (u[b >> 2] >> (8 * (b & 3))) & 0xffu;
                w |= (DILATE ? (uint32_t) (byte != 0) : (byte & 1u)) << (31 - b);
            }
            packed[idx] = w;
        }
        return;
    }
    const int lane = threadIdx.x & 31;
    for (int64_t first = thread / 32 * per; first < words; first += stride / 32 * per) {
        uint32_t mine = 0;
#pragma unroll 8
        for (int k = 0; k < per; k++) {
            const WordAt at(min(first + k, words - 1), 1, nw);
            const int x = at.x * 32 + lane;
            bool bit = !DILATE;
            if (x < nx) {
                const uint8_t v = __ldg(in + at.row * nx + x);
                bit = DILATE ? v != 0 : v & 1;
            }
            const uint32_t word = __brev(__ballot_sync(0xffffffffu, bit));
            if (lane == k) mine = word;
        }
        if (lane < per && first + lane < words) packed[first + lane] = mine;
    }
}

unsigned grid_for(int64_t n) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (unsigned) std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), (int64_t) sms * 16));
}

int bucket_smem(int radius) {
    const int rb = std::max(4, (int) round_up(radius, 4));
    return (radius + 1) * (kTileRows + 2 * radius) * tile_words(rb) * 4;
}

// The kernel of a radius, allowed its shared memory, and the blocks of it that run at once.
template <bool DILATE>
int morph_kernel(int radius, void (**kernel)(const uint32_t *, uint32_t *, const MorphTile), int *resident) {
    switch ((radius + 3) / 4) {
    case 0:
    case 1: *kernel = morph_partials<DILATE, 4>; break;
    case 2: *kernel = morph_partials<DILATE, 8>; break;
    case 3: *kernel = morph_partials<DILATE, 12>; break;
    case 4: *kernel = morph_partials<DILATE, 16>; break;
    case 5: *kernel = morph_partials<DILATE, 20>; break;
    case 6: *kernel = morph_partials<DILATE, 24>; break;
    case 7: *kernel = morph_partials<DILATE, 28>; break;
    default: *kernel = morph_partials<DILATE, 32>; break;
    }
    int dev = 0, sms = 148, per_sm = 1;
    cudaError_t e = allow_dynamic_smem(*kernel, bucket_smem(radius));
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, *kernel, kMorphThreads, bucket_smem(radius));
    if (e != cudaSuccess) return set_cuda_error(e, "morphology set-up");
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    *resident = std::max(1, per_sm) * sms;
    return MAXI_OK;
}

// The cut of a volume into tiles and blocks of planes: the number of planes per block that
// ends first, counting rounds of resident blocks and about one plane's time to start and
// finish a block.  It is small volumes that this is for (128^3, r = 8: 44 us with 2 planes
// per block, 134 with 32, which leave 16 blocks); large ones are even from 16 planes on.  At
// least two planes: the scratch then stays within (radius + 1) words per word, of rows rounded up to
// 4 words.
MorphTile morph_tile(int64_t nz, int64_t ny, int64_t nw, int radius, int pmax, int resident) {
    MorphTile t{};
    t.nw = (int) nw;
    t.pitch = round_up(nw, 4);
    t.ny = (int) ny;
    t.nz = (int) nz;
    t.radius = radius;
    t.pmax = pmax;
    const int rb = std::max(4, (int) round_up(radius, 4));
    t.x_tiles = (int) ceil_div(nw, tile_words(rb));
    t.y_tiles = (int) ceil_div(ny, kTileRows);
    int64_t best = 0;
    for (int p = kMaxPlanes; p >= 2; p--) {
        const int64_t rounds = ceil_div((int64_t) t.x_tiles * t.y_tiles * ceil_div(nz, p), resident), cost = rounds * (p + 1);
        if (!best || cost < best) best = cost, t.planes = p;
    }
    t.blocks = (int) ceil_div(nz, t.planes);
    fill_pairs(t, radius, tile_words(rb) * 4);
    return t;
}
// The scratch: `radius` planes that reach over each cut between two blocks, from either side.  The
// first block's planes below 0 and the last one's above the volume are never written, so that the
// layout starts with the first block's plane `radius`.
int64_t partial_words(const MorphTile &t) {
    return (t.nz + 2 * (int64_t) t.radius * (t.blocks - 1)) * t.ny * t.pitch;
}
Partials partials(const MorphTile &t, const uint32_t *words) {
    return {words, t.nz, t.ny, t.pitch, t.radius, t.planes};
}

template <bool DILATE>
int morph_partial_planes(const uint32_t *in, uint32_t *partial, const MorphTile &t,
                         void (*kernel)(const uint32_t *, uint32_t *, const MorphTile), cudaStream_t st) {
    const int64_t grid = (int64_t) t.x_tiles * t.y_tiles * t.blocks;
    if (grid >= (int64_t(1) << 31)) return set_error(MAXI_ERR_UNSUPPORTED, "volume of too many tiles");
    kernel<<<(unsigned) grid, kMorphThreads, bucket_smem(t.radius), st>>>(in, partial, t);
    return MAXI_OK;
}

// A whole call, from the scratch on.  U8: `in` and `out` are voxels in rows of nx, else
// packed words (nx: 32 per word).
template <bool DILATE, bool U8>
int morph_run(const void *in, void *out, int64_t nz, int64_t ny, int64_t nx, int radius, cudaStream_t st,
              std::unique_lock<std::mutex> &hold) {
    const int64_t nw = ceil_div(nx, 32), words = nz * ny * nw;
    void (*kernel)(const uint32_t *, uint32_t *, const MorphTile) = nullptr;
    int resident = 0;
    int rc = morph_kernel<DILATE>(radius, &kernel, &resident);
    if (rc) return rc;
    const MorphTile t = morph_tile(nz, ny, nw, radius, U8 ? radius : 31 - radius, resident);
    // (uint8: the packed input, then) the partial planes
    const int64_t packed_words = U8 ? round_up(words, 4) : 0;
    uint32_t *scratch = nullptr;
    if ((rc = acquire_scratch((size_t) (packed_words + partial_words(t)) * sizeof(uint32_t), hold, &scratch, "morphology"))) return rc;
    uint32_t *partial = scratch + packed_words - (int64_t) t.radius * t.ny * t.pitch;
    if constexpr (U8) {
        const bool vec = nx % 32 == 0 && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
        const uint8_t *src = static_cast<const uint8_t *>(in);
        uint8_t *dst = static_cast<uint8_t *>(out);
        const int per = words_per_warp(words, 148 * 16);
        const unsigned g = grid_for(vec ? words : ceil_div(words, per) * 32);
        // (32 words a warp: their number known to the compiler, 0.5 to 0.9% of a call)
        auto pack = vec ? morph_pack<DILATE, true, 32> : per == 32 ? morph_pack<DILATE, false, 32> : morph_pack<DILATE, false, 0>;
        auto combine = vec ? morph_combine_u8<DILATE, true, 32>
                           : per == 32 ? morph_combine_u8<DILATE, false, 32> : morph_combine_u8<DILATE, false, 0>;
        pack<<<g, 256, 0, st>>>(src, scratch, words, (int) nx, t.nw, per);
        if ((rc = morph_partial_planes<DILATE>(scratch, partial, t, kernel, st))) return rc;
        combine<<<g, 256, 0, st>>>(partials(t, partial), dst, words, (int) nx, t.nw, per);
    } else {
        if ((rc = morph_partial_planes<DILATE>(static_cast<const uint32_t *>(in), partial, t, kernel, st))) return rc;
        morph_combine<DILATE><<<grid_for(words), 256, 0, st>>>(partials(t, partial), static_cast<uint32_t *>(out), words, t.nw);
    }
    return MAXI_OK;
}

int check_shape(int64_t nz, int64_t ny, int64_t n_inner, int64_t radius) {
    if (nz <= 0 || ny <= 0 || n_inner <= 0)
        return set_error(MAXI_ERR_INVALID_ARGUMENT, "shape (%lld, %lld, %lld) has an empty axis", (long long) nz,
                         (long long) ny, (long long) n_inner);
    if (radius < 0) return set_error(MAXI_ERR_INVALID_ARGUMENT, "negative radius");
    if (radius > kMorphMaxRadius)
        return set_error(MAXI_ERR_UNSUPPORTED, "sphere radius %lld: at most %d per call (apply radius-32 spheres "
                         "repeatedly for larger ones, as the reference's morph_3d does with 16)",
                         (long long) radius, kMorphMaxRadius);
    if (nz >= (int64_t(1) << 31) || ny >= (int64_t(1) << 31) || n_inner >= (int64_t(1) << 31))
        return set_error(MAXI_ERR_UNSUPPORTED, "axes of 2^31 or more are not served");
    return MAXI_OK;
}

}  // namespace

}  // namespace maxi

using namespace maxi;

extern "C" int maxi_morphology_sphere_bitpacked(const uint32_t *voxels, uint32_t *result, int64_t nz, int64_t ny,
                                                int64_t nw, int64_t radius, int dilate, void *stream) {
    clear_error();
    if (!voxels || !result) return set_error(MAXI_ERR_INVALID_ARGUMENT, "NULL pointer");
    int rc = check_shape(nz, ny, nw, radius);
    if (rc) return rc;
    if (radius > 31)  // the kernel row would lose offset 0
        return set_error(MAXI_ERR_UNSUPPORTED, "bit-packed sphere radius %lld: at most 31", (long long) radius);
    if ((rc = require_device())) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    std::unique_lock<std::mutex> hold;
    rc = dilate ? morph_run<true, false>(voxels, result, nz, ny, nw * 32, (int) radius, st, hold)
                : morph_run<false, false>(voxels, result, nz, ny, nw * 32, (int) radius, st, hold);
    cudaError_t e = cudaGetLastError();
    cudaError_t e2 = cudaStreamSynchronize(st);  // the scratch is free for the next call
    if (rc) return rc;
    if (e == cudaSuccess) e = e2;
    return e == cudaSuccess ? MAXI_OK : set_cuda_error(e, "bit-packed sphere morphology");
}

extern "C" int maxi_morphology_sphere(const uint8_t *voxels, uint8_t *result, int64_t nz, int64_t ny, int64_t nx,
                                      int64_t radius, int dilate, void *stream) {
    clear_error();
    if (!voxels || !result) return set_error(MAXI_ERR_INVALID_ARGUMENT, "NULL pointer");
    int rc = check_shape(nz, ny, nx, radius);
    if (rc) return rc;
    if ((rc = require_device())) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    std::unique_lock<std::mutex> hold;
    rc = dilate ? morph_run<true, true>(voxels, result, nz, ny, nx, (int) radius, st, hold)
                : morph_run<false, true>(voxels, result, nz, ny, nx, (int) radius, st, hold);
    cudaError_t e = cudaGetLastError();
    cudaError_t e2 = cudaStreamSynchronize(st);  // the scratch is free for the next call
    if (rc) return rc;
    if (e == cudaSuccess) e = e2;
    return e == cudaSuccess ? MAXI_OK : set_cuda_error(e, "sphere morphology");
}
