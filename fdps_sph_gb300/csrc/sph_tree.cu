// Morton keys, radix sort, particle permutation and octree construction.
//
// Replaces the tree construction FDPS performs inside every
// calcForceAllAndWriteBack call (main.cpp:93-101, 139-146; tree parameters
// main.cpp:86-90).  FDPS itself is not vendored with the reference, so the
// rules below are this project's specification, restated bit-for-bit by the
// CPU oracle (oracle/sph_oracle.c: or_root_box, or_morton_keys, or_sort_perm,
// or_tree_build):
//   * root cube: centre of the particle bounding box, side = largest extent
//     x (1 + 2^-10); keys = 3 x 21-bit Morton interleave (x high, z low);
//   * stable ascending sort of the keys (ties keep the previous order);
//   * a cell is split while it holds more than n_leaf particles and is above
//     level 21; children are the non-empty octants in octant order;
//   * monopole moments are sums over the particles of a leaf (ascending) and
//     over the children of a cell (octant order), each operation rounded once
//     (no fused multiply-add), so that centres of mass and hence the gravity
//     opening decisions are bit-identical to the oracle's.
#include <algorithm>
#include <climits>

#include "sph_physics.cuh"

namespace sph {

constexpr int SCAN_BLOCKS = 256;
constexpr int SCAN_THREADS = 256;

template <class T>
__device__ __forceinline__ T warp_incl_scan(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// inclusive block scan for blockDim.x <= 1024; returns inclusive value, *total = block sum
template <class T>
__device__ T block_incl_scan(T v, T *total) {
    __shared__ T ws[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    T x = warp_incl_scan(v);
    if (lane == 31) ws[wid] = x;
    __syncthreads();
    if (wid == 0) {
        T y = (lane < nw) ? ws[lane] : 0;
        y = warp_incl_scan(y);
        if (lane < nw) ws[lane] = y;
    }
    __syncthreads();
    if (wid > 0) x += ws[wid - 1];
    *total = ws[nw - 1];
    __syncthreads();
    return x;
}

// the sum of the blocks' parts before this block's, the sum of all in *total (SCAN_BLOCKS <= blockDim.x)
template <class T>
__device__ T parts_before(const T *part, T *total) {
    __shared__ T mine;
    const T v = threadIdx.x < SCAN_BLOCKS ? part[threadIdx.x] : 0;
    const T x = block_incl_scan(v, total);
    if (threadIdx.x == blockIdx.x) mine = x - v;
    __syncthreads();
    return mine;
}

__global__ void k_scan_reduce(const int *in, LenArg len, int *part) {
    after_previous();
    const int n = len.get();
    const int chunk = (n + gridDim.x - 1) / gridDim.x;
    const int b0 = blockIdx.x * chunk;
    const int b1 = min(n, b0 + chunk);
    int s = 0;
    for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) s += in[i];
    int tot;
    block_incl_scan(s, &tot);
    if (threadIdx.x == 0) part[blockIdx.x] = tot;
}

__global__ void k_scan_down(const int *in, int *out, LenArg len, const int *part, int *total) {
    after_previous();
    const int n = len.get();
    const int chunk = (n + gridDim.x - 1) / gridDim.x;
    const int b0 = blockIdx.x * chunk;
    const int b1 = min(n, b0 + chunk);
    int all;
    int base = parts_before(part, &all);
    if (blockIdx.x == 0 && threadIdx.x == 0 && total) *total = all;
    for (int t0 = b0; t0 < b1; t0 += blockDim.x) {
        const int i = t0 + threadIdx.x;
        const int v = (i < b1) ? in[i] : 0;
        int tot;
        const int x = block_incl_scan(v, &tot);
        if (i < b1) out[i] = base + x - v;
        base += tot;
    }
}

}  // namespace sph

using namespace sph;

// exclusive scan of int32 in two launches (every block of the second sums the first's parts itself); length from
// device (len_dev, if non-null) or host
int sph_scan_exclusive(sph_ctx *ctx, const int *in, int *out, const int *len_dev, int len_host, int *total_dev) {
    LenArg L{len_dev, len_host, 0};
    launch_after(true, k_scan_reduce, SCAN_BLOCKS, SCAN_THREADS, 0, ctx->stream, in, L, ctx->scan.part);
    ++ctx->launches;
    launch_after(true, k_scan_down, SCAN_BLOCKS, SCAN_THREADS, 0, ctx->stream, in, out, L, ctx->scan.part, total_dev);
    ++ctx->launches;
    SPH_CUDA(ctx, cudaGetLastError());
    return SPH_OK;
}

namespace sph {

// A few words for the host, written to pinned memory by a kernel: the host waits for them in every step, and a copy by
// the copy engine is a detour of the stream.  With the words that need clearing cleared by kernels that run anyway, a
// step of 5,000 particles 448 -> 427 us, of 100,000 1.247 -> 1.206 ms, of 10,000 in FP64 1.95 -> 1.90 ms.
__global__ void k_publish(const int *src, int n, int *host) {
    after_previous();
    if ((int)threadIdx.x < n) host[threadIdx.x] = src[threadIdx.x];
}

}  // namespace sph

// src[0 .. n) (n <= 64 ints) into the first words of host_scalars, in stream order
int sph_publish(sph_ctx *ctx, const int *src, int n) {
    launch_after(true, k_publish, 1, 64, 0, ctx->stream, src, n, (int *)ctx->host_scalars); ++ctx->launches;
    SPH_CUDA(ctx, cudaGetLastError());
    return SPH_OK;
}

namespace sph {

// ---------------------------------------------------------------------------
// root box and keys

// The boxes are reduced on order-preserving integer images of the doubles (dorder_key), so the minima and maxima
// run on the integer pipe: the FP64 pipe takes 16 cycles a warp instruction.  (-0 counts as +0; a NaN is left out, as by
// fmin and fmax.)
struct Box {
    long long lo[3], hi[3];
    __device__ __forceinline__ void empty() {
        for (int d = 0; d < 3; ++d) {
            lo[d] = LLONG_MAX;
            hi[d] = LLONG_MIN;
        }
    }
    __device__ __forceinline__ void add(int d, long long a, long long b) {
        lo[d] = min(lo[d], a);
        hi[d] = max(hi[d], b);
    }
    __device__ __forceinline__ void add(double px, double py, double pz) {
        const long long k[3] = {dorder_key(px), dorder_key(py), dorder_key(pz)};
        for (int d = 0; d < 3; ++d)
            if (llabs(k[d]) <= 0x7ff0000000000000LL) add(d, k[d], k[d]);
    }
    // of the whole block, valid in thread 0
    __device__ void reduce() {
        __shared__ long long s[6][32];
        for (int d = 0; d < 3; ++d)
            for (int o = 16; o > 0; o >>= 1)
                add(d, __shfl_xor_sync(0xffffffffu, lo[d], o), __shfl_xor_sync(0xffffffffu, hi[d], o));
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (lane == 0)
            for (int d = 0; d < 3; ++d) {
                s[d][wid] = lo[d];
                s[3 + d][wid] = hi[d];
            }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
                for (int d = 0; d < 3; ++d) add(d, s[d][w], s[3 + d][w]);
    }
};

// block b: the box of every gridDim.x-th 256 positions; also clears the counts the key kernel and the sort's first
// pass add to (n_clear words) and the error word
__global__ void k_bbox_partial(const double *x, const double *y, const double *z, int n, long long *part,
                               uint32_t *clear, int n_clear, int *err) {
    after_previous();
    if (blockIdx.x == 0 && threadIdx.x == 0) *err = 0;
    Box b;
    b.empty();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b.add(x[i], y[i], z[i]);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_clear; i += gridDim.x * blockDim.x) clear[i] = 0;
    b.reduce();
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) {
            part[blockIdx.x * 6 + d] = b.lo[d];
            part[blockIdx.x * 6 + 3 + d] = b.hi[d];
        }
}

// the root cube from the particle box exactly as or_root_box, and the opening-radius table
__device__ void root_cube(const Box &x, double theta, double *rb) {
    double lo[3], hi[3];
    for (int d = 0; d < 3; ++d) {
        lo[d] = dorder_value(x.lo[d]);
        hi[d] = dorder_value(x.hi[d]);
    }
    double L = 0.0;
    for (int d = 0; d < 3; ++d) {
        const double e = __dsub_rn(hi[d], lo[d]);
        if (e > L) L = e;
    }
    if (!(L > 0.0)) L = 1.0;
    const double half = __dmul_rn(L, 0.50048828125);
    for (int d = 0; d < 3; ++d) rb[d] = __dsub_rn(__dmul_rn(__dadd_rn(lo[d], hi[d]), 0.5), half);
    const double len = __dadd_rn(half, half);
    rb[3] = len;
    rb[4] = __ddiv_rn(2097152.0, len);
    // rc2[l] = (len / 2^l)^2 / theta^2, as or_rcrit_table
    double r = __ddiv_rn(__dmul_rn(len, len), __dmul_rn(theta, theta));
    for (int l = 0; l < MAX_LEVELS; ++l) {
        rb[8 + l] = r;
        r = __dmul_rn(r, 0.25);
    }
}

// one block reduces the partial boxes (min / max are exact in any order), then one thread forms the root cube
__global__ void k_bbox_final(const long long *part, int nb, double theta, double *rb) {
    after_previous();
    Box x;
    x.empty();
    for (int b = threadIdx.x; b < nb; b += blockDim.x)
        for (int d = 0; d < 3; ++d) x.add(d, part[b * 6 + d], part[b * 6 + 3 + d]);
    x.reduce();
    if (threadIdx.x == 0) root_cube(x, theta, rb);
}

// per run: one block per tile reduces its particles' box and clears its digit counts (the key kernel's and the
// first pass's), one block per run the tiles of the run
__global__ void k_bbox_tiles(const double *x, const double *y, const double *z, const int4 *tiles, long long *part,
                             uint32_t *hist, uint32_t *next) {
    after_previous();
    const int4 t = tiles[blockIdx.x];
    Box b;
    b.empty();
    for (int i = t.x + threadIdx.x; i < t.x + t.y; i += blockDim.x) b.add(x[i], y[i], z[i]);
    if (threadIdx.x < 256) {
        hist[(int64_t)blockIdx.x * 256 + threadIdx.x] = 0;
        next[(int64_t)blockIdx.x * 256 + threadIdx.x] = 0;
    }
    b.reduce();
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) {
            part[blockIdx.x * 8 + d] = b.lo[d];
            part[blockIdx.x * 8 + 3 + d] = b.hi[d];
        }
}

// also the run's octree root (level 0: cell r = run r) and, from block 0, an empty meta block
__global__ void k_bbox_runs(const long long *part, const int4 *info, double theta, double *rb, int *meta, int *start,
                            int *count, int *level, int *parent, int *first_child, int *n_child) {
    after_previous();
    const int4 r = info[blockIdx.x];
    Box x;
    x.empty();
    for (int b = r.z + threadIdx.x; b < r.z + r.w; b += blockDim.x)
        for (int d = 0; d < 3; ++d) x.add(d, part[b * 8 + d], part[b * 8 + 3 + d]);
    if (blockIdx.x == 0 && threadIdx.x < META_N) meta[threadIdx.x] = threadIdx.x == 1 ? (int)gridDim.x : 0;
    x.reduce();
    if (threadIdx.x == 0) {
        const int c = blockIdx.x;
        root_cube(x, theta, rb + (int64_t)c * RB_STRIDE);
        start[c] = r.x;
        count[c] = r.y;
        level[c] = 0;
        parent[c] = -1;
        first_child[c] = -1;
        n_child[c] = 0;
    }
}

__device__ __forceinline__ uint64_t spread3(uint64_t v) {
    v &= 0x1fffffULL;
    v = (v | (v << 32)) & 0x1f00000000ffffULL;
    v = (v | (v << 16)) & 0x1f0000ff0000ffULL;
    v = (v | (v << 8)) & 0x100f00f00f00f00fULL;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ULL;
    v = (v | (v << 2)) & 0x1249249249249249ULL;
    return v;
}

// floor of the scaled coordinate, held to the 21 bits of a key (the conversion truncates and takes what is below 0 as 0)
__device__ __forceinline__ uint64_t cell_coord(double v, double lo, double scale) {
    return min(__double2uint_rz(__dmul_rn(__dsub_rn(v, lo), scale)), 2097151u);
}

__device__ __forceinline__ bool not_finite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }

// ---------------------------------------------------------------------------
// LSD radix sort of (key, value), 8 passes of 8 bits over tiles of RS_TILE keys, stable.  With a tile table (tiles
// aligned to run starts; each entry: start, length, first tile of its run, tiles of its run) every run is sorted
// inside its own range; without one the tiles cover [0, n).
//
// What bounds it is latency: a pass moves 24 bytes per key, but it is a chain of dependent launches, and a
// small run's tiles do not fill the chip.  So a pass is one launch where a run has at most RS_DIRECT tiles: the
// digit counts of every tile are in place when the pass starts (the key kernel counts the first digit, each
// pass counts the next digit of its outputs with one atomic per key into the counts of the tile they land
// in; three count arrays rotate, each cleared a pass before it is added to), and every block adds up the counts of
// its run's tiles itself.  Above RS_DIRECT tiles one more launch
// per pass (k_rs_scan) prepares the offsets, since the blocks' own sums grow with the square of the tiles.  Before: a
// histogram, three scan launches and a scatter of 256 threads per pass; keys, sort and permutation of 1M particles
// 0.52 -> 0.38 ms, of 5,003 particles 0.27 -> 0.10 ms.

constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_WKEYS = RS_TILE / RS_WARPS;
constexpr int RS_ROUNDS = RS_WKEYS / 32;

// the lanes with this lane's digit (0..255; 256: none): nine votes (about 100 cycles a warp; __match_any_sync took
// 1,000 with 16 warps on the SM)
__device__ __forceinline__ unsigned same_digit(int d) {
    unsigned m = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 9; ++b) {
        const unsigned v = __ballot_sync(0xffffffffu, (d >> b) & 1);
        m &= (d >> b) & 1 ? v : ~v;
    }
    return m;
}

__device__ __forceinline__ int4 rs_tile(const int4 *tiles, int n, int nb) {
    if (tiles) return tiles[blockIdx.x];
    const int s = blockIdx.x * RS_TILE;
    return make_int4(s, min(RS_TILE, n - s), 0, nb);
}

// keys against the particle's run's root cube, and the counts of their lowest digit added to the tile's (zero on
// entry).  Four blocks per tile, one key per thread: bound by the FP64 pipe (9 instructions a key; 21
// with floor, comparisons and finiteness on it too: keys, sort and permutation of 1M particles 381 against 361 us), so a small run's keys should spread over the SMs.
__global__ void __launch_bounds__(RS_THREADS) k_keys_hist(const double *x, const double *y, const double *z, int n,
                                                          const double *rb, const int *prun, const int4 *tiles, int nb,
                                                          uint64_t *keys, uint32_t *hist, int *err) {
    after_previous();
    __shared__ uint32_t h[256];
    const int t = threadIdx.x, tile = blockIdx.x / RS_SUB, p = blockIdx.x % RS_SUB * RS_THREADS + t;
    if (t < 256) h[t] = 0;
    __syncthreads();
    const int4 tl = tiles ? tiles[tile] : make_int4(tile * RS_TILE, min(RS_TILE, n - tile * RS_TILE), 0, nb);
    if (p < tl.y) {
        const double *q = rb + (prun ? (int64_t)prun[tl.x] * RB_STRIDE : 0);
        const int i = tl.x + p;
        const double px = x[i], py = y[i], pz = z[i];
        if (not_finite(px) || not_finite(py) || not_finite(pz)) atomicOr(err, ERR_NONFINITE);
        const uint64_t key = (spread3(cell_coord(px, q[0], q[4])) << 2) | (spread3(cell_coord(py, q[1], q[4])) << 1) |
                             spread3(cell_coord(pz, q[2], q[4]));
        keys[i] = key;
        atomicAdd(&h[key & 255u], 1u);
    }
    __syncthreads();
    if (t < 256 && h[t]) atomicAdd(&hist[(int64_t)tile * 256 + t], h[t]);
}

// per run (blockIdx.x: only a grid's first extent goes beyond 65,535) and 32 digits (blockIdx.y): off[tile][digit] = keys
// of the digit in the run's earlier tiles, tot[first tile][digit] = in all of them.  Warp w sums the w-th 32nd of the
// tiles, a digit per lane.
__global__ void __launch_bounds__(1024) k_rs_scan(const uint32_t *hist, const int4 *info, uint32_t *off,
                                                  uint32_t *tot) {
    after_previous();
    __shared__ uint32_t s[32][32];
    const int4 r = info[blockIdx.x];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d = blockIdx.y * 32 + lane;
    const int per = (r.w + 31) / 32, t0 = r.z + w * per, t1 = min(r.z + r.w, t0 + per);
    uint32_t v = 0;
#pragma unroll 8
    for (int t = t0; t < t1; ++t) v += hist[(int64_t)t * 256 + d];
    s[w][lane] = v;
    __syncthreads();
    uint32_t base = 0;
    for (int k = 0; k < w; ++k) base += s[k][lane];
    if (w == 31) tot[(int64_t)r.z * 256 + d] = base + v;
#pragma unroll 8
    for (int t = t0; t < t1; ++t) {
        off[(int64_t)t * 256 + d] = base;
        base += hist[(int64_t)t * 256 + d];
    }
}

// One pass over a tile: stable in-tile ranking by warp multisplit (each warp ranks its 128 keys, four rounds of 32
// consecutive keys, by votes against per-warp digit counters, which then become per-digit
// offsets), the tile reordered by digit in shared memory and written out in runs of equal digit.  16 warps of 128
// keys instead of 8 of 256: the rounds of a warp are a serial chain.
__global__ void __launch_bounds__(RS_THREADS, 4) k_rs_scatter(const uint64_t *kin, const uint32_t *vin, uint64_t *kout,
                                                           uint32_t *vout, int n, int shift, const uint32_t *hist,
                                                           uint32_t *next, uint32_t *clear, const uint32_t *off,
                                                           const uint32_t *tot, int nb, const int4 *tiles) {
    after_previous();
    // per-warp digit counts, then per-warp offsets within a digit; then the reordered tile
    __shared__ __align__(8) unsigned char s_buf[RS_TILE * (sizeof(uint64_t) + sizeof(uint32_t))];
    static_assert(sizeof(s_buf) >= RS_WARPS * 256 * sizeof(uint32_t), "the counters fit the tile's buffer");
    uint32_t(*wc)[256] = reinterpret_cast<uint32_t(*)[256]>(s_buf);
    uint64_t *sk = reinterpret_cast<uint64_t *>(s_buf);
    uint32_t *sv = reinterpret_cast<uint32_t *>(sk + RS_TILE);
    __shared__ uint32_t dstart[256];         // first tile position of each digit
    __shared__ uint32_t gofs[256];           // a digit's first output minus its first tile position
    __shared__ uint32_t s_pre[2][256], s_tot[2][256];
    __shared__ uint64_t s_scan[8];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int4 tl = rs_tile(tiles, n, nb);
    const int base = tl.x;
    const int cnt = tl.y;
    const int run0 = tiles ? tiles[tl.z].x : 0;   // the run's first particle
    for (int k = t; k < RS_WARPS * 256; k += RS_THREADS) (&wc[0][0])[k] = 0u;
    if (clear && t < 256) clear[(int64_t)blockIdx.x * 256 + t] = 0;   // what the next pass counts into
    uint64_t key[RS_ROUNDS];
    uint32_t val[RS_ROUNDS], rk[RS_ROUNDS];
    const int p0 = w * RS_WKEYS + lane;   // tile position of the thread's first key
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
        const bool ok = p0 + r * 32 < cnt;
        const int i = base + p0 + r * 32;
        key[r] = ok ? kin[i] : 0ULL;
        val[r] = ok ? (vin ? vin[i] : (uint32_t)i) : 0u;   // the first pass's values are the indices
    }
    auto digit = [&](int r) { return p0 + r * 32 < cnt ? (int)((key[r] >> shift) & 255u) : 256; };   // 256: no item
    {   // the digit's keys in the run's earlier tiles, and in all of them
        const int d = t & 255, half = t >> 8;
        uint32_t pre = 0, all = 0;
        if (off) {
            if (half == 0) {
                pre = off[(int64_t)blockIdx.x * 256 + d];
                all = tot[(int64_t)tl.z * 256 + d];
            }
        } else {
            const int own = blockIdx.x - tl.z;
            const uint32_t *h = hist + (int64_t)tl.z * 256 + d;
#pragma unroll 16
            for (int k = half; k < tl.w; k += 2) {
                const uint32_t v = h[k * 256];
                all += v;
                pre += k < own ? v : 0u;
            }
        }
        s_pre[half][d] = pre;
        s_tot[half][d] = all;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
        const int d = digit(r);
        const unsigned peers = same_digit(d);
        uint32_t b0 = 0;
        if (d < 256) b0 = wc[w][d];
        rk[r] = b0 + (uint32_t)__popc(peers & lt);
        __syncwarp();
        if (d < 256 && lane == __ffs(peers) - 1) wc[w][d] = b0 + (uint32_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        uint32_t c = 0, all = 0;
        if (t < 256) {
            uint32_t v[RS_WARPS];   // all read before the first is written: one trip, not a chain
#pragma unroll
            for (int ww = 0; ww < RS_WARPS; ++ww) v[ww] = wc[ww][t];
#pragma unroll
            for (int ww = 0; ww < RS_WARPS; ++ww) {
                wc[ww][t] = c;
                c += v[ww];
            }
            all = s_tot[0][t] + s_tot[1][t];
        }
        // the digits' starts in the tile and in the run, one scan for both (digits 0..255: warps 0..7)
        uint64_t x = c | (uint64_t)all << 32;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (t < 256 && lane == 31) s_scan[w] = x;
        __syncthreads();
        if (t < 256) {
            for (int k = 0; k < w; ++k) x += s_scan[k];
            const uint32_t ds = (uint32_t)x - c;
            dstart[t] = ds;
            gofs[t] = (uint32_t)run0 + (uint32_t)(x >> 32) - all + s_pre[0][t] + s_pre[1][t] - ds;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r)
        if (digit(r) < 256) rk[r] += dstart[digit(r)] + wc[w][digit(r)];
    __syncthreads();   // the counters have been read: the tile goes over them
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r)
        if (digit(r) < 256) {
            sk[rk[r]] = key[r];
            sv[rk[r]] = val[r];
        }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RS_TILE / RS_THREADS; ++k) {
        const int p = k * RS_THREADS + t;
        if (p < cnt) {
            const uint64_t kk = sk[p];
            const uint32_t g = gofs[(kk >> shift) & 255u] + (uint32_t)p;
            kout[g] = kk;
            vout[g] = sv[p];
            if (next)
                atomicAdd(&next[(int64_t)(tl.z + (int)(g - (uint32_t)run0) / RS_TILE) * 256 +
                                ((kk >> (shift + 8)) & 255u)], 1u);
        }
    }
}

// All passes in one launch, a block per run, for runs of at most RB_KEYS keys: the keys stay in registers and move
// through shared memory, so a pass is a few barriers instead of a launch.  A warp ranks its 256 consecutive keys as
// k_rs_scatter does; the digit counts of the 32 warps become offsets by four threads per digit.  Bound by the one SM's
// issue rate (votes).  Keys to permutation of 3,000 particles 88 -> 61 us, of 5,000 91 -> 75 us;
// from 10,000 on the passes of many blocks are as fast.
constexpr int RB_T = 1024, RB_ITEMS = 8, RB_KEYS = RB_T * RB_ITEMS, RB_W = RB_T / 32;
constexpr size_t RB_SMEM = RB_KEYS * (sizeof(uint64_t) + sizeof(uint16_t)) + RB_W * 256 * sizeof(uint16_t);
__global__ void __launch_bounds__(RB_T) k_rs_block(const uint64_t *kin, uint64_t *kout, uint32_t *vout,
                                                   const int4 *info) {
    after_previous();
    extern __shared__ __align__(16) unsigned char rb_smem[];
    uint64_t *sk = reinterpret_cast<uint64_t *>(rb_smem);
    uint16_t *sv = reinterpret_cast<uint16_t *>(sk + RB_KEYS);
    uint16_t(*wc)[256] = reinterpret_cast<uint16_t(*)[256]>(sv + RB_KEYS);
    __shared__ uint32_t s_scan[RB_W];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int4 run = info[blockIdx.x];
    const int cnt = run.y, p0 = w * (RB_ITEMS * 32) + lane;   // the thread's first position
    const bool busy = w * (RB_ITEMS * 32) < cnt;              // the warp holds keys
    uint64_t key[RB_ITEMS];
    uint32_t val[RB_ITEMS], rk[RB_ITEMS];
#pragma unroll
    for (int r = 0; r < RB_ITEMS; ++r) {
        const int p = p0 + 32 * r;
        key[r] = p < cnt ? kin[run.x + p] : 0ull;
        val[r] = (uint32_t)p;
    }
    for (int shift = 0; shift < 8 * RS_PASSES; shift += 8) {
        auto digit = [&](int r) { return p0 + 32 * r < cnt ? (int)((key[r] >> shift) & 255u) : 256; };   // 256: none
        reinterpret_cast<uint4 *>(wc)[t] = make_uint4(0u, 0u, 0u, 0u);
        static_assert(RB_W * 256 * sizeof(uint16_t) == RB_T * sizeof(uint4), "cleared in one store per thread");
        __syncthreads();
        if (busy) {
#pragma unroll
            for (int r = 0; r < RB_ITEMS; ++r) {
                const int d = digit(r);
                const unsigned peers = same_digit(d);
                uint32_t b = 0;
                if (d < 256) b = wc[w][d];
                rk[r] = b + (uint32_t)__popc(peers & lt);
                __syncwarp();
                if (d < 256 && lane == __ffs(peers) - 1) wc[w][d] = (uint16_t)(b + (uint32_t)__popc(peers));
                __syncwarp();
            }
        }
        __syncthreads();
        {   // thread (digit, quarter of the warps): counts -> first positions
            const int d = t >> 2, w0 = (t & 3) * (RB_W / 4);
            uint32_t c[RB_W / 4], sum = 0;
#pragma unroll
            for (int k = 0; k < RB_W / 4; ++k) {
                c[k] = wc[w0 + k][d];
                sum += c[k];
            }
            uint32_t incl = warp_incl_scan(sum);   // lanes in (digit, quarter) order
            if (lane == 31) s_scan[w] = incl;
            __syncthreads();
            uint32_t base = incl - sum;
            const uint32_t ws = s_scan[lane];
            base += __shfl_sync(0xffffffffu, warp_incl_scan(ws) - ws, w);
#pragma unroll
            for (int k = 0; k < RB_W / 4; ++k) {
                wc[w0 + k][d] = (uint16_t)base;
                base += c[k];
            }
        }
        __syncthreads();
        if (busy) {
#pragma unroll
            for (int r = 0; r < RB_ITEMS; ++r) {
                const int d = digit(r);
                if (d < 256) {
                    const uint32_t q = wc[w][d] + rk[r];
                    sk[q] = key[r];
                    sv[q] = (uint16_t)val[r];
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < RB_ITEMS; ++r) {
            const int p = p0 + 32 * r;
            if (p < cnt) {
                key[r] = sk[p];
                val[r] = sv[p];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RB_ITEMS; ++r) {
        const int p = p0 + 32 * r;
        if (p < cnt) {
            kout[run.x + p] = key[r];
            vout[run.x + p] = (uint32_t)run.x + val[r];
        }
    }
}

// gather all particle arrays through the permutation.  The blocks of one y share the fields out: a thread with all 34
// is a chain of nine rounds of loads, and a small run's threads do not fill the chip.  Nine
// shares against one below 311,000 particles: keys to permutation of 5,000 particles 83 -> 75 us, of 100,000 133 -> 125,
// of 200,000 172 -> 168.
__global__ void k_permute(const double *F, double *F2, int64_t cap, int n, const uint32_t *perm, const int64_t *id,
                          int64_t *id2, const int32_t *slot, int32_t *slot2, const int32_t *mat, int32_t *mat2,
                          const int *prun, int *prun2) {
    after_previous();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int src = (int)perm[k];
    const int per = (SPH_NFIELD + gridDim.y - 1) / gridDim.y, f0 = blockIdx.y * per, f1 = min(SPH_NFIELD, f0 + per);
#pragma unroll 4
    for (int f = f0; f < f1; ++f) F2[(int64_t)f * cap + k] = F[(int64_t)f * cap + src];
    if (blockIdx.y > 0) return;
    id2[k] = id[src];
    slot2[k] = slot[src];
    mat2[k] = mat[src];
    prun2[k] = prun[src];
}

// ---------------------------------------------------------------------------
// octree

// ---------------------------------------------------------------------------
// The octree in one pass over the sorted keys.
//
// A cell of level L >= 1 is a maximal run of particles of one run whose keys share their first L
// octal digits, and it exists exactly when the range of level L - 1 around it (its parent) holds
// more than n_leaf particles (L <= KEY_LEVELS); level 0 holds one root per run.  Sizes shrink
// with the level, so for particle i, with l_i the deepest level whose range around i holds more
// than n_leaf particles, i starts a cell at every level L with d_i < L <= min(l_i + 1, KEY_LEVELS),
// d_i being the number of leading digits i shares with i - 1 (-1 at a run start, where the root
// starts too).  l_i is the largest common-digit count over the windows [j, j + n_leaf] of the run
// that contain i.  Cells are numbered level by level and, inside a level, by start -- the order
// of a level-by-level split in octant order -- so the tree is the same, cell for cell.

constexpr int OT_B = 256;      // particles per block of the one-pass build
constexpr int OT_HALO = 16;    // keys staged beyond each side of a block (windows of n_leaf <= 16 stay in it)

// the leading octal digits (levels 1..KEY_LEVELS of a 63-bit key) two keys share
__device__ __forceinline__ int key_common(uint64_t a, uint64_t b) {
    const uint64_t x = a ^ b;
    return x ? min(KEY_LEVELS, (__clzll((long long)x) - 1) / 3) : KEY_LEVELS;
}

// per particle: the levels at which it starts a cell (lo | hi << 8, empty when hi < lo), and per
// block and level the number of cells starting in the block (cnt[L * n_blocks + block])
__global__ void __launch_bounds__(OT_B) k_cell_levels(int n, int n_leaf, const uint64_t *keys,
                                                      const int *prun, const int4 *info,
                                                      int *lev, int *cnt) {
    after_previous();
    __shared__ uint64_t sk[OT_B + 2 * OT_HALO];
    __shared__ int sc[MAX_LEVELS];
    const int t = threadIdx.x, b0 = blockIdx.x * OT_B, i = b0 + t;
    for (int k = t; k < OT_B + 2 * OT_HALO; k += OT_B) {
        const int g = b0 - OT_HALO + k;
        sk[k] = (g >= 0 && g < n) ? keys[g] : 0ull;
    }
    if (t < MAX_LEVELS) sc[t] = 0;
    __syncthreads();
    auto key_at = [&](int g) { const int k = g - b0 + OT_HALO; return (k >= 0 && k < OT_B + 2 * OT_HALO) ? sk[k] : keys[g]; };
    int lo = 1, hi = 0;
    if (i < n) {
        const int4 ri = info[prun[i]];
        const int rs = ri.x, re = ri.x + ri.y;
        const uint64_t ki = key_at(i);
        const int d = i == rs ? -1 : key_common(key_at(i - 1), ki);
        int ell = -1;
        const int j1 = min(i, re - 1 - n_leaf);
        for (int j = max(rs, i - n_leaf); j <= j1; ++j) ell = max(ell, key_common(key_at(j), key_at(j + n_leaf)));
        lo = d + 1;
        hi = min(ell + 1, KEY_LEVELS);
        if (i == rs) hi = max(hi, 0);
        lev[i] = lo | (hi << 8);
    }
    const int lane = t & 31;
    for (int L = 0; L < MAX_LEVELS; ++L) {
        const unsigned bal = __ballot_sync(0xffffffffu, L >= lo && L <= hi);
        if (lane == 0 && bal) atomicAdd(&sc[L], __popc(bal));
    }
    __syncthreads();
    if (t < MAX_LEVELS) cnt[(int64_t)t * gridDim.x + blockIdx.x] = sc[t];
}

// the cells: cell id = the exclusive scan of the block-and-level counts (level-major) plus the
// rank of the particle among its block's starts at that level; start, count (to the end of the
// run of keys that share its digits), level.  Also the level offsets in meta; more cells than
// the capacity sets ERR_CELL_OVERFLOW and leaves no cells.
__global__ void __launch_bounds__(OT_B) k_cell_emit(int n, int64_t cap, const uint64_t *keys,
                                                    const int *prun, const int4 *info,
                                                    const int *lev, const int *cnt,
                                                    const int *off, int *meta, int *start, int *count,
                                                    int *level) {
    after_previous();
    __shared__ unsigned sb[MAX_LEVELS][OT_B / 32];   // per level and warp: the lanes that start a cell
    const int nb = gridDim.x, t = threadIdx.x, lane = t & 31, warp = t >> 5, i = blockIdx.x * OT_B + t;
    const int64_t last = (int64_t)(MAX_LEVELS - 1) * nb + nb - 1;
    const int64_t total = (int64_t)off[last] + cnt[last];
    const bool overflow = total > cap;
    if (blockIdx.x == 0 && t <= MAX_LEVELS) {
        meta[t] = overflow ? 0 : (t < MAX_LEVELS ? off[(int64_t)t * nb] : (int)total);
        if (t == 0 && overflow) atomicOr(&meta[META_ERR], ERR_CELL_OVERFLOW);
    }
    int lo = 1, hi = 0;
    if (i < n) {
        const int v = lev[i];
        lo = v & 255;
        hi = v >> 8;
    }
#pragma unroll
    for (int L = 0; L < MAX_LEVELS; ++L) {
        const unsigned v = __ballot_sync(0xffffffffu, L >= lo && L <= hi);
        if (lane == 0) sb[L][warp] = v;
    }
    __syncthreads();
    if (overflow || i >= n || hi < lo) return;
    const int4 ri = info[prun[i]];
    const int re = ri.x + ri.y;
    const uint64_t ki = keys[i];
    const unsigned below = (1u << lane) - 1u;
    // The range's end: the first particle of the run past i whose key differs in the first L digits.  Deepest level
    // first, every level from the end of the one below, in steps of 1, 8, 64, ..., then by halving: most cells hold a
    // few particles.  Against a halving of the whole run for every level the tree of 1M particles takes 308 us instead
    // of 328, and as long up to 200,000, where the few cells of the upper levels are the longest chain (steps of 1, 2,
    // 4, ... are 4 us slower there).
    int a = i + 1;
    for (int L = hi; L >= lo; --L) {
        int r = __popc(sb[L][warp] & below);
        for (int w = 0; w < warp; ++w) r += __popc(sb[L][w]);
        const int id = off[(int64_t)L * nb + blockIdx.x] + r;
        int b = re;
        for (int step = 1; a + step - 1 < re; step <<= 3) {
            const int p = a + step - 1;
            if (key_common(keys[p], ki) < L) {
                b = p;
                break;
            }
            a = p + 1;
        }
        while (a < b) {
            const int mid = (a + b) >> 1;
            if (key_common(keys[mid], ki) >= L) a = mid + 1;
            else b = mid;
        }
        start[id] = i;
        count[id] = a - i;
        level[id] = L;
    }
}

// parent, first child and child count of every cell, by binary searches over the starts of the
// levels above and below (each level's cells are sorted by start)
__global__ void k_cell_link(const int *meta, const int *start, const int *count, const int *level, int *parent,
                            int *first_child, int *n_child, int *arrive) {
    after_previous();
    const int nc = meta[MAX_LEVELS];
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
        const int L = level[c], s = start[c], e = s + count[c];
        int p = -1;
        if (L > 0) {   // the last cell of level L - 1 starting at or before s
            int a = meta[L - 1], b = meta[L];
            while (a < b) {
                const int mid = (a + b) >> 1;
                if (start[mid] <= s) a = mid + 1;
                else b = mid;
            }
            p = a - 1;
        }
        int f = -1, nch = 0;
        if (L < KEY_LEVELS) {   // the cells of level L + 1 starting in [s, e)
            const int a0 = meta[L + 1], b0 = meta[L + 2];
            int a = a0, b = b0;
            while (a < b) {
                const int mid = (a + b) >> 1;
                if (start[mid] < s) a = mid + 1;
                else b = mid;
            }
            const int fl = a;
            b = b0;
            while (a < b) {
                const int mid = (a + b) >> 1;
                if (start[mid] < e) a = mid + 1;
                else b = mid;
            }
            nch = a - fl;
            f = nch ? fl : -1;
        }
        parent[c] = p;
        first_child[c] = f;
        n_child[c] = nch;
        arrive[c] = 0;
    }
}

// Moments, boxes and hmax of every cell in one launch, bottom-up.  A thread takes a leaf; then the warp's lanes climb
// together: after a cell is written its lane counts it in at the parent (arrive[], zeroed before the launch), and the
// child that arrives last has its parent's children summed in octant order and climbs on.  The sums and their order are
// those of a level-by-level pass (leaf particles ascending, then children in octant order, one rounding per operation),
// independent of which lane arrives last; no lane waits for another warp (a climb ends at the first parent with
// children still to come, or at the root, after at most KEY_LEVELS steps).  Children written by other threads are read
// through L2 after the fence that orders them before their arrival.
//
// Bound by the FP64 pipe (a warp instruction every 16 cycles and more per SM, however few lanes take part) and, in a
// small run, by the chain of climbs.  So boxes and hmax are found on integer images and rounded once per leaf, not once
// per particle; a climber's four sums run on four lanes, eight climbers at once (a quarter of the additions issued);
// and the centres of mass are divided in k_cell_roles, by full warps.  The tree of 1M / 100,000 / 5,000
// particles 437 / 123 / 90 -> 340 / 107 / 78 us.
__global__ void __launch_bounds__(128)
k_moments_up(const int *meta, const double *x, const double *y, const double *z, const double *m, const double *h,
             const int *start, const int *count, const int *first_child, const int *n_child, const int *parent,
             int *arrive, double4 *mom, float4 *blo, float4 *bhi) {
    after_previous();
    const int nc = meta[MAX_LEVELS], lane = threadIdx.x & 31, q = lane >> 2, comp = lane & 3;
    for (int cw = blockIdx.x * blockDim.x + (threadIdx.x & ~31); cw < nc; cw += gridDim.x * blockDim.x) {
        int c = cw + lane;
        bool on = c < nc && n_child[c] == 0;
        if (on) {
            double ms = 0.0, mx = 0.0, my = 0.0, mz = 0.0;
            long long lo[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, hi[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN}, hm = 0;
            const int s = start[c], e = s + count[c];
            for (int j = s; j < e; ++j) {
                const double mj = m[j], p[3] = {x[j], y[j], z[j]};
                ms = __dadd_rn(ms, mj);
                mx = __dadd_rn(mx, __dmul_rn(mj, p[0]));
                my = __dadd_rn(my, __dmul_rn(mj, p[1]));
                mz = __dadd_rn(mz, __dmul_rn(mj, p[2]));
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const long long k = dorder_key(p[d]);
                    lo[d] = min(lo[d], k);
                    hi[d] = max(hi[d], k);
                }
                const long long hk = __double_as_longlong(h[j]);   // a positive double's order is its integer image's
                if (hk <= __double_as_longlong((double)INFINITY)) hm = max(hm, hk);   // (as fmax: no NaN)
            }
            mom[c] = make_double4(mx, my, mz, ms);
            blo[c] = make_float4(__double2float_rd(dorder_value(lo[0])), __double2float_rd(dorder_value(lo[1])),
                                 __double2float_rd(dorder_value(lo[2])), 0.0f);
            bhi[c] = make_float4(__double2float_ru(dorder_value(hi[0])), __double2float_ru(dorder_value(hi[1])),
                                 __double2float_ru(dorder_value(hi[2])), __double2float_ru(__longlong_as_double(hm)));
        }
        for (int up = 0; up < KEY_LEVELS + 1; ++up) {
            int p = -1, f = 0, nch = 0;
            if (on) p = parent[c];
            on = p >= 0;
            if (on) {
                f = first_child[p];
                nch = n_child[p];
                // release: this cell's moments (written by lanes of this warp, ordered by the barrier below) before its
                // arrival; acquire: every sibling's arrival (and so its moments) before the reads
                asm volatile("fence.acq_rel.gpu;" ::: "memory");
                on = atomicAdd(&arrive[p], 1) == nch - 1;
                asm volatile("fence.acq_rel.gpu;" ::: "memory");
            }
            unsigned left = __ballot_sync(0xffffffffu, on);
            if (!left) break;
            __syncwarp();   // the reads below follow the fences
            c = p;
            while (left) {   // eight climbers at a time, four lanes each
                unsigned rest = left;
                for (int k = 0; k < q && rest; ++k) rest &= rest - 1;
                const int src = rest ? __ffs(rest) - 1 : 0;
                const int pp = __shfl_sync(0xffffffffu, p, src), ff = __shfl_sync(0xffffffffu, f, src),
                          nn = __shfl_sync(0xffffffffu, nch, src);
                if (rest) {
                    const double *mq = reinterpret_cast<const double *>(mom + ff) + comp;
                    double v = 0.0;
                    for (int k = 0; k < nn; ++k) v = __dadd_rn(v, __ldcg(mq + 4 * k));
                    reinterpret_cast<double *>(mom + pp)[comp] = v;
                    float lo = INFINITY, hi = comp == 3 ? 0.0f : -INFINITY;
                    const float *lq = reinterpret_cast<const float *>(blo + ff) + comp;
                    const float *hq = reinterpret_cast<const float *>(bhi + ff) + comp;
                    for (int k = 0; k < nn; ++k) {
                        lo = fminf(lo, __ldcg(lq + 4 * k));
                        hi = fmaxf(hi, __ldcg(hq + 4 * k));
                    }
                    reinterpret_cast<float *>(blo + pp)[comp] = comp == 3 ? 0.0f : lo;
                    reinterpret_cast<float *>(bhi + pp)[comp] = hi;
                }
                for (int k = 0; k < 8 && left; ++k) left &= left - 1;
            }
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// What a cell of the finished tree is to the passes: its packed record, its centre of mass, the walk units it contributes (sph_nbr.cu) and
// whether it is a gravity i-group: at most n_group particles under a parent (or as a root) with more, or a leaf of the
// deepest level with more.  Counts and places come from one scan of both numbers in 64 bits (units low, groups high),
// in the launch sequence of the tree and with its one read of totals.  Latency-bound like the whole tree of a small
// run: as two passes of their own after the tree, with six launches and a read back to the host each, a step of 5,000
// particles took 580 us, this way 523.

// the walk units contributed by cell c; EMIT writes them to out
template <bool EMIT>
__device__ int cell_units(int c, int n_roots, int first, const int *start, int cnt, const int *count,
                          const int *n_child, int nch, int2 *out) {
    const bool root = c < n_roots;   // level 0: one root per run
    int k = 0;
    if (root && cnt <= UNIT) {
        if (EMIT) out[k] = make_int2(start[c], cnt);
        ++k;
    } else if (root && nch == 0) {
        for (int s = 0; s < cnt; s += UNIT) {
            if (EMIT) out[k] = make_int2(start[c] + s, min(UNIT, cnt - s));
            ++k;
        }
    } else if (cnt > UNIT && nch > 0) {
        int us = -1, un = 0;
        for (int q = 0; q < nch; ++q) {
            const int ch = first + q, cc = count[ch];
            if (cc <= UNIT) {
                if (us >= 0 && un + cc <= UNIT) {
                    un += cc;
                } else {
                    if (us >= 0) {
                        if (EMIT) out[k] = make_int2(us, un);
                        ++k;
                    }
                    us = start[ch];
                    un = cc;
                }
            } else {
                if (us >= 0) {
                    if (EMIT) out[k] = make_int2(us, un);
                    ++k;
                }
                us = -1;
                un = 0;
                if (n_child[ch] == 0) {   // a leaf above the unit size (only at the deepest level)
                    for (int s = 0; s < cc; s += UNIT) {
                        if (EMIT) out[k] = make_int2(start[ch] + s, min(UNIT, cc - s));
                        ++k;
                    }
                }
            }
        }
        if (us >= 0) {
            if (EMIT) out[k] = make_int2(us, un);
            ++k;
        }
    }
    return k;
}

__global__ void __launch_bounds__(1024)
k_cell_roles(const int *meta, int n_group, const int *start, const int *count, const int *first_child,
             const int *n_child, const int *parent, const double4 *mom, double4 *com, int4 *cinfo, long long *role,
             long long *part) {
    after_previous();
    const int nc = meta[MAX_LEVELS], n_roots = meta[1];
    const int chunk = (nc + gridDim.x - 1) / gridDim.x;
    const int b1 = min(nc, (int)(blockIdx.x + 1) * chunk);
    long long sum = 0;
    for (int c = blockIdx.x * chunk + threadIdx.x; c < b1; c += blockDim.x) {
        const int cnt = count[c], nch = n_child[c], f = first_child[c], p = parent[c];
        cinfo[c] = make_int4(f, nch, start[c], cnt);
        const double4 q = mom[c];
        com[c] = make_double4(__ddiv_rn(q.x, q.w), __ddiv_rn(q.y, q.w), __ddiv_rn(q.z, q.w), q.w);
        const bool group = cnt <= n_group ? (p < 0 || count[p] > n_group) : nch == 0;
        const int k = cell_units<false>(c, n_roots, f, start, cnt, count, n_child, nch, nullptr);
        const long long v = (long long)k | (long long)group << 32;
        role[c] = v;
        sum += v;
    }
    long long tot;
    block_incl_scan(sum, &tot);
    if (threadIdx.x == 0) part[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(1024)
k_role_emit(const int *meta, const int4 *cinfo, const int *start, const int *count, const int *n_child,
            const long long *role, const long long *part, int2 *units, int *group_cell, long long *total) {
    after_previous();
    const int nc = meta[MAX_LEVELS], n_roots = meta[1];
    const int chunk = (nc + gridDim.x - 1) / gridDim.x;
    const int b0 = blockIdx.x * chunk, b1 = min(nc, b0 + chunk);
    long long all;
    long long base = parts_before(part, &all);
    if (blockIdx.x == 0 && threadIdx.x == 0) *total = all;
    for (int t0 = b0; t0 < b1; t0 += blockDim.x) {
        const int c = t0 + threadIdx.x;
        const long long v = c < b1 ? role[c] : 0;
        long long tot;
        const long long at = base + block_incl_scan(v, &tot) - v;
        if ((int)v) {
            const int4 ci = cinfo[c];
            cell_units<true>(c, n_roots, ci.x, start, ci.w, count, n_child, ci.y, units + (int)at);
        }
        if (v >> 32) group_cell[at >> 32] = c;
        base += tot;
    }
}

__global__ void k_hmax(int l, const int *meta, const double *h, const int *start, const int *count,
                       const int *first_child, const int *n_child, float4 *bhi) {
    const int L0 = meta[l], L1 = meta[l + 1];
    for (int c = L0 + blockIdx.x * blockDim.x + threadIdx.x; c < L1; c += gridDim.x * blockDim.x) {
        float hm = 0.0f;
        const int nch = n_child[c];
        if (nch == 0) {
            for (int j = start[c]; j < start[c] + count[c]; ++j) hm = fmaxf(hm, __double2float_ru(h[j]));
        } else {
            for (int k = 0; k < nch; ++k) hm = fmaxf(hm, bhi[first_child[c] + k].w);
        }
        bhi[c].w = hm;
    }
}

}  // namespace sph

// ---------------------------------------------------------------------------
// host side

template <class T>
static int dalloc(sph_ctx *ctx, T **p, int64_t n) {
    if (*p) cudaFree(*p);
    *p = nullptr;
    ctx->allocations += 1;
    if (n <= 0) n = 1;
    cudaError_t e = cudaMalloc((void **)p, sizeof(T) * (size_t)n);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return sph_fail(ctx, SPH_ERR_OOM, "device allocation of %lld bytes failed: %s",
                        (long long)(sizeof(T) * (size_t)n), cudaGetErrorString(e));
    }
    return SPH_OK;
}

int sph_tree_reserve(sph_ctx *ctx, int64_t n) {
    Tree &t = ctx->tree;
    const int64_t want = 2 * n + 64;
    if (t.cap < want) {
        const int64_t c = want + want / 4;
        SPH_TRY(dalloc(ctx, &t.start, c));
        SPH_TRY(dalloc(ctx, &t.count, c));
        SPH_TRY(dalloc(ctx, &t.level, c));
        SPH_TRY(dalloc(ctx, &t.first_child, c));
        SPH_TRY(dalloc(ctx, &t.n_child, c));
        SPH_TRY(dalloc(ctx, &t.parent, c));
        SPH_TRY(dalloc(ctx, &t.mom, c));
        SPH_TRY(dalloc(ctx, &t.com, c));
        SPH_TRY(dalloc(ctx, &t.blo, c));
        SPH_TRY(dalloc(ctx, &t.bhi, c));
        SPH_TRY(dalloc(ctx, &t.tmp_cnt, c));
        SPH_TRY(dalloc(ctx, &t.tmp_off, c));
        SPH_TRY(dalloc(ctx, &t.tmp_b, 9 * c));
        SPH_TRY(dalloc(ctx, &t.cinfo, c));
        t.cap = c;
    }
    SphSuper &S = ctx->sup;
    if (S.cap_units < n) {   // units and groups hold one particle or more each, and no particle twice
        const int64_t c = n + n / 8 + 64;
        SPH_TRY(dalloc(ctx, &S.units, c));
        SPH_TRY(dalloc(ctx, &S.umark, c));
        SPH_TRY(dalloc(ctx, &S.uoff, c));
        SPH_TRY(dalloc(ctx, &S.uidx, c));
        S.cap_units = c;
    }
    GravLists &G = ctx->grav;
    if (G.cap_groups < n) {
        const int64_t c = n + n / 8 + 64;
        SPH_TRY(dalloc(ctx, &G.group_cell, c));
        SPH_TRY(dalloc(ctx, &G.n_epj, c + 1));
        SPH_TRY(dalloc(ctx, &G.n_spj, c + 1));
        SPH_TRY(dalloc(ctx, &G.off_epj, c + 1));
        SPH_TRY(dalloc(ctx, &G.off_spj, c + 1));
        G.cap_groups = c;
    }
    if (!t.meta) SPH_TRY(dalloc(ctx, &t.meta, META_N));
    if (t.rb_cap < ctx->runs.cap_R) {
        SPH_TRY(dalloc(ctx, &t.rb, (int64_t)RB_STRIDE * ctx->runs.cap_R));
        t.rb_cap = ctx->runs.cap_R;
    }
    Sort &s = ctx->sort;
    if (s.cap < n) {
        const int64_t c = n + n / 8 + 1024;
        SPH_TRY(dalloc(ctx, &s.k0, c));
        SPH_TRY(dalloc(ctx, &s.k1, c));
        SPH_TRY(dalloc(ctx, &s.v0, c));
        SPH_TRY(dalloc(ctx, &s.v1, c));
        s.cap = c;
    }
    if (s.nblocks_cap < ctx->runs.cap_T) {   // tiles of all runs (each run starts a tile)
        SPH_TRY(dalloc(ctx, &s.hist, RS_HISTS * 256 * (int64_t)ctx->runs.cap_T));
        SPH_TRY(dalloc(ctx, &s.hoff, 2 * 256 * (int64_t)ctx->runs.cap_T));
        s.nblocks_cap = ctx->runs.cap_T;
    }
    if (!ctx->scan.part) {
        SPH_TRY(dalloc(ctx, &ctx->scan.part, 2 * SCAN_BLOCKS));   // 32- or 64-bit parts
        SPH_TRY(dalloc(ctx, &ctx->scan.total, 16));
    }
    return SPH_OK;
}

// sorts the keys in sort.k0 (their first digit counted in sort.hist) into ctx->keys, the order into sort.v0
static int radix_sort(sph_ctx *ctx, int n) {
    Sort &s = ctx->sort;
    const int nb = ctx->runs.T;
    const int4 *tiles = ctx->runs.tiles;
    static_assert(RS_TILE == RUN_TILE, "run tiles are radix tiles");
    if (ctx->runs.max_tiles <= RB_KEYS / RUN_TILE) {
        static_assert(RB_KEYS % RUN_TILE == 0, "whole tiles");
        SPH_CUDA(ctx, cudaFuncSetAttribute(k_rs_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RB_SMEM));
        launch_after(true, k_rs_block, ctx->runs.R, RB_T, RB_SMEM, ctx->stream, s.k0, ctx->keys, s.v0, ctx->runs.info);
        ++ctx->launches;
        SPH_CUDA(ctx, cudaGetLastError());
        return SPH_OK;
    }
    const bool scan = ctx->runs.max_tiles > RS_DIRECT;
    const int64_t row = 256 * (int64_t)nb;   // digit counts of one pass
    for (int pass = 0; pass < RS_PASSES; ++pass) {
        const bool odd = pass & 1, last = pass == RS_PASSES - 1;
        uint32_t *hist = s.hist + pass % RS_HISTS * row;
        uint32_t *next = last ? nullptr : s.hist + (pass + 1) % RS_HISTS * row;
        uint32_t *clear = last ? nullptr : s.hist + (pass + 2) % RS_HISTS * row;
        if (scan) {
            launch_after(true, k_rs_scan, dim3(ctx->runs.R, 8), 1024, 0, ctx->stream, hist, ctx->runs.info, s.hoff,
                         s.hoff + row);
            ++ctx->launches;
        }
        launch_after(true, k_rs_scatter, nb, RS_THREADS, 0, ctx->stream, odd ? s.k1 : s.k0,
                     pass == 0 ? nullptr : (odd ? s.v1 : s.v0), last ? ctx->keys : (odd ? s.k0 : s.k1),
                     odd ? s.v0 : s.v1, n, 8 * pass, hist, next, clear, scan ? s.hoff : nullptr, s.hoff + row, nb,
                     tiles); ++ctx->launches;
    }
    SPH_CUDA(ctx, cudaGetLastError());
    return SPH_OK;
}

// the octree over the sorted particles in one pass (k_cell_levels, a scan, k_cell_emit,
// k_cell_link), then the moments bottom-up in one launch, then the cells' records and roles
static int enqueue_tree(sph_ctx *ctx) {
    const int64_t cap = ctx->cap;
    const int n = (int)ctx->n;
    Tree &t = ctx->tree;
    cudaStream_t st = ctx->stream;
    const double *x = FLD(ctx->F, SPH_X, cap), *y = FLD(ctx->F, SPH_Y, cap), *z = FLD(ctx->F, SPH_Z, cap);
    const double *m = FLD(ctx->F, SPH_MASS, cap), *h = FLD(ctx->F, SPH_SMTH, cap);
    const int grid = 2 * ctx->num_sms;
    const int nb = sph_div_up(n, OT_B);
    // scratch: tmp_off the particles' cell levels, tmp_cnt the block-and-level counts, tmp_b their scan
    launch_after(true, k_cell_levels, nb, OT_B, 0, st, n, ctx->cfg.n_leaf, ctx->keys, ctx->runs.prun, ctx->runs.info,
                 t.tmp_off, t.tmp_cnt); ++ctx->launches;
    SPH_TRY(sph_scan_exclusive(ctx, t.tmp_cnt, t.tmp_b, nullptr, MAX_LEVELS * nb, nullptr));
    launch_after(true, k_cell_emit, nb, OT_B, 0, st, n, t.cap, ctx->keys, ctx->runs.prun, ctx->runs.info, t.tmp_off,
                 t.tmp_cnt, t.tmp_b, t.meta, t.start, t.count, t.level); ++ctx->launches;
    // (eight blocks per SM: the searches are chains of loads; with two the tree of 1M particles takes 309 us, not 292)
    launch_after(true, k_cell_link, 4 * grid, 256, 0, st, t.meta, t.start, t.count, t.level, t.parent, t.first_child,
                 t.n_child, t.tmp_cnt);
    ++ctx->launches;
    // moments bottom-up in one launch (tmp_cnt, free again and cleared, counts the arrivals)
    // one thread per cell: the leaves' fences and arrivals all in flight at once
    const int grid_up = (int)std::min<int64_t>((t.cap + 127) / 128, 1 << 16);
    launch_after(true, k_moments_up, grid_up, 128, 0, st, t.meta, x, y, z, m, h, t.start, t.count, t.first_child,
                 t.n_child, t.parent, t.tmp_cnt, t.mom, t.blo, t.bhi); ++ctx->launches;
    // packed records, centres of mass, walk units, gravity groups (tmp_b, free again, as 64-bit numbers)
    static_assert(SCAN_BLOCKS <= SCAN_THREADS, "parts_before");
    // more threads for large trees, whose cells are read once each (tree of 200,000 / 1M particles 107 / 292 -> 101 /
    // 258 us; of 3,000-20,000 2 us slower, of 40,000-100,000 the same)
    const int rt = n < 660 * ctx->num_sms ? SCAN_THREADS : 1024;
    long long *role = (long long *)t.tmp_b, *part = (long long *)ctx->scan.part;
    launch_after(true, k_cell_roles, SCAN_BLOCKS, rt, 0, st, t.meta, ctx->cfg.n_group, t.start, t.count,
                 t.first_child, t.n_child, t.parent, t.mom, t.com, t.cinfo, role, part); ++ctx->launches;
    launch_after(true, k_role_emit, SCAN_BLOCKS, rt, 0, st, t.meta, t.cinfo, t.start, t.count, t.n_child,
                 role, part, ctx->sup.units, ctx->grav.group_cell, (long long *)(t.meta + META_ROLES)); ++ctx->launches;
    SPH_CUDA(ctx, cudaGetLastError());
    return sph_publish(ctx, t.meta, META_N);
}

// the device work of sph_sort_and_build up to the cell-count read: root cubes, keys, the
// segmented radix sort, the permutation (and its host-side buffer swaps), the octree levels,
// the moments.  No host synchronisation and no allocation inside, so it can be captured.
static int enqueue_sort_tree(sph_ctx *ctx) {
    const int n = (int)ctx->n;
    const int64_t cap = ctx->cap;
    double *x = FLD(ctx->F, SPH_X, cap), *y = FLD(ctx->F, SPH_Y, cap), *z = FLD(ctx->F, SPH_Z, cap);
    Tree &t = ctx->tree;
    cudaStream_t st = ctx->stream;
    // root cube of every run (one block per tile, then one per run)
    const Runs &R = ctx->runs;
    uint32_t *hist = ctx->sort.hist, *next = hist + 256 * (int64_t)R.T;
    k_bbox_tiles<<<R.T, 512, 0, st>>>(x, y, z, R.tiles, (long long *)R.part, hist, next); ++ctx->launches;
    launch_after(true, k_bbox_runs, R.R, 256, 0, st, (const long long *)R.part, R.info, ctx->cfg.theta, t.rb, t.meta,
                 t.start, t.count, t.level, t.parent, t.first_child, t.n_child); ++ctx->launches;
    launch_after(true, k_keys_hist, R.T * RS_SUB, RS_THREADS, 0, st, x, y, z, n, t.rb, R.prun, R.tiles, R.T,
                 ctx->sort.k0, ctx->sort.hist, t.meta + META_ERR); ++ctx->launches;
    SPH_TRY(radix_sort(ctx, n));
    // permute the particle state into key order
    const int pb = (int)sph_div_up(n, 256);
    const int py = pb < 8 * ctx->num_sms ? 9 : 1;
    launch_after(true, k_permute, dim3(pb, py), 256, 0, st, ctx->F, ctx->F2, cap, n, ctx->sort.v0, ctx->id, ctx->id2,
                 ctx->slot, ctx->slot2, ctx->mat, ctx->mat2, R.prun, ctx->runs.prun2); ++ctx->launches;
    std::swap(ctx->F, ctx->F2);
    std::swap(ctx->runs.prun, ctx->runs.prun2);
    std::swap(ctx->id, ctx->id2);
    std::swap(ctx->slot, ctx->slot2);
    std::swap(ctx->mat, ctx->mat2);
    SPH_TRY(time_mark(ctx, SEG_SORT));
    return enqueue_tree(ctx);
}

// Everything the captured work depends on: sizes, the buffers that trade places (the permutation swaps the state
// buffers, so a step alternates between two keys), and the number of allocations: a buffer that moved is told from the
// one that was captured even where the others came to lie at their old addresses.
static void graph_key(const sph_ctx *ctx, uintptr_t key[GRAPH_KEY_N]) {
    const Tree &t = ctx->tree;
    const uintptr_t k[GRAPH_KEY_N] = {
        (uintptr_t)ctx->n,         (uintptr_t)ctx->cap,        (uintptr_t)ctx->runs.R,   (uintptr_t)ctx->runs.T,
        (uintptr_t)ctx->F,         (uintptr_t)ctx->F2,         (uintptr_t)ctx->id,       (uintptr_t)ctx->slot,
        (uintptr_t)ctx->mat,       (uintptr_t)ctx->runs.prun,  (uintptr_t)ctx->keys,     (uintptr_t)ctx->sort.k0,
        (uintptr_t)ctx->sort.hist, (uintptr_t)t.start,         (uintptr_t)t.rb,          (uintptr_t)t.cap,
        (uintptr_t)ctx->runs.tiles, (uintptr_t)ctx->runs.part, (uintptr_t)ctx->scan.part, (uintptr_t)t.cinfo,
        (uintptr_t)ctx->cfg.n_leaf, (uintptr_t)(ctx->runs.max_tiles > RS_DIRECT) +
            (uintptr_t)(ctx->runs.max_tiles > RB_KEYS / RUN_TILE), (uintptr_t)ctx->cfg.n_group,
        (uintptr_t)ctx->sup.units, (uintptr_t)ctx->grav.group_cell, ctx->allocations};
    for (int i = 0; i < GRAPH_KEY_N; ++i) key[i] = k[i];
}

// replays the captured sort + octree for this key (capturing it the first time)
static int sort_tree_graph(sph_ctx *ctx) {
    uintptr_t key[GRAPH_KEY_N];
    graph_key(ctx, key);
    TreeGraph *g = nullptr;
    for (TreeGraph &c : ctx->tree_graphs)
        if (c.exec && std::equal(key, key + GRAPH_KEY_N, c.key)) g = &c;
    if (g) {
        // the captured work's host side: the buffer swaps of the permutation
        std::swap(ctx->F, ctx->F2);
        std::swap(ctx->runs.prun, ctx->runs.prun2);
        std::swap(ctx->id, ctx->id2);
        std::swap(ctx->slot, ctx->slot2);
        std::swap(ctx->mat, ctx->mat2);
        ctx->launches += g->launches;
        ctx->graph_replays += 1;
    } else {
        g = &ctx->tree_graphs[ctx->graph_next];
        ctx->graph_next = (ctx->graph_next + 1) % (int)(sizeof(ctx->tree_graphs) / sizeof(ctx->tree_graphs[0]));
        if (g->exec) cudaGraphExecDestroy(g->exec);
        g->exec = nullptr;
        cudaGraph_t graph = nullptr;
        const int64_t l0 = ctx->launches;
        SPH_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        const int rc = enqueue_sort_tree(ctx);
        const cudaError_t ce = cudaStreamEndCapture(ctx->stream, &graph);
        if (rc != SPH_OK) {
            if (graph) cudaGraphDestroy(graph);
            return rc;
        }
        if (ce != cudaSuccess) {
            cudaGetLastError();
            return sph_fail(ctx, SPH_ERR_CUDA, "capture of the octree build failed: %s", cudaGetErrorString(ce));
        }
        const cudaError_t ie = cudaGraphInstantiate(&g->exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ie != cudaSuccess) {
            g->exec = nullptr;
            cudaGetLastError();
            return sph_fail(ctx, SPH_ERR_CUDA, "instantiation of the octree build failed: %s", cudaGetErrorString(ie));
        }
        std::copy(key, key + GRAPH_KEY_N, g->key);
        g->launches = ctx->launches - l0;
        ctx->graph_captures += 1;
    }
    SPH_CUDA(ctx, cudaGraphLaunch(g->exec, ctx->stream));
    return SPH_OK;
}

int sph_sort_and_build(sph_ctx *ctx) {
    const int n = (int)ctx->n;
    Tree &t = ctx->tree;
    SPH_TRY(sph_tree_reserve(ctx, n));
    cudaStream_t st = ctx->stream;
    // With event timing on the work is launched directly (its segments are timed); otherwise the
    // 14 to 29 launches of the sort and the octree (by the sort's route) replay as one CUDA graph.
    if (ctx->timing || !ctx->use_graphs) SPH_TRY(enqueue_sort_tree(ctx));
    else SPH_TRY(sort_tree_graph(ctx));
    SPH_TRY(time_mark(ctx, SEG_TREE));
    // the counts and the error word, published at the end of the tree's launches; the packs run behind them
    const int *hs = (int *)ctx->host_scalars;
    SPH_CUDA(ctx, cudaEventRecord(ctx->tree_done, st));
    SPH_TRY(sph_nbr_prepare(ctx));
    SPH_CUDA(ctx, cudaEventSynchronize(ctx->tree_done));
    if (hs[META_ERR] & ERR_NONFINITE) return sph_fail(ctx, SPH_ERR_NONFINITE, "non-finite particle position");
    if (hs[META_ERR] & ERR_CELL_OVERFLOW) return sph_fail(ctx, SPH_ERR_CAPACITY, "octree cell capacity exceeded");
    t.n_cell_host = hs[MAX_LEVELS];
    int depth = 0;
    for (int l = 0; l < MAX_LEVELS; ++l)
        if (hs[l + 1] > hs[l]) depth = l;
    t.depth = depth;
    ctx->sup.n_units = hs[META_ROLES];
    ctx->grav.ng = hs[META_ROLES + 1];
    ctx->grav.valid = false;
    ctx->grav.counts_valid = false;
    return SPH_OK;
}

int sph_tree_refresh_hmax(sph_ctx *ctx, const double *h) {
    Tree &t = ctx->tree;
    const int grid = 2 * ctx->num_sms;
    for (int l = t.depth; l >= 0; --l)
        k_hmax<<<grid, 128, 0, ctx->stream>>>(l, t.meta, h, t.start, t.count, t.first_child, t.n_child, t.bhi); ++ctx->launches;
    SPH_CUDA(ctx, cudaGetLastError());
    return SPH_OK;
}
