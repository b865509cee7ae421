// Device building blocks shared by the uniform-batch morphology kernels
// (morphology.cu) and the ragged-batch ones (ragged.cu): operator traits, the
// reference's border mapping, and the separable min/max of one staged 2-D
// tile.
#pragma once

#include <cmath>

#include "tm_common.cuh"

namespace tmc {
namespace morph {

}  // namespace morph

// 3-D items on shared-memory tiles (stencil3d.cu).  Sets *done = false and
// returns TM_OK, launching nothing, when the element does not fit the tile
// kernel (more than 1024 active taps, or a tile beyond shared memory).
template <typename T, bool MAX>
int stencil3d_uniform(const T *in, T *out, int64_t batch, const int64_t *shape, const float *structure,
                      const uint8_t *footprint, const int64_t *sshape, const int64_t *origin, int mode, float cval,
                      cudaStream_t s, bool *done);

namespace morph {

// ---------------------------------------------------------------- op traits
template <typename T, bool MAX>
struct MorphOp;

template <>
struct MorphOp<float, false> {  // grey erosion
    __device__ __forceinline__ static float identity() { return INFINITY; }
    __device__ __forceinline__ static float combine(float a, float b) { return fminf(a, b); }
    __device__ __forceinline__ static float apply(float v, float s) { return v - s; }
};
template <>
struct MorphOp<float, true> {  // grey dilation
    __device__ __forceinline__ static float identity() { return -INFINITY; }
    __device__ __forceinline__ static float combine(float a, float b) { return fmaxf(a, b); }
    __device__ __forceinline__ static float apply(float v, float s) { return v + s; }
};
template <>
struct MorphOp<uint8_t, false> {  // binary erosion (AND)
    __device__ __forceinline__ static uint8_t identity() { return 1; }
    __device__ __forceinline__ static uint8_t combine(uint8_t a, uint8_t b) { return a < b ? a : b; }
    __device__ __forceinline__ static uint8_t apply(uint8_t v, float) { return v; }
};
template <>
struct MorphOp<uint8_t, true> {  // binary dilation (OR)
    __device__ __forceinline__ static uint8_t identity() { return 0; }
    __device__ __forceinline__ static uint8_t combine(uint8_t a, uint8_t b) { return a > b ? a : b; }
    __device__ __forceinline__ static uint8_t apply(uint8_t v, float) { return v; }
};

// Border mapping (torchmorph/csrc/grey_kernel.cu:63-97).  Returns -1 when
// the constant value must be used.
__host__ __device__ __forceinline__ int map_coord(int c, int n, int mode) {
    if ((unsigned)c < (unsigned)n) return c;
    switch (mode) {
    case TM_MODE_NEAREST:
        return c < 0 ? 0 : n - 1;
    case TM_MODE_REFLECT: {
        int period = 2 * n;
        int r = c % period;
        if (r < 0) r += period;
        return r >= n ? period - 1 - r : r;
    }
    case TM_MODE_MIRROR: {
        int period = 2 * (n - 1);
        if (period <= 0) return 0;
        int r = c % period;
        if (r < 0) r += period;
        return r >= n ? period - r : r;
    }
    case TM_MODE_WRAP: {
        int r = c % n;
        return r < 0 ? r + n : r;
    }
    default:
        return -1;
    }
}

// ------------------------------------------------------------ flat 2-D tile
constexpr int kTileW = 128;
constexpr int kTileH = 32;
constexpr int kFlatThreads = 256;
constexpr int kRun = 8;
// Row pitches, in elements, of the row-pass buffer and of a staged tile for a window of kw
// columns (room for full runs past the last column).  An odd number of 4-byte words: threads
// on the same column of consecutive rows then hit different banks, of bytes as of floats
// (binary 45 x 45 of 4 x 2048^2 160 us with an odd number of bytes, 1 x 66 86 us).
template <typename T>
constexpr int kRowsPitch = sizeof(T) == 4 ? kTileW + 1 : kTileW + 4;
template <typename T>
__host__ __device__ inline int stage_pitch(int kw) {
    constexpr int per_word = 4 / (int)sizeof(T);
    return (((kTileW + kw - 1 + (kRun - 1) + per_word - 1) / per_word) | 1) * per_word;
}

// Shared memory of a tile for a window of runtime size: the staged tile and, for windows of more
// than one column, the row pass.
template <typename T>
inline size_t flat_smem(int kh, int kw) {
    return (size_t)(kTileH + kh - 1) * (stage_pitch<T>(kw) + (kw > 1 ? kRowsPitch<T> : 0)) * sizeof(T);
}

// Stage rows [gy0, gy0 + RH) x columns [gx0, gx0 + RW) of one H x W image into shared
// memory (row stride ld), mapping out-of-image coordinates with the border mode.  Warp w
// takes rows w, w + 8, ...; a lane maps its NC columns of a chunk once for all rows
// and issues the loads of 2 rows before it stores any, so border tiles cost what
// interior ones do and a warp keeps 2 NC loads in flight.
template <typename T, int NC>
__device__ __forceinline__ void stage_columns(const T *__restrict__ src, int H, int W, int gy0, int gx0, int RH,
                                              int RW, int ld, int mode, T cval, T *tile) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int nwarps = kFlatThreads / 32, RB = 2;
    for (int cb = lane; cb < RW; cb += 32 * NC) {
        int mx[NC];  // -1: the constant; columns past the region repeat one inside it, unstored
#pragma unroll
        for (int j = 0; j < NC; j++) mx[j] = map_coord(gx0 + min(cb + 32 * j, RW - 1), W, mode);
        const int last = (RW - 1 - cb) / 32;  // chunk columns 0 .. last are inside the region
        for (int rb = warp; rb < RH; rb += nwarps * RB) {
            T v[RB][NC];
#pragma unroll
            for (int k = 0; k < RB; k++) {
                const int my = map_coord(gy0 + min(rb + nwarps * k, RH - 1), H, mode);
                const T *row = src + (int64_t)max(my, 0) * W;
#pragma unroll
                for (int j = 0; j < NC; j++) v[k][j] = my >= 0 && mx[j] >= 0 ? row[mx[j]] : cval;
            }
#pragma unroll
            for (int k = 0; k < RB; k++) {
                const int r = rb + nwarps * k;
                if (r >= RH) break;
                T *t = tile + r * ld + cb;
#pragma unroll
                for (int j = 0; j < NC; j++)
                    if (j <= last) t[32 * j] = v[k][j];
            }
        }
    }
}

template <typename T>
__device__ __forceinline__ void stage_tile(const T *__restrict__ src, int H, int W, int gy0, int gx0, int RH, int RW,
                                           int ld, int mode, T cval, T *tile) {
    if constexpr (sizeof(T) == 1) {
        // one chunk up to 192 columns (binary 9 x 45 of 4 x 2048^2: 48 us, 62 with two; floats lose
        // more by the second form than they gain: 4 x 4 36 -> 41 us)
        if (RW > 160 && RW <= 192) {
            stage_columns<T, 6>(src, H, W, gy0, gx0, RH, RW, ld, mode, cval, tile);
            return;
        }
    }
    stage_columns<T, 5>(src, H, W, gy0, gx0, RH, RW, ld, mode, cval, tile);
}

struct Flat2DParams {
    int H, W;        // item size (1-D items use H = 1)
    int kh, kw;      // window
    int lo_y, lo_x;  // window of output (y, x) covers rows y+lo_y .. y+lo_y+kh-1
    int mode;
    int64_t batch;
    float cval;
    float sval;  // constant structure value (flat footprint)
    int y_first;  // first row of a launch (0 but for items taller than a grid)
    FastDiv d_rows;  // divides by kTileH + kh - 1
};


// One run of RUN consecutive outputs of a 1-D sliding window of width k >= RUN over
// src[0 .. RUN + k - 2] (src elements `step` apart in shared memory), by the van Herk/
// Gil-Werman split: every window of the run contains the block [RUN - 1, k - 1]; the left
// part is a suffix of [j, RUN - 2], the right part a prefix of [k, j + k - 1].  Every
// element of the span is read once (k + RUN - 1 reads, about k + 3 RUN combines).
template <typename T, bool MAX, int RUN>
__device__ __forceinline__ void van_herk_run(const T *src, int step, int k, T *res) {
    using Op = MorphOp<T, MAX>;
    T mid = src[(RUN - 1) * step];
    for (int t = RUN; t < k; t++) mid = Op::combine(mid, src[t * step]);
    T suf[RUN];
    suf[RUN - 1] = mid;
#pragma unroll
    for (int j = RUN - 2; j >= 0; j--) suf[j] = Op::combine(src[j * step], suf[j + 1]);
    res[0] = suf[0];
    T pre = src[k * step];
#pragma unroll
    for (int j = 1; j < RUN; j++) {
        res[j] = Op::combine(suf[j], pre);
        if (j + 1 < RUN) pre = Op::combine(pre, src[(k + j) * step]);
    }
}

// kRun outputs from the fewest reads: one run of 8, two of 4 for windows of 4 .. 7, four of 2 below
// (white top-hat 2 x 2 of 4 x 2048^2: 144 us tap by tap, 108 so; 128 in the kernel before).
template <typename T, bool MAX>
__device__ __forceinline__ void window_run(const T *src, int step, int k, T *res) {
    using Op = MorphOp<T, MAX>;
    if (k >= kRun) {
        van_herk_run<T, MAX, kRun>(src, step, k, res);
    } else if (k >= kRun / 2) {
        van_herk_run<T, MAX, kRun / 2>(src, step, k, res);
        van_herk_run<T, MAX, kRun / 2>(src + (kRun / 2) * step, step, k, res + kRun / 2);
    } else if (k > 1) {
#pragma unroll
        for (int j = 0; j < kRun; j += 2) van_herk_run<T, MAX, 2>(src + j * step, step, k, res + j);
    } else {
#pragma unroll
        for (int j = 0; j < kRun; j++) res[j] = src[j * step];
    }
}

// Row pass then column pass of one staged tile: `tile` points at the first
// input column the tile needs (row stride ld), `rows` receives the row-pass
// result (RH x kTileW at pitch kRowsPitch); outputs go to dst at (y0.., x0..).
// (RH rows of the region and the columns inside the item are computed; d_rows divides by RH.)
template <typename T, bool MAX>
__device__ __forceinline__ void flat_tile_compute(const T *tile, int ld, T *rows, const Flat2DParams &p, T *dst,
                                                  int x0, int y0) {
    const int RH = kTileH + p.kh - 1;
    const int cols = min(kTileW, p.W - x0), outs = min(kTileH, p.H - y0);
    const int runs = (cols + kRun - 1) / kRun;
    // (every row of the region, also below the outputs of a tile at the item's end: the
    // work unit's division stays a constant one; those rows are stale and unused)
    constexpr int kPitch = kRowsPitch<T>;
    auto column_pass = [&](const T *from, int pitch) {
        for (int w = threadIdx.x; w < kTileW * (kTileH / kRun); w += kFlatThreads) {
            const int c = w % kTileW, r = (w / kTileW) * kRun;
            if (c >= cols || r >= outs) continue;
            // kTileH is a multiple of kRun, so the run reads rows
            // r .. r + kRun + kh - 2 <= RH - 1: always inside the row buffer
            T res[kRun];
            window_run<T, MAX>(from + r * pitch + c, pitch, p.kh, res);
            T *o = dst + (int64_t)(y0 + r) * p.W + x0 + c;
#pragma unroll
            for (int j = 0; j < kRun; j++, o += p.W)
                if (r + j < outs) __stcs(o, MorphOp<T, MAX>::apply(res[j], p.sval));
        }
    };
    if (p.kw == 1) {  // no row pass (and no buffer for one: 81 x 1 of 4 x 2048^2 207 us with them, 72 without)
        column_pass(tile, ld);
        return;
    }
    for (int w = threadIdx.x; w < RH * runs; w += kFlatThreads) {
        // consecutive threads take the same run of consecutive rows
        const int u = (int)fdiv(w, p.d_rows), r = w - u * RH;
        if (r >= outs + p.kh - 1) continue;
        const int c = kRun * u;
        T res[kRun];
        window_run<T, MAX>(tile + r * ld + c, 1, p.kw, res);
#pragma unroll
        for (int j = 0; j < kRun; j++) rows[r * kPitch + c + j] = res[j];
    }
    __syncthreads();
    column_pass(rows, kPitch);
}

// Compile-time window (KH x KW): each thread walks down one column of the
// tile (two threads per column, 16 output rows each), computes every input
// row's horizontal minimum/maximum once and keeps the last KH of them in
// registers, so one pass produces the outputs without a row buffer.
// Adjacent lanes own adjacent columns: conflict-free shared-memory reads and
// 128-byte global stores.
template <typename T, bool MAX, int KH, int KW>
__device__ __forceinline__ void flat_tile_walk(const T *tile, int ld, const Flat2DParams &p, T *dst, int x0,
                                               int y0) {
    using Op = MorphOp<T, MAX>;
    constexpr int kSegRows = kTileH / 2;
    const int c = threadIdx.x % kTileW, seg = threadIdx.x / kTileW;
    const int gx = x0 + c;
    if (gx >= p.W) return;
    const int r0 = seg * kSegRows;
    const T *src = tile + r0 * ld + c;
    T h[KH];
#pragma unroll
    for (int k = 0; k < KH - 1; k++) {
        T acc = src[k * ld];
#pragma unroll
        for (int t = 1; t < KW; t++) acc = Op::combine(acc, src[k * ld + t]);
        h[k] = acc;
    }
    T *o = dst + (int64_t)(y0 + r0) * p.W + gx;
    const int rows_left = p.H - (y0 + r0);
#pragma unroll 4
    for (int r = 0; r < kSegRows; r++) {
        const T *row = src + (r + KH - 1) * ld;
        T acc = row[0];
#pragma unroll
        for (int t = 1; t < KW; t++) acc = Op::combine(acc, row[t]);
        h[KH - 1] = acc;
        T v = h[0];
#pragma unroll
        for (int k = 1; k < KH; k++) v = Op::combine(v, h[k]);
        if (r < rows_left) __stcs(o + (int64_t)r * p.W, Op::apply(v, p.sval));  // outputs: streaming stores
#pragma unroll
        for (int k = 0; k < KH - 1; k++) h[k] = h[k + 1];
    }
}

template <typename T, bool MAX, int KH, int KW>
__device__ __forceinline__ void tile_compute(const T *tile, int ld, T *rows, const Flat2DParams &p, T *dst, int x0,
                                             int y0) {
    if constexpr (KH > 0)
        flat_tile_walk<T, MAX, KH, KW>(tile, ld, p, dst, x0, y0);
    else
        flat_tile_compute<T, MAX>(tile, ld, rows, p, dst, x0, y0);
}

}  // namespace morph
}  // namespace tmc
