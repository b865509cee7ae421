// FP32 Sinkhorn for batches of histogram pairs sharing one (d, d) matrix
// (GB300, sm_103a): the plain CUDA-core path next to the tensor-core solver.
//
// Every half-step of every pair is one contraction with the shared matrix:
//   scaling form  out[b,i] = num[b,i] / (sum_j K[i,j] s[b,j] + 1e-12)
//   log form      out[b,i] = num[b,i] - LSE_j(-M[i,j]/eps + s[b,j])
// (u-update: num = a | log a, matrix K | M, s = v | log v; v-update: b,
// K^T | M^T, u), the contract of the reference's fused iterations
// (torchmorph/csrc/ot_kernel.cu:188-283, torchmorph/optimal_transport.py:
// 71-125): u first, +1e-12 in the scaling denominators, -inf wherever every
// term of a log-sum-exp is -inf.
//
// Design.  Both forms are GEMM-shaped: the (d x d) matrix is shared by the n
// pairs, so a CTA owns a tile of 128 matrix rows x TB pairs and reuses every
// staged matrix entry for all TB pairs (the reference streams the matrix once
// per group of 8 pairs).  Matrix and scaling tiles are staged in shared
// memory 16 columns at a time (register prefetch of the next chunk, one
// barrier per chunk); each thread accumulates 8 rows x TB/16 pairs.  The log
// form works in base 2 (entries pre-scaled by log2(e) when staged) with a
// running maximum per output, rescaled only when a group of 4 terms raises it,
// so a term costs one add, one subtract and one ex2.
//
// The whole iteration loop is ONE cooperative persistent launch: all CTAs
// are co-resident and meet at bounded grid barriers between half-steps, so a
// solve of any length costs one launch (the reference enqueues two kernels
// per iteration and replays captured chunks of them).  With a threshold the
// u-update of every check_every-th iteration also sums the L1 row-marginal
// residual |a_i - u_i (K v)_i| of the plan that iteration started from (per
// 128-row block, in fixed order), the next phase reduces it per pair, and
// all CTAs stop together once every pair is at or below the threshold -- no
// host round trip.  A barrier wait that exceeds its poll budget records
// TM_DEV_ERR_TIMEOUT in the device status word and makes every CTA leave.
#include <algorithm>
#include <atomic>
#include <cmath>

#include "tm_tma.cuh"

namespace tmc {
namespace {

constexpr int kSkThreads = 256;
constexpr int kSkRows = 128;       // matrix rows per tile
constexpr int kSkChunk = 16;       // contraction columns staged per step
constexpr int kSkPitch = kSkChunk + 4;  // padded row of a staged tile (floats)
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kNoMax = -3.0e38f;  // running-maximum start (below every finite term)

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Cost of the d points 0, 1, ..., d - 1 on a line, the reference's default
// cost (build_cost_matrix((d,), p) for p = 1 or 2): |i - j|, exact in float32.
// A NULL cost matrix selects it; entries are then computed where they are
// used and no (d, d) matrix is ever stored or read.
__device__ __forceinline__ float line_cost(int i, int j) { return (float)(i > j ? i - j : j - i); }

struct SkControl {
    unsigned barrier_count;
    unsigned barrier_gen;
    int abort;
    int iterations;  // iterations completed by the last launch
    int pad[60];
};
static_assert(sizeof(SkControl) == 256, "control block is 256 bytes");

struct SkArgs {
    const float *num_u, *num_v;  // a, b (scaling) or log a, log b (log form)
    const float *mat, *mat_t;    // K, K^T or M, M^T (row-major d x d)
    float *u, *v;                // scalings or log-scalings, updated in place
    int n, d;
    float mscale;                // log form: -log2(e) / eps applied to staged matrix entries
    float inv_eps;               // scaling form with the line cost: K = exp(-|i - j| * inv_eps)
    int max_iter, check_every;   // check_every = 0: no residual checks
    float threshold;
    double *partial;             // [row blocks][n] residual partial sums
    double *err;                 // [n] residual of the last check
    int *notconv;                // [checks] set when some pair is above the threshold
    SkControl *ctl;
    int *status;
    long long spin_limit;
    bool vec;                    // d % 4 == 0 and 16-byte aligned operands: float4 staging
    bool paired;                 // mat_t is the transpose of mat (the caller's own matrices need not be)
};


struct SkStage {
    float mat[2][kSkRows * kSkPitch];
    float sc[2][64 * kSkPitch];
};

// One tile of one half-step: rows [i0, i0 + 128) of the matrix, pairs
// [b0, b0 + 16 * MB).  Thread layout: lane % 16 = row group tr (rows tr + 16 r,
// r < 8), lane / 16 + 2 * warp = pair group tb (pairs tb + 16 m, m < MB), so a
// staged matrix row is read by 16 lanes at 20-float pitch (two wavefronts) and
// a scaling row is broadcast to 16 lanes; outputs are written 16 consecutive
// rows at a time.
template <bool LOG, int MB>
__device__ void sk_tile(const SkArgs &A, SkStage &st, int i0, int b0, const float *__restrict__ num,
                        const float *__restrict__ mat, const float *scale, float *out, double *partial_row) {
    constexpr int TB = 16 * MB;
    const int n = A.n, d = A.d;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tr = lane & 15, tb = (lane >> 4) + 2 * warp;
    // entries beyond the matrix or the batch contribute nothing: a zero kernel
    // weight (scaling form), an infinite cost and a -inf log-scaling (log form;
    // the cost is scaled by the negative mscale when staged)
    const float fill = LOG ? INFINITY : 0.0f;
    const float sfill = LOG ? -INFINITY : 0.0f;
    const float mscale = A.mscale;

    // staging assignment: matrix tile 128 x 16 = 512 float4 (two per thread),
    // scaling tile TB x 16 = TB * 4 float4 (threads < TB * 4)
    float4 pm[2], ps;
    auto load = [&](int j0) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int f = tid + h * kSkThreads;
            const int row = f >> 2, q = f & 3;
            const int i = i0 + row, j = j0 + 4 * q;
            float4 x = make_float4(fill, fill, fill, fill);
            if (!mat) {  // the line cost (symmetric: the same for K and K^T)
                if (i < d) {
                    float c[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        c[e] = fill;
                        if (j + e < d) c[e] = LOG ? line_cost(i, j + e) : expf(-line_cost(i, j + e) * A.inv_eps);
                    }
                    x = make_float4(c[0], c[1], c[2], c[3]);
                }
            } else if (i < d) {
                const float *src = mat + (size_t)i * d + j;
                if (A.vec) {
                    if (j < d) x = *reinterpret_cast<const float4 *>(src);
                } else {
                    if (j < d) x.x = src[0];
                    if (j + 1 < d) x.y = src[1];
                    if (j + 2 < d) x.z = src[2];
                    if (j + 3 < d) x.w = src[3];
                }
            }
            pm[h] = x;
        }
        ps = make_float4(sfill, sfill, sfill, sfill);
        if (tid < TB * 4) {
            const int p = tid >> 2, q = tid & 3;
            const int b = b0 + p, j = j0 + 4 * q;
            if (b < n) {
                // u and v are rewritten by other CTAs during the launch: L2 loads, never L1
                const float *src = scale + (size_t)b * d + j;
                if (A.vec) {
                    if (j < d) ps = __ldcg(reinterpret_cast<const float4 *>(src));
                } else {
                    if (j < d) ps.x = __ldcg(src);
                    if (j + 1 < d) ps.y = __ldcg(src + 1);
                    if (j + 2 < d) ps.z = __ldcg(src + 2);
                    if (j + 3 < d) ps.w = __ldcg(src + 3);
                }
            }
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int f = tid + h * kSkThreads;
            float4 x = pm[h];
            if (LOG) {  // base-2 exponent of the matrix term; -inf stays -inf
                x.x *= mscale;
                x.y *= mscale;
                x.z *= mscale;
                x.w *= mscale;
            }
            *reinterpret_cast<float4 *>(&st.mat[buf][(f >> 2) * kSkPitch + 4 * (f & 3)]) = x;
        }
        if (tid < TB * 4) {
            float4 x = ps;
            if (LOG) {
                x.x *= kLog2e;
                x.y *= kLog2e;
                x.z *= kLog2e;
                x.w *= kLog2e;
            }
            *reinterpret_cast<float4 *>(&st.sc[buf][(tid >> 2) * kSkPitch + 4 * (tid & 3)]) = x;
        }
    };

    float acc[8][MB];  // scaling: sum; log: scaled sum
    float mx[LOG ? 8 : 1][LOG ? MB : 1];
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
        for (int m = 0; m < MB; m++) {
            acc[r][m] = 0.0f;
            if (LOG) mx[LOG ? r : 0][LOG ? m : 0] = kNoMax;
        }

    const int nchunks = (d + kSkChunk - 1) / kSkChunk;
    load(0);
    __syncthreads();  // the previous tile's readers are done with buffer 0
    store(0);
    __syncthreads();
    for (int c = 0; c < nchunks; c++) {
        const int buf = c & 1;
        if (c + 1 < nchunks) load((c + 1) * kSkChunk);
        const float *ms = st.mat[buf];
        const float *ss = st.sc[buf];
#pragma unroll
        for (int jq = 0; jq < kSkChunk / 4; jq++) {
            float4 sv[MB];
#pragma unroll
            for (int m = 0; m < MB; m++)
                sv[m] = *reinterpret_cast<const float4 *>(&ss[(tb + 16 * m) * kSkPitch + 4 * jq]);
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const float4 kv = *reinterpret_cast<const float4 *>(&ms[(tr + 16 * r) * kSkPitch + 4 * jq]);
#pragma unroll
                for (int m = 0; m < MB; m++) {
                    if (!LOG) {
                        float a = acc[r][m];
                        a = fmaf(kv.x, sv[m].x, a);
                        a = fmaf(kv.y, sv[m].y, a);
                        a = fmaf(kv.z, sv[m].z, a);
                        a = fmaf(kv.w, sv[m].w, a);
                        acc[r][m] = a;
                    } else {
                        const float z0 = kv.x + sv[m].x, z1 = kv.y + sv[m].y;
                        const float z2 = kv.z + sv[m].z, z3 = kv.w + sv[m].w;
                        const float cm = fmaxf(fmaxf(z0, z1), fmaxf(z2, z3));
                        float &M = mx[LOG ? r : 0][LOG ? m : 0];
                        if (cm > M) {  // rare after the first chunks: rescale the sum
                            acc[r][m] *= ex2(M - cm);
                            M = cm;
                        }
                        acc[r][m] += (ex2(z0 - M) + ex2(z1 - M)) + (ex2(z2 - M) + ex2(z3 - M));
                    }
                }
            }
        }
        if (c + 1 < nchunks) store(buf ^ 1);
        __syncthreads();
    }

    // epilogue: outputs, and the residual partial of the plan this half-step starts from
#pragma unroll
    for (int m = 0; m < MB; m++) {
        const int b = b0 + tb + 16 * m;
        float res = 0.0f;
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = i0 + tr + 16 * r;
            if (b < n && i < d) {
                const size_t idx = (size_t)b * d + i;
                const float nu = num[idx];
                float o;
                if (!LOG) {
                    if (partial_row) res += fabsf(nu - __ldcg(out + idx) * acc[r][m]);
                    o = nu / (acc[r][m] + 1e-12f);
                } else {
                    const float M = mx[LOG ? r : 0][LOG ? m : 0];
                    const bool none = !(M > kNoMax);  // every term was -inf
                    const float lse2 = M + log2f(acc[r][m]);
                    if (partial_row) {
                        const float old = __ldcg(out + idx);
                        const float plan_row = none ? 0.0f : ex2(fmaf(old, kLog2e, lse2));
                        res += fabsf(ex2(nu * kLog2e) - plan_row);
                    }
                    o = none ? -INFINITY : nu - lse2 * kLn2;
                }
                out[idx] = o;
            }
        }
        if (partial_row) {
            // the 16 lanes of this half-warp hold the 128 rows of pair b
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) res += __shfl_xor_sync(0xffffffffu, res, o);
            if (tr == 0 && b < n) partial_row[b] = (double)res;
        }
    }
}

template <bool LOG, int MB>
__global__ void __launch_bounds__(kSkThreads, 2) sk_solve_kernel(SkArgs A) {
    __shared__ __align__(16) SkStage st;
    constexpr int TB = 16 * MB;
    const int row_blocks = (A.d + kSkRows - 1) / kSkRows;
    const int pair_blocks = (A.n + TB - 1) / TB;
    const int tiles = row_blocks * pair_blocks;
    int check = 0;
    int it = 0;
    for (; it < A.max_iter; it++) {
        const bool checking = A.check_every > 0 && (it + 1) % A.check_every == 0;
        // u-update (tiles ordered row block major: CTAs running at once share matrix rows in L2)
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            const int rb = t / pair_blocks, pb = t % pair_blocks;
            sk_tile<LOG, MB>(A, st, rb * kSkRows, pb * TB, A.num_u, A.mat, A.v, A.u,
                             checking ? A.partial + (size_t)rb * A.n : nullptr);
        }
        if (!grid_barrier_bounded(A.ctl, gridDim.x, A.status, A.spin_limit)) return;
        if (checking) {  // per-pair residual sums, one warp per pair, fixed order
            const int warps = gridDim.x * (kSkThreads / 32);
            const int lane = threadIdx.x & 31;
            for (int b = blockIdx.x * (kSkThreads / 32) + (threadIdx.x >> 5); b < A.n; b += warps) {
                double s = 0.0;
                for (int r = lane; r < row_blocks; r += 32) s += __ldcg(A.partial + (size_t)r * A.n + b);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) {
                    A.err[b] = s;
                    if (!(s <= (double)A.threshold)) atomicOr(&A.notconv[check], 1);
                }
            }
        }
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            const int rb = t / pair_blocks, pb = t % pair_blocks;
            sk_tile<LOG, MB>(A, st, rb * kSkRows, pb * TB, A.num_v, A.mat_t, A.u, A.v, nullptr);
        }
        if (!grid_barrier_bounded(A.ctl, gridDim.x, A.status, A.spin_limit)) return;
        if (checking) {
            const bool stop = *((volatile int *)&A.notconv[check]) == 0;
            check++;
            if (stop) {
                it++;
                break;
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) A.ctl->iterations = it;
}

// ----------------------------------------------------- resident row slabs
// The tile kernel above gives a CTA 128 matrix rows, so a problem of a few
// hundred points keeps a handful of SMs busy and every half-step waits for
// their 128-row contractions.  Where the matrix is small, sk_slab_kernel cuts
// it into slabs of 8 to 32 rows instead: CTA (c, g) keeps rows [c R, c R + R) of K
// and of K^T in its shared memory for the whole solve and updates the pairs of
// group g, one CTA per SM, so a half-step reads only the other side's scalings
// (from L2) and costs one barrier among the CTAs of the group (pairs never
// meet; with a stopping test the decision is common and so is the barrier).
//
// Bound: the barrier and the L2 round trips of the scalings, not arithmetic
// (16 pairs x 784 points: 0.2 us of FMAs per CTA and half-step, 5.4 us taken).
// (In the scaling form sk_cluster_kernel below takes the problems that fit its clusters.)
// Measured per iteration, tile kernel -> slabs (GB300, whole solves of 50): scaling
// form 16 x 784 88 -> 10.9 us, 16 x 1600 172 -> 26 us, 48 x 64 20 -> 8 us, 256 x 784
// 136 -> 71 us; log form 16 x 784 127 -> 18 us, 31 x 1600 870 -> 115 us.
//
// W = ceil(d / 128) warps (at most 8) form a set that takes one tile of 8 rows x PT
// pairs at a time, the 8 / W sets of a CTA different tiles.  A thread owns 4
// columns (8 above 1024 points, V = 2: W = ceil(d / 256)) for all 8 rows and PT
// pairs: the scalings go from L2 straight into its registers.  The 8 x PT partial sums of
// the set's threads are reduced by transposing butterflies (62 shuffles for 64
// sums) and across the warps in shared memory; then one thread per (row, pair)
// finishes the output.  The log form takes the maximum of every (row, pair) in a
// first pass and sums 2^(z - max) in a second.
constexpr int kSlabRows = 8;       // rows per tile
constexpr int kSlabMaxCtas = 160;  // CTAs of a launch (residual partials are sized for these)
constexpr int kSlabWarps = kSkThreads / 32;
constexpr int kSlabMaxGroups = 60;  // arrival counters in the control block
constexpr int64_t kOneWaveMaxPairs = 1 << 14;  // larger batches are the tile kernel's by any of the rules below

template <bool LOG, int V>
struct SlabTile {
    static constexpr int PT = LOG || V > 1 ? 4 : 8;  // pairs per tile
    static constexpr int N = kSlabRows * PT;         // sums per thread
    static constexpr int kCols = 128 * V;            // columns per warp
};

struct SlabShape {
    int rows;    // R: rows per CTA, a multiple of kSlabRows
    int ctas;    // CTAs of a group
    int groups;  // pair groups
    int pairs;   // pairs per group
    int pitch;   // floats per slab row (d rounded up to 4)
    size_t smem;
};

// Arrival counter barrier: the count only grows, so a CTA arrives with one add and
// waits for `target` (modulo 2^32).  Bounded like grid_barrier_bounded.  One thread:
__device__ inline bool grid_arrive_wait(SkControl *ctl, int *counter, unsigned target, int *status,
                                        long long spin_limit) {
    __threadfence();
    atomicAdd(counter, 1);
    bool ok = true;
    long long polls = 0;
    volatile int *abort = &ctl->abort;
    for (;;) {
        unsigned cnt;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cnt) : "l"(counter) : "memory");
        if ((int)(cnt - target) >= 0) break;
        if (++polls > spin_limit || ((polls & 63) == 0 && *abort)) {
            ok = false;
            break;
        }
    }
    if (!ok) {
        atomicExch(&ctl->abort, 1);
        if (status) atomicExch(status, TM_DEV_ERR_TIMEOUT);
    }
    __threadfence();
    return ok;
}

__device__ inline bool slab_barrier(SkControl *ctl, int *counter, unsigned target, int *status,
                                    long long spin_limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) s_ok = grid_arrive_wait(ctl, counter, target, status, spin_limit);
    __syncthreads();
    return s_ok != 0;
}

// Barrier of the `threads` threads of warp set `set` (hardware barriers 1 .. 8).
__device__ __forceinline__ void set_sync(int set, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(set + 1), "r"(threads) : "memory");
}

// v[0..N) of every lane -> sums (or maxima) over the 32 lanes: lane l is left with
// entries l (N / 32) + k, k < N / 32, in v[k].
template <int N, bool MAX>
__device__ __forceinline__ void transpose_reduce(float (&v)[N]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16, half = N / 2; o > 0; o >>= 1, half >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < half; k++) {
            const float send = up ? v[k] : v[k + half], keep = up ? v[k + half] : v[k];
            const float got = __shfl_xor_sync(0xffffffffu, send, o);
            v[k] = MAX ? fmaxf(keep, got) : keep + got;
        }
    }
}

// One half-step of the CTA's rows: out[b, i] for i in [i0, i0 + R), b in [b_lo, b_hi).
template <bool LOG, int V>
__device__ __forceinline__ void slab_half(const SkArgs &A, const SlabShape &sh, int i0, int b_lo, int b_hi,
                                          const float *slab, float *red_all, const float *__restrict__ num,
                                          const float *scale, float *out, double *partial_row) {
    constexpr int PT = SlabTile<LOG, V>::PT, N = SlabTile<LOG, V>::N, COLS = SlabTile<LOG, V>::kCols;
    const int d = A.d, pitch = sh.pitch;
    const int W = (d + COLS - 1) / COLS, sets = kSlabWarps / W, set = (threadIdx.x >> 5) / W;
    if (set >= sets) return;  // left-over warps (they meet the others at the next block barrier)
    const int st = threadIdx.x - set * W * 32, warp = st >> 5, lane = st & 31, nthr = W * 32;
    float *red = red_all + (size_t)set * (W + 1) * N;  // [W][N] partial sums, then N maxima
    const float sfill = LOG ? -INFINITY : 0.0f;
    // this thread's columns: 4 (st + v W 32) .. + 3, v < V
    auto load_scale = [&](float4(&x)[PT][V], int b0) {
#pragma unroll
        for (int p = 0; p < PT; p++)
#pragma unroll
            for (int v = 0; v < V; v++) {
                const int j = 4 * (st + v * nthr);
                float4 q = make_float4(sfill, sfill, sfill, sfill);
                if (b0 + p < b_hi && j < d) {
                    // u and v are rewritten by other CTAs during the launch: L2 loads, never L1
                    const float *src = scale + (size_t)(b0 + p) * d + j;
                    if (A.vec) {
                        q = __ldcg(reinterpret_cast<const float4 *>(src));
                    } else {
                        q.x = __ldcg(src);
                        if (j + 1 < d) q.y = __ldcg(src + 1);
                        if (j + 2 < d) q.z = __ldcg(src + 2);
                        if (j + 3 < d) q.w = __ldcg(src + 3);
                    }
                }
                x[p][v] = q;
            }
    };
    const int ntiles = (b_hi - b_lo + PT - 1) / PT;
    float4 sv[PT][V], nx[PT][V];
    if (!LOG && set < ntiles) load_scale(nx, b_lo + set * PT);
    for (int t = set; t < ntiles; t += sets) {
        const int b0 = b_lo + t * PT;
        if (LOG) load_scale(nx, b0);
#pragma unroll
        for (int p = 0; p < PT; p++)
#pragma unroll
            for (int v = 0; v < V; v++) {
                sv[p][v] = nx[p][v];
                if (LOG) {
                    sv[p][v].x *= kLog2e;
                    sv[p][v].y *= kLog2e;
                    sv[p][v].z *= kLog2e;
                    sv[p][v].w *= kLog2e;
                }
            }
        if (!LOG && t + sets < ntiles) load_scale(nx, b0 + sets * PT);  // in flight behind this tile
        for (int r0 = 0; r0 < sh.rows && i0 + r0 < d; r0 += kSlabRows) {
            // the outputs this thread finishes: entry e = 8 p + r of the tile
            constexpr int kOwn = N / 32;  // at least 32 threads
            float nu[kOwn], old[kOwn];
#pragma unroll
            for (int k = 0; k < kOwn; k++) {
                const int e = st + k * nthr, i = i0 + r0 + (e & 7), b = b0 + (e >> 3);
                const bool own = e < N && i < d && b < b_hi;
                nu[k] = own ? num[(size_t)b * d + i] : 0.0f;
                old[k] = own && partial_row ? __ldcg(out + (size_t)b * d + i) : 0.0f;
            }
            const float *rows = slab + (size_t)r0 * pitch;
            float acc[N];
            if (LOG) {
#pragma unroll
                for (int k = 0; k < N; k++) acc[k] = kNoMax;
#pragma unroll
                for (int v = 0; v < V; v++) {
                    // (at most one turn: the loop keeps the row loads of one v from being moved
                    // across the others', which would not fit in registers)
                    for (int j = 4 * (st + v * nthr); j < pitch; j += 4 * V * nthr)
#pragma unroll
                    for (int r = 0; r < kSlabRows; r++) {
                        const float4 kv = *reinterpret_cast<const float4 *>(rows + (size_t)r * pitch + j);
#pragma unroll
                        for (int p = 0; p < PT; p++)
                            acc[p * kSlabRows + r] =
                                fmaxf(acc[p * kSlabRows + r], fmaxf(fmaxf(kv.x + sv[p][v].x, kv.y + sv[p][v].y),
                                                                    fmaxf(kv.z + sv[p][v].z, kv.w + sv[p][v].w)));
                    }
                }
                transpose_reduce<N, true>(acc);
#pragma unroll
                for (int k = 0; k < N / 32; k++) red[warp * N + lane * (N / 32) + k] = acc[k];
                set_sync(set, nthr);
                if (st < N) {
                    float m = kNoMax;
                    for (int w = 0; w < W; w++) m = fmaxf(m, red[w * N + st]);
                    red[W * N + st] = m;
                }
                set_sync(set, nthr);
            }
#pragma unroll
            for (int k = 0; k < N; k++) acc[k] = 0.0f;
#pragma unroll
            for (int v = 0; v < V; v++) {
                for (int j = 4 * (st + v * nthr); j < pitch; j += 4 * V * nthr)
#pragma unroll
                for (int r = 0; r < kSlabRows; r++) {
                    const float4 kv = *reinterpret_cast<const float4 *>(rows + (size_t)r * pitch + j);
#pragma unroll
                    for (int p = 0; p < PT; p++) {
                        float x = acc[p * kSlabRows + r];
                        if (!LOG) {
                            x = fmaf(kv.x, sv[p][v].x, x);
                            x = fmaf(kv.y, sv[p][v].y, x);
                            x = fmaf(kv.z, sv[p][v].z, x);
                            x = fmaf(kv.w, sv[p][v].w, x);
                        } else {
                            const float M = red[W * N + p * kSlabRows + r];
                            x += (ex2((kv.x + sv[p][v].x) - M) + ex2((kv.y + sv[p][v].y) - M)) +
                                 (ex2((kv.z + sv[p][v].z) - M) + ex2((kv.w + sv[p][v].w) - M));
                        }
                        acc[p * kSlabRows + r] = x;
                    }
                }
            }
            transpose_reduce<N, false>(acc);
#pragma unroll
            for (int k = 0; k < N / 32; k++) red[warp * N + lane * (N / 32) + k] = acc[k];
            set_sync(set, nthr);
#pragma unroll
            for (int k = 0; k < kOwn; k++) {
                const int e = st + k * nthr, i = i0 + r0 + (e & 7), b = b0 + (e >> 3);
                if (e >= N) break;  // N is a multiple of 32: whole warps leave
                float sum = 0.0f, res = 0.0f;
                for (int w = 0; w < W; w++) sum += red[w * N + e];
                const bool own = i < d && b < b_hi;
                if (own) {
                    float o;
                    if (!LOG) {
                        if (partial_row) res = fabsf(nu[k] - old[k] * sum);
                        o = nu[k] / (sum + 1e-12f);
                    } else {
                        const float M = red[W * N + e];
                        const bool none = !(M > kNoMax);  // every term was -inf
                        const float lse2 = M + log2f(sum);
                        if (partial_row) {
                            const float plan_row = none ? 0.0f : ex2(fmaf(old[k], kLog2e, lse2));
                            res = fabsf(ex2(nu[k] * kLog2e) - plan_row);
                        }
                        o = none ? -INFINITY : nu[k] - lse2 * kLn2;
                    }
                    out[(size_t)b * d + i] = o;
                }
                if (partial_row) {  // 8 adjacent lanes hold the tile's rows of one pair
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) res += __shfl_xor_sync(0xffffffffu, res, o);
                    if ((e & 7) == 0 && own) {
                        if (r0 == 0) partial_row[b] = (double)res;
                        else partial_row[b] += (double)res;  // this thread's own earlier store
                    }
                }
            }
            set_sync(set, nthr);  // the partial sums are rewritten by the next tile
        }
    }
}

template <bool LOG, int V>
__global__ void __launch_bounds__(kSkThreads, 1) sk_slab_kernel(SkArgs A, SlabShape sh) {
    extern __shared__ __align__(16) float slab_smem[];
    const int rows = sh.rows, pitch = sh.pitch;
    float *su = slab_smem;                              // rows of K (u-update)
    float *sv = slab_smem + (size_t)rows * pitch;       // rows of K^T (v-update)
    float *red = slab_smem + (size_t)2 * rows * pitch;  // partial sums and maxima
    const int slab = blockIdx.x % sh.ctas, group = blockIdx.x / sh.ctas;
    const int i0 = slab * rows, d = A.d;
    const int b_lo = group * sh.pairs, b_hi = min(A.n, b_lo + sh.pairs);
    const float fill = LOG ? -INFINITY : 0.0f;
    for (int r = 0; r < rows; r++) {
        const int i = i0 + r;
        for (int j = threadIdx.x; j < pitch; j += kSkThreads) {
            float x = fill, y = fill;
            if (i < d && j < d) {
                if (A.mat) {
                    x = A.mat[(size_t)i * d + j];
                    y = A.mat_t[(size_t)i * d + j];
                } else {  // the line cost is symmetric
                    x = LOG ? line_cost(i, j) : expf(-line_cost(i, j) * A.inv_eps);
                    y = x;
                }
                if (LOG) {
                    x *= A.mscale;
                    y *= A.mscale;
                }
            }
            su[r * pitch + j] = x;
            sv[r * pitch + j] = y;
        }
    }
    __syncthreads();
    // with a stopping test every CTA takes part in one decision; without, a group is on its own
    const bool common = A.check_every > 0;
    int *counter = &A.ctl->pad[common ? 0 : group];
    const unsigned arrivals = common ? gridDim.x : (unsigned)sh.ctas;
    unsigned target = 0;
    int check = 0, it = 0;
    for (; it < A.max_iter; it++) {
        const bool checking = common && (it + 1) % A.check_every == 0;
        slab_half<LOG, V>(A, sh, i0, b_lo, b_hi, su, red, A.num_u, A.v, A.u,
                       checking ? A.partial + (size_t)slab * A.n : nullptr);
        if (!slab_barrier(A.ctl, counter, target += arrivals, A.status, A.spin_limit)) return;
        if (checking) {  // per-pair residual sums, one warp per pair, fixed order
            const int warps = gridDim.x * kSlabWarps;
            const int lane = threadIdx.x & 31;
            for (int b = blockIdx.x * kSlabWarps + (threadIdx.x >> 5); b < A.n; b += warps) {
                double s = 0.0;
                for (int r = lane; r < sh.ctas; r += 32) s += __ldcg(A.partial + (size_t)r * A.n + b);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) {
                    A.err[b] = s;
                    if (!(s <= (double)A.threshold)) atomicOr(&A.notconv[check], 1);
                }
            }
        }
        slab_half<LOG, V>(A, sh, i0, b_lo, b_hi, sv, red, A.num_v, A.u, A.v, nullptr);
        if (!slab_barrier(A.ctl, counter, target += arrivals, A.status, A.spin_limit)) return;
        if (checking) {
            const bool stop = *((volatile int *)&A.notconv[check]) == 0;
            check++;
            if (stop) {
                it++;
                break;
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) A.ctl->iterations = it;
}

// The shape the slab kernel runs an (n, d) problem in, or false where the tile kernel
// keeps it.  Of R = 8 .. 32 rows per CTA that fit in shared memory the one with the
// fewest tile rounds per half-step wins, on a tie the larger (fewer CTAs meet at a
// barrier, each scaling is read by fewer of them).  A round costs about 1.4 us (log
// form 2 us, 2.8 us above 1024 points), the tile kernel 0.085 (0.28) us per column and
// wave: many pairs over many points stay with it (scaling 256 x 1700: 282 us an
// iteration against 352 in slabs; log 512 x 1200: 714 against 895).
template <bool LOG, int V>
inline bool slab_shape(int64_t n, int64_t d, int sms, SlabShape *out) {
    constexpr int PT = SlabTile<LOG, V>::PT, N = SlabTile<LOG, V>::N;
    const int64_t W = ceil_div(d, (int64_t)SlabTile<LOG, V>::kCols), sets = kSlabWarps / W;
    if (W > kSlabWarps || n > kOneWaveMaxPairs) return false;
    int64_t best = 0;
    for (int rows = kSlabRows; rows <= 4 * kSlabRows; rows += kSlabRows) {
        SlabShape s;
        s.rows = rows;
        s.ctas = (int)ceil_div(d, (int64_t)rows);
        s.pitch = (int)((d + 3) & ~(int64_t)3);
        s.smem = ((size_t)2 * rows * s.pitch + (size_t)sets * (W + 1) * N) * sizeof(float);
        if (s.ctas > sms || s.smem > (size_t)224 * 1024) continue;
        const int64_t tiles = ceil_div(n, PT);
        int64_t groups = std::min<int64_t>(std::min<int64_t>(sms / s.ctas, tiles), kSlabMaxGroups);
        const int64_t tiles_per = ceil_div(tiles, groups);
        s.groups = (int)ceil_div(tiles, tiles_per);
        s.pairs = (int)(tiles_per * PT);
        const int64_t rounds = (rows / kSlabRows) * ceil_div(tiles_per, sets);
        if (best == 0 || rounds <= best) {
            best = rounds;
            *out = s;
        }
    }
    // a round against d columns of the tile kernel's waves
    const int64_t waves = ceil_div(ceil_div(d, kSkRows) * ceil_div(n, 64), 2 * (int64_t)sms);
    return best > 0 && best * (LOG ? (V > 1 ? 10 : 7) : 16) < d * waves;
}

// ------------------------------------------------------ a cluster per few pairs
// Pairs never meet, so the iterations need no barrier wider than the CTAs that share a pair's
// matrix.  sk_cluster_kernel gives PT pairs to a cluster of C CTAs that keep K among them: CTA
// r holds rows [r R, r R + R), R = d / C rounded up to a
// multiple of 4, in shared memory and both updates use them.
//   u: warps take rows, lanes columns; u of the own rows stays in the CTA.
//   v: every thread sums its 4 columns over every S-th of the own rows; the S sums are added
//      and stored in the shared memory of the CTA that owns the columns; after a cluster
//      barrier the owner adds the C of them, divides, and stores v to all CTAs, followed by
//      the second barrier.
// So an iteration reads the slab twice from shared memory and costs two cluster barriers; no
// scaling goes through L2.  A stopping test adds one barrier of the whole grid per check.
//
// Bound: shared memory (two reads of the slab, 1.6 us for 784 points in clusters of 12) and
// what separates the phases: two cluster barriers, the sums' shuffles and remote stores
// (2 us at any size).  Measured per iteration, slabs -> clusters (GB300): 16 pairs x 64 points
// 7.1 -> 2.1 us, 16 x 256 6.7 -> 2.7, 64 x 256 6.9 -> 3.0, 16 x 400 6.6 -> 3.7, 32 x 512 7.0 ->
// 4.6, 1 x 784 6.5 -> 4.8, 16 x 784 9.2 -> 5.8 us (8 clusters of 12; of 16 only 7 fit on the
// device).  4-byte remote stores of the partial sums, all S splits of them: 16 x 784 8.8 us;
// 8 warps without row guards on the loads: 9.7.
constexpr int kClThreads = 512;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClRows = 8;    // row sums of a warp at a time
constexpr int kClMaxCtas = 16;
constexpr size_t kClMaxSmem = 227 * 1024;

struct ClusterShape {
    int pairs;  // PT
    int ctas;   // C
    int rows;   // R
    int pitch;  // floats per row (d rounded up to 4)
    int split;  // S
    int clusters;
    size_t smem;
};

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(const void *p, int rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, float x) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(x) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t addr, float4 x) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w)
                 : "memory");
}

// v[0..N) of every lane -> sums over the 32 lanes: lane l is left with entry l / (32 / N)
template <int N>
__device__ __forceinline__ float lane_reduce(float (&v)[N]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int half = N / 2; half > 0; half >>= 1) {
        const int o = half * (32 / N);
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < half; k++) {
            const float send = up ? v[k] : v[k + half], keep = up ? v[k + half] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    float x = v[0];
#pragma unroll
    for (int o = 32 / N / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

template <int PT>
__global__ void __launch_bounds__(kClThreads, 1) sk_cluster_kernel(SkArgs A, ClusterShape sh) {
    extern __shared__ __align__(16) float cl_smem[];
    __shared__ double s_res[kClWarps][PT];
    __shared__ float s_ok;
    constexpr int N = kClRows * PT, kShare = 32 / N;
    const int rows = sh.rows, pitch = sh.pitch;
    float *K = cl_smem;                         // [rows][pitch]
    float *vs = K + (size_t)rows * pitch;       // v: [PT][pitch]
    float *us = vs + PT * pitch;                // u of the own rows: [rows][PT]
    float *recv = us + PT * rows;               // partial sums of the own columns: [C][PT][rows]
    float *more = recv + sh.ctas * PT * rows;   // partial sums of splits 2 .. S - 1: [PT][pitch] each
    const int d = A.d, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x % sh.ctas, b0 = blockIdx.x / sh.ctas * PT;
    const int i0 = rank * rows, own = max(0, min(rows, d - i0));
    for (int r = 0; r < own; r++)
        for (int j = tid; j < pitch; j += kClThreads) {
            float x = 0.0f;
            if (j < d) x = A.mat ? A.mat[(size_t)(i0 + r) * d + j] : expf(-line_cost(i0 + r, j) * A.inv_eps);
            K[r * pitch + j] = x;
        }
    for (int k = tid; k < PT * pitch; k += kClThreads) {
        const int p = k / pitch, j = k - p * pitch;
        vs[k] = b0 + p < A.n && j < d ? A.v[(size_t)(b0 + p) * d + j] : 0.0f;
    }
    // v: this thread's columns 4 tc .. + 3, rows ts, ts + S, ...; where the sums go
    const int lanes_v = kClThreads / sh.split, ts = tid / lanes_v, tc = tid - ts * lanes_v;
    const bool v_sum = 4 * tc < pitch;
    const int to_cta = v_sum ? 4 * tc / rows : 0;  // (R is a multiple of 4)
    const uint32_t to = cluster_addr(recv + rank * PT * rows + (4 * tc - to_cta * rows), to_cta);
    float *local = ts == 1 ? vs : more + (ts - 2) * PT * pitch;  // (v is not read between the u sums and its update)
    // ... and what it finishes: v of (pair vp, own column vi)
    const int vp = tid / rows, vi = tid - vp * rows;
    const bool v_own = vp < PT && b0 + vp < A.n && vi < own;
    const size_t v_at = (size_t)(b0 + vp) * d + i0 + vi;
    const float nv = v_own ? A.num_v[v_at] : 0.0f;
    // u: of pair up, rows warp + 16 (8 g + uk)
    const int ue = lane / kShare, up = ue / kClRows, uk = ue % kClRows;
    unsigned arrived = 0;
    int it = 0, check = 0;
    cluster_sync();  // K and v are in place, and every CTA runs
    for (; it < A.max_iter; it++) {
        const bool last = it + 1 == A.max_iter, checking = A.check_every > 0 && (it + 1) % A.check_every == 0;
        float res = 0.0f;
        for (int r0 = warp; r0 < rows; r0 += kClWarps * kClRows) {
            const int ur = r0 + kClWarps * uk;
            const bool u_own = b0 + up < A.n && ur < own;
            const size_t u_at = (size_t)(b0 + up) * d + i0 + ur;
            const float nu = u_own ? __ldg(A.num_u + u_at) : 0.0f;
            float acc[N];
#pragma unroll
            for (int k = 0; k < N; k++) acc[k] = 0.0f;
            for (int j = 4 * lane; j < pitch; j += 128) {
                float4 x[PT], kv[kClRows];
#pragma unroll
                for (int p = 0; p < PT; p++) x[p] = *reinterpret_cast<const float4 *>(vs + p * pitch + j);
#pragma unroll
                for (int k = 0; k < kClRows; k++) {
                    kv[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (r0 + kClWarps * k < own) kv[k] = *reinterpret_cast<const float4 *>(K + (r0 + kClWarps * k) * pitch + j);
                }
#pragma unroll
                for (int k = 0; k < kClRows; k++) {
                    if (r0 + kClWarps * k >= own) break;
#pragma unroll
                    for (int p = 0; p < PT; p++) {
                        float a = acc[p * kClRows + k];
                        a = fmaf(kv[k].x, x[p].x, a);
                        a = fmaf(kv[k].y, x[p].y, a);
                        a = fmaf(kv[k].z, x[p].z, a);
                        acc[p * kClRows + k] = fmaf(kv[k].w, x[p].w, a);
                    }
                }
            }
            const float sum = lane_reduce<N>(acc);
            const float u = nu / (sum + 1e-12f);
            if (lane % kShare == 0 && ur < own) {
                if (checking && u_own) res += fabsf(nu - (it ? us[ur * PT + up] : A.u[u_at]) * sum);
                us[ur * PT + up] = u_own ? u : 0.0f;
            }
        }
        if (checking) {  // residual of the plan this iteration starts from
#pragma unroll
            for (int o = 4 * kShare; o >= kShare; o >>= 1) res += __shfl_xor_sync(0xffffffffu, res, o);
            if (lane % (kClRows * kShare) == 0) s_res[warp][lane / (kClRows * kShare)] = (double)res;
        }
        __syncthreads();
        if (checking && tid < PT && b0 + tid < A.n) {
            double s = 0.0;
            for (int w = 0; w < kClWarps; w++) s += s_res[w][tid];
            __stcg(A.partial + (size_t)((check & 1) * kClMaxCtas + rank) * A.n + b0 + tid, s);
            __threadfence();
        }
        float4 sum[PT];
#pragma unroll
        for (int p = 0; p < PT; p++) sum[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (v_sum) {
#pragma unroll 8
            for (int r = ts; r < own; r += sh.split) {
                const float4 kv = *reinterpret_cast<const float4 *>(K + r * pitch + 4 * tc);
#pragma unroll
                for (int p = 0; p < PT; p++) {
                    const float x = us[r * PT + p];
                    sum[p].x = fmaf(kv.x, x, sum[p].x);
                    sum[p].y = fmaf(kv.y, x, sum[p].y);
                    sum[p].z = fmaf(kv.z, x, sum[p].z);
                    sum[p].w = fmaf(kv.w, x, sum[p].w);
                }
            }
            if (ts > 0)
#pragma unroll
                for (int p = 0; p < PT; p++) *reinterpret_cast<float4 *>(local + p * pitch + 4 * tc) = sum[p];
        }
        if (sh.split > 1) {
            __syncthreads();
            if (v_sum && ts == 0)
                for (int q = 1; q < sh.split; q++)
#pragma unroll
                    for (int p = 0; p < PT; p++) {
                        const float *from = q == 1 ? vs : more + (q - 2) * PT * pitch;
                        const float4 x = *reinterpret_cast<const float4 *>(from + p * pitch + 4 * tc);
                        sum[p] = make_float4(sum[p].x + x.x, sum[p].y + x.y, sum[p].z + x.z, sum[p].w + x.w);
                    }
        }
        if (v_sum && ts == 0)
#pragma unroll
            for (int p = 0; p < PT; p++) cluster_store(to + (uint32_t)(p * rows) * 4u, sum[p]);
        cluster_sync();
        if (vp < PT && vi < own) {
            float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
            const float *from = recv + vp * rows + vi;
            const int step = PT * rows;
            int c = 0;
            for (; c + 4 <= sh.ctas; c += 4) {
                s0 += from[c * step];
                s1 += from[(c + 1) * step];
                s2 += from[(c + 2) * step];
                s3 += from[(c + 3) * step];
            }
            for (; c < sh.ctas; c++) s0 += from[c * step];
            const float v = v_own ? nv / (((s0 + s1) + (s2 + s3)) + 1e-12f) : 0.0f;
            const float *at = vs + vp * pitch + i0 + vi;
            for (int q = 0; q < sh.ctas; q++) cluster_store(cluster_addr(at, q), v);
        }
        cluster_sync();
        bool stop = last;
        if (checking) {
            // one barrier of all clusters: CTA 0 of each goes for all of its CTAs
            if (rank == 0 && tid == 0) {
                arrived += gridDim.x / sh.ctas;
                const float ok = grid_arrive_wait(A.ctl, &A.ctl->pad[0], arrived, A.status, A.spin_limit) ? 1.0f : 0.0f;
                for (int q = 0; q < sh.ctas; q++) cluster_store(cluster_addr(&s_ok, q), ok);
            }
            cluster_sync();
            if (s_ok == 0.0f) return;  // (alike in the whole cluster)
            bool above = false;
            for (int b = tid; b < A.n; b += kClThreads) {
                double s = 0.0;
                for (int r = 0; r < sh.ctas; r++)
                    s += __ldcg(A.partial + (size_t)((check & 1) * kClMaxCtas + r) * A.n + b);
                above |= !(s <= (double)A.threshold);
                if (blockIdx.x == 0) A.err[b] = s;
            }
            stop = !__syncthreads_or(above) || last;
            check++;
        }
        if (stop) {
            it++;
            break;
        }
    }
    for (int k = tid; k < PT * own; k += kClThreads) {
        const int p = k / own, i = k - p * own;
        if (b0 + p < A.n) {
            A.u[(size_t)(b0 + p) * d + i0 + i] = us[i * PT + p];
            A.v[(size_t)(b0 + p) * d + i0 + i] = vs[p * pitch + i0 + i];
        }
    }
    if (blockIdx.x == 0 && tid == 0) A.ctl->iterations = it;
}

cudaLaunchConfig_t cluster_config(int ctas, int blocks, size_t smem, cudaStream_t s, cudaLaunchAttribute *attr) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)ctas;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Estimated us per iteration (GB300, fitted to 64 .. 784 points, within 15%).
double cluster_time(const ClusterShape &s) {
    return 2.0 + 0.02 * s.ctas + (double)s.rows * s.pitch * (4.6e-5 + 0.9e-5 * s.pairs);
}

// Clusters of `ctas` CTAs with one CTA per SM that the device holds at once (0: none).
int cluster_count(int ctas) {
    static std::atomic<int> cached[64][kClMaxCtas + 1];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int c = cached[dev][ctas].load(std::memory_order_relaxed);
    if (c == 0) {
        const void *kern = (const void *)sk_cluster_kernel<4>;
        cudaLaunchAttribute attr{};
        cudaLaunchConfig_t cfg = cluster_config(ctas, ctas, kClMaxSmem - 2048, nullptr, &attr);
        int n = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            allow_shared_memory(kern, cfg.dynamicSmemBytes) != TM_OK ||
            cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return 0;  // (not kept: the next call asks again)
        }
        c = n > 0 ? n : -1;
        cached[dev][ctas].store(c, std::memory_order_relaxed);
    }
    return c > 0 ? c : 0;
}

// The cluster shape for an (n, d) problem: of those that hold all pairs at once (with a
// stopping test they meet) the one with the least time, or false.  Any shape that fits beats
// the slabs, whose half-steps never take less than 3.2 us (16 point counts 4 .. 850, 22 pair
// counts 1 .. 608, fixed iterations and stopping test: no solve of 40 iterations was slower).
bool cluster_shape(int64_t n, int64_t d, ClusterShape *out) {
    if (n > kOneWaveMaxPairs) return false;
    double best = 0;
    for (int ctas : {1, 2, 4, 6, 8, 10, 12, 16})
        for (int pairs = 1; pairs <= 4; pairs *= 2) {
            ClusterShape s;
            s.pairs = pairs;
            s.ctas = ctas;
            s.rows = (int)(ceil_div(d, (int64_t)ctas) + 3) & ~3;
            s.pitch = (int)((d + 3) & ~(int64_t)3);
            if (s.pitch / 4 > kClThreads || pairs * s.rows > kClThreads) continue;
            s.split = 1;
            while (s.split < 16 && kClThreads / (2 * s.split) * 4 >= s.pitch) s.split *= 2;
            s.clusters = (int)ceil_div(n, pairs);
            s.smem = ((size_t)s.rows * s.pitch +
                      (size_t)pairs * ((size_t)s.pitch * std::max(s.split - 1, 1) + (size_t)(ctas + 1) * s.rows)) *
                     sizeof(float);
            if (s.smem > kClMaxSmem - 2048 || s.clusters > cluster_count(ctas)) continue;
            const double us = cluster_time(s);
            if (best == 0 || us < best) {
                best = us;
                *out = s;
            }
        }
    return best > 0;
}

// K = exp(-C / eps) and K^T (scaling form), or C^T alone (log form, EXP = false),
// through 32 x 32 shared-memory tiles so both writes are coalesced.  inv_eps is
// the float32 reciprocal of eps: torch evaluates a CUDA tensor divided by a
// scalar as the product with that reciprocal.
template <bool EXP>
__global__ void sk_prepare_kernel(const float *__restrict__ C, float *__restrict__ K, float *__restrict__ KT,
                                  int d, float inv_eps) {
    __shared__ float tile[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int i = by + r, j = bx + threadIdx.x;
        if (i < d && j < d) {
            float x = C[(size_t)i * d + j];
            if (EXP) {
                x = expf(-x * inv_eps);  // the reference's torch.exp(-cost_matrix / epsilon) on CUDA
                K[(size_t)i * d + j] = x;
            }
            tile[r][threadIdx.x] = x;
        }
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int j = bx + r, i = by + threadIdx.x;
        if (i < d && j < d) KT[(size_t)j * d + i] = tile[threadIdx.x][r];
    }
}

__global__ void sk_fill_kernel(float *__restrict__ x, float *__restrict__ y, size_t count, float value) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < count; k += (size_t)gridDim.x * blockDim.x) {
        x[k] = value;
        y[k] = value;
    }
}

// y = log(x) elementwise (the reference's u.log(), a.log()), two arrays at once.
__global__ void sk_log_kernel(const float *__restrict__ x0, float *__restrict__ y0, const float *__restrict__ x1,
                              float *__restrict__ y1, size_t count) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < count; k += (size_t)gridDim.x * blockDim.x) {
        y0[k] = logf(x0[k]);
        y1[k] = logf(x1[k]);
    }
}

// ------------------------------------------------- transport cost and residual
// cost[b] = sum_ij P_ij C_ij and err[b] = sum_i |a_i - sum_j P_ij| with
// P_ij = exp((log u_i - C_ij / eps) + log v_j), the reference's plan
// (optimal_transport.py:136-144) without materialising it.  A CTA takes 128
// rows x 16 pairs; per row and pair, fp32 sums over 16-column chunks are
// added in fp64, and the row blocks are reduced in fixed order by
// sk_cost_reduce_kernel.
__global__ void __launch_bounds__(kSkThreads)
    sk_cost_kernel(const float *__restrict__ lu, const float *__restrict__ lv, const float *__restrict__ C,
                   const float *__restrict__ a, int n, int d, float inv_eps, double *__restrict__ cost_part,
                   double *__restrict__ err_part) {
    constexpr int TB = 16;
    __shared__ __align__(16) float sc[kSkRows * kSkPitch];
    __shared__ __align__(16) float sv[TB * kSkPitch];
    const int pair_blocks = (n + TB - 1) / TB;
    const int rb = blockIdx.x / pair_blocks, pb = blockIdx.x % pair_blocks;
    const int i0 = rb * kSkRows, b0 = pb * TB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tr = lane & 15, tb = (lane >> 4) + 2 * warp;
    const int b = b0 + tb;
    float lui[8];
    double cacc[8], racc[8];
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int i = i0 + tr + 16 * r;
        lui[r] = (i < d && b < n) ? lu[(size_t)b * d + i] : -INFINITY;
        cacc[r] = racc[r] = 0.0;
    }
    for (int j0 = 0; j0 < d; j0 += kSkChunk) {
        __syncthreads();
        for (int f = tid; f < kSkRows * kSkChunk; f += kSkThreads) {
            const int row = f / kSkChunk, col = f % kSkChunk;
            const int i = i0 + row, j = j0 + col;
            sc[row * kSkPitch + col] = (i < d && j < d) ? (C ? C[(size_t)i * d + j] : line_cost(i, j)) : 0.0f;
        }
        for (int f = tid; f < TB * kSkChunk; f += kSkThreads) {
            const int p = f / kSkChunk, col = f % kSkChunk;
            const int bb = b0 + p, j = j0 + col;
            sv[p * kSkPitch + col] = (bb < n && j < d) ? lv[(size_t)bb * d + j] : -INFINITY;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; r++) {
            float cs = 0.0f, rs = 0.0f;
#pragma unroll
            for (int k = 0; k < kSkChunk; k++) {
                const float c = sc[(tr + 16 * r) * kSkPitch + k];
                const float p = expf((lui[r] - c * inv_eps) + sv[tb * kSkPitch + k]);
                cs = fmaf(p, c, cs);
                rs += p;
            }
            cacc[r] += (double)cs;
            racc[r] += (double)rs;
        }
    }
    double cs = 0.0, es = 0.0;
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int i = i0 + tr + 16 * r;
        if (i < d && b < n) {
            cs += cacc[r];
            es += fabs((double)a[(size_t)b * d + i] - racc[r]);
        }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        cs += __shfl_xor_sync(0xffffffffu, cs, o);
        es += __shfl_xor_sync(0xffffffffu, es, o);
    }
    if (tr == 0 && b < n) {
        cost_part[(size_t)rb * n + b] = cs;
        err_part[(size_t)rb * n + b] = es;
    }
}

// The same sums for problems whose 128-row x 16-pair blocks would leave SMs idle: a
// CTA takes 4 rows x 4 pairs with 16 lanes across the columns of each, reading the
// cost rows and log v through L1 (float4 where aligned).  fp32 sums over 16 terms
// are added in fp64, the lanes by shuffles.
// 16 pairs x 784 points: 179 us with 7 blocks of the kernel above, 15 us with these.
constexpr int kCostRows = 4, kCostPairs = 4, kCostLanes = 16;

__global__ void __launch_bounds__(kSkThreads)
    sk_cost_rows_kernel(const float *__restrict__ lu, const float *__restrict__ lv, const float *__restrict__ C,
                        const float *__restrict__ a, int n, int d, float inv_eps, bool vec,
                        double *__restrict__ cost_part, double *__restrict__ err_part) {
    __shared__ double s_cost[kCostRows][kCostPairs], s_err[kCostRows][kCostPairs];
    const int lane = threadIdx.x & (kCostLanes - 1), cell = threadIdx.x / kCostLanes;
    const int row = cell % kCostRows, pair = cell / kCostRows;
    const int pair_blocks = (n + kCostPairs - 1) / kCostPairs;
    const int rb = blockIdx.x / pair_blocks, pb = blockIdx.x % pair_blocks;
    const int i = rb * kCostRows + row, b = pb * kCostPairs + pair;
    double cacc = 0.0, racc = 0.0;
    if (i < d && b < n) {
        const float x = lu[(size_t)b * d + i];
        const float *crow = C ? C + (size_t)i * d : nullptr;
        const float *vrow = lv + (size_t)b * d;
        for (int j0 = 4 * lane; j0 < d; j0 += 16 * kCostLanes) {
            float cs = 0.0f, rs = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int j = j0 + 4 * kCostLanes * q;
                if (j >= d) break;
                float c[4], v[4];
                if (vec) {
                    const float4 v4 = *reinterpret_cast<const float4 *>(vrow + j);
                    v[0] = v4.x, v[1] = v4.y, v[2] = v4.z, v[3] = v4.w;
                    if (crow) {
                        const float4 c4 = *reinterpret_cast<const float4 *>(crow + j);
                        c[0] = c4.x, c[1] = c4.y, c[2] = c4.z, c[3] = c4.w;
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; e++) c[e] = line_cost(i, j + e);
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const bool in = j + e < d;
                        c[e] = !in ? 0.0f : (crow ? crow[j + e] : line_cost(i, j + e));
                        v[e] = in ? vrow[j + e] : -INFINITY;
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float p = expf((x - c[e] * inv_eps) + v[e]);
                    cs = fmaf(p, c[e], cs);
                    rs += p;
                }
            }
            cacc += (double)cs;
            racc += (double)rs;
        }
    }
#pragma unroll
    for (int o = kCostLanes / 2; o > 0; o >>= 1) {
        cacc += __shfl_xor_sync(0xffffffffu, cacc, o);
        racc += __shfl_xor_sync(0xffffffffu, racc, o);
    }
    if (lane == 0) {
        s_cost[row][pair] = cacc;
        s_err[row][pair] = i < d && b < n ? fabs((double)a[(size_t)b * d + i] - racc) : 0.0;
    }
    __syncthreads();
    if (threadIdx.x < kCostPairs && pb * kCostPairs + (int)threadIdx.x < n) {
        double cs = 0.0, es = 0.0;
#pragma unroll
        for (int r = 0; r < kCostRows; r++) {
            cs += s_cost[r][threadIdx.x];
            es += s_err[r][threadIdx.x];
        }
        const size_t o = (size_t)rb * n + pb * kCostPairs + threadIdx.x;
        cost_part[o] = cs;
        err_part[o] = es;
    }
}

// Which cost kernel takes an (n, d) problem: 128-row blocks once there is one for every
// SM (4096 pairs x 64 points: 0.1 ms less than 4-row blocks), 4-row blocks below.
inline bool cost_by_rows(int64_t n, int64_t d, int sms) {
    return ceil_div(d, kSkRows) * ceil_div(n, 16) < (int64_t)sms;
}

// One warp per pair adds the row blocks in a fixed order.
__global__ void sk_cost_reduce_kernel(const double *__restrict__ cost_part, const double *__restrict__ err_part,
                                      int n, int row_blocks, double *__restrict__ cost, double *__restrict__ err) {
    const int b = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (b >= n) return;
    double c = 0.0, e = 0.0;
    for (int r = lane; r < row_blocks; r += 32) {
        c += cost_part[(size_t)r * n + b];
        e += err_part[(size_t)r * n + b];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c += __shfl_xor_sync(0xffffffffu, c, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
    }
    if (lane != 0) return;
    if (cost) cost[b] = c;
    if (err) err[b] = e;
}

// ---------------------------------------------------------------- the plan
// plan[b, i, j] = exp((log u[b,i] - C[i,j] / eps) + log v[b,j]) with the
// reference's operations and rounding on CUDA tensors (optimal_transport.py:
// 228-237): C / eps as torch evaluates a CUDA tensor divided by a scalar (a
// product with the float32 reciprocal of eps), then the two additions in that
// order, each rounded (explicit _rn operations: no multiply-add contraction).
// One pass that writes each plan entry once (HBM-write bound); C is re-read
// from L2 per pair.
__global__ void sk_plan_kernel(const float *__restrict__ lu, const float *__restrict__ lv, const float *__restrict__ C,
                               int n, int d, float inv_eps, bool vec, float *__restrict__ plan) {
    const int64_t rows = (int64_t)n * d;
    for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
        const int b = (int)(row / d), i = (int)(row % d);
        const float x = lu[row];
        const float *crow = C ? C + (size_t)i * d : nullptr;
        const float *vrow = lv + (size_t)b * d;
        float *prow = plan + (size_t)row * d;
        if (vec) {
            for (int j = 4 * threadIdx.x; j < d; j += 4 * blockDim.x) {
                const float4 c = crow ? *reinterpret_cast<const float4 *>(crow + j)
                                      : make_float4(line_cost(i, j), line_cost(i, j + 1), line_cost(i, j + 2),
                                                    line_cost(i, j + 3));
                const float4 v = *reinterpret_cast<const float4 *>(vrow + j);
                float4 o;
                o.x = expf(__fadd_rn(__fsub_rn(x, __fmul_rn(c.x, inv_eps)), v.x));
                o.y = expf(__fadd_rn(__fsub_rn(x, __fmul_rn(c.y, inv_eps)), v.y));
                o.z = expf(__fadd_rn(__fsub_rn(x, __fmul_rn(c.z, inv_eps)), v.z));
                o.w = expf(__fadd_rn(__fsub_rn(x, __fmul_rn(c.w, inv_eps)), v.w));
                *reinterpret_cast<float4 *>(prow + j) = o;
            }
        } else {
            for (int j = threadIdx.x; j < d; j += blockDim.x) {
                const float c = crow ? crow[j] : line_cost(i, j);
                prow[j] = expf(__fadd_rn(__fsub_rn(x, __fmul_rn(c, inv_eps)), vrow[j]));
            }
        }
    }
}

// --------------------------------------------- gradient w.r.t. the cost
// grad_C[i, j] = sum_b g[b] P_b[i, j]: the envelope-theorem gradient of the
// regularised transport cost with respect to the cost matrix, scaled by the
// upstream gradient of each pair's distance.  A CTA owns a 64 x 64 block of
// (i, j) (each thread 4 x 4 entries) and walks the pairs, 8 at a time, with
// the block's log-potentials staged in shared memory; plan entries are
// recomputed (base 2) and never stored.
constexpr int kGradTile = 64;
constexpr int kGradPairs = 8;

__global__ void __launch_bounds__(kSkThreads)
    sk_cost_grad_kernel(const float *__restrict__ lu, const float *__restrict__ lv, const float *__restrict__ C,
                        const float *__restrict__ gout, int n, int d, float mscale, float *__restrict__ grad) {
    __shared__ float su[kGradPairs][kGradTile];
    __shared__ float sv[kGradPairs][kGradTile];
    __shared__ float sg[kGradPairs];
    const int i0 = blockIdx.y * kGradTile, j0 = blockIdx.x * kGradTile;
    const int tid = threadIdx.x;
    const int ti = tid / 16, tj = tid % 16;  // entries (i0 + ti + 16 r, j0 + tj + 16 s)
    float mc[4][4], acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const int i = i0 + ti + 16 * r, j = j0 + tj + 16 * s;
            mc[r][s] = (i < d && j < d) ? (C ? C[(size_t)i * d + j] : line_cost(i, j)) * mscale : -INFINITY;
            acc[r][s] = 0.0f;
        }
    for (int p0 = 0; p0 < n; p0 += kGradPairs) {
        __syncthreads();
        for (int f = tid; f < kGradPairs * kGradTile; f += kSkThreads) {
            const int p = f / kGradTile, x = f % kGradTile;
            const int b = p0 + p;
            su[p][x] = (b < n && i0 + x < d) ? lu[(size_t)b * d + i0 + x] * kLog2e : -INFINITY;
            sv[p][x] = (b < n && j0 + x < d) ? lv[(size_t)b * d + j0 + x] * kLog2e : -INFINITY;
        }
        if (tid < kGradPairs) sg[tid] = p0 + tid < n ? gout[p0 + tid] : 0.0f;
        __syncthreads();
#pragma unroll
        for (int p = 0; p < kGradPairs; p++) {
            const float g = sg[p];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float x = su[p][ti + 16 * r];
#pragma unroll
                for (int s = 0; s < 4; s++) acc[r][s] = fmaf(g, ex2(mc[r][s] + (x + sv[p][tj + 16 * s])), acc[r][s]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const int i = i0 + ti + 16 * r, j = j0 + tj + 16 * s;
            if (i < d && j < d) grad[(size_t)i * d + j] = acc[r][s];
        }
}

// ------------------------------------------------------------------ host
int check_ptr(const void *p, const char *name) {
    if (!p) return fail(TM_ERR_INVALID_ARGUMENT, "%s is NULL", name);
    return TM_OK;
}

int check_nd(int64_t n, int64_t d) {
    if (n < 1 || d < 1) return fail(TM_ERR_INVALID_ARGUMENT, "need n >= 1 pairs and d >= 1 points, got (%lld, %lld)",
                                    (long long)n, (long long)d);
    if (n > (1 << 24) || d > (1 << 20) || n * d > ((int64_t)1 << 31))
        return fail(TM_ERR_TOO_LARGE, "problem too large: (%lld, %lld)", (long long)n, (long long)d);
    return TM_OK;
}

bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

// Launches the slab kernel where the problem has its shape (the tuning table does not
// reach these: its variants are shapes of the tile kernel).
template <bool LOG, int V>
bool sk_slab_launch(SkArgs &A, cudaStream_t s, int *st) {
    SlabShape sh;
    if (!slab_shape<LOG, V>(A.n, A.d, std::min(sm_count(), kSlabMaxCtas), &sh)) return false;
    const void *kern = (const void *)sk_slab_kernel<LOG, V>;
    auto run = [&]() -> int {
        const int ready = allow_shared_memory(kern, sh.smem);
        if (ready != TM_OK) return ready;
        TM_CHECK_CUDA(cudaMemsetAsync(A.ctl, 0, sizeof(SkControl), s));
        void *params[] = {&A, &sh};
        TM_CHECK_CUDA(cudaLaunchCooperativeKernel(kern, dim3(sh.ctas * sh.groups), dim3(kSkThreads), params, sh.smem, s));
        TM_LAUNCH_CHECK("sk_slab_kernel");
        return TM_OK;
    };
    *st = run();
    return true;
}

bool sk_slab(bool log_form, SkArgs &A, cudaStream_t s, int *st) {
    const bool wide = A.d > kSlabWarps * SlabTile<false, 1>::kCols;
    if (log_form) return wide ? sk_slab_launch<true, 2>(A, s, st) : sk_slab_launch<true, 1>(A, s, st);
    return wide ? sk_slab_launch<false, 2>(A, s, st) : sk_slab_launch<false, 1>(A, s, st);
}

// Launches the cluster kernel where a shape fits (the scaling form, K^T that of K).
bool sk_cluster(bool log_form, const SkArgs &A, cudaStream_t s, int *st) {
    ClusterShape sh;
    if (log_form || !A.paired || !cluster_shape(A.n, A.d, &sh)) return false;
    auto run = [&](auto kernel) -> int {
        TM_CHECK_CUDA(cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        const int ready = allow_shared_memory((const void *)kernel, sh.smem);
        if (ready != TM_OK) return ready;
        TM_CHECK_CUDA(cudaMemsetAsync(A.ctl, 0, sizeof(SkControl), s));
        cudaLaunchAttribute attr[2]{};
        cudaLaunchConfig_t cfg = cluster_config(sh.ctas, sh.clusters * sh.ctas, sh.smem, s, attr);
        if (A.check_every > 0) {  // the clusters wait for one another
            attr[1].id = cudaLaunchAttributeCooperative;
            attr[1].val.cooperative = 1;
            cfg.numAttrs = 2;
        }
        TM_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, A, sh));
        TM_LAUNCH_CHECK("sk_cluster_kernel");
        return TM_OK;
    };
    *st = sh.pairs == 1   ? run(sk_cluster_kernel<1>)
          : sh.pairs == 2 ? run(sk_cluster_kernel<2>)
                          : run(sk_cluster_kernel<4>);
    return true;
}

// The persistent solver on caller-provided state.  control: 256-byte control
// block; partial/err/notconv only when check_every > 0.
int sk_launch(bool log_form, SkArgs A, cudaStream_t s) {
    int *status = nullptr;
    int st = device_status_word(&status);
    if (st != TM_OK) return st;
    A.status = status;
    A.spin_limit = grid_wait_budget();
    if (sk_cluster(log_form, A, s, &st)) return st;
    if (sk_slab(log_form, A, s, &st)) return st;
    // autotuned variant: bit 0 = 64 pairs per tile (else 16), bit 1 = one CTA per SM
    // (else two); built-in: 64 pairs per tile above 24 pairs, two CTAs per SM
    const int variant = tune_variant(kTuneSinkhornF32, tune_class(kTuneSinkhornF32, A.n, A.d));
    const bool wide = variant < 0 ? A.n > 24 : (variant & 1) != 0;
    const void *kern;
    if (log_form) kern = wide ? (const void *)sk_solve_kernel<true, 4> : (const void *)sk_solve_kernel<true, 1>;
    else kern = wide ? (const void *)sk_solve_kernel<false, 4> : (const void *)sk_solve_kernel<false, 1>;
    int per_sm = 0;
    TM_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSkThreads, 0));
    if (per_sm < 1) return fail(TM_ERR_UNSUPPORTED, "Sinkhorn kernel does not fit on an SM");
    if (variant >= 0 && (variant & 2)) per_sm = 1;
    const int tb = wide ? 64 : 16;
    const int64_t tiles = ceil_div(A.d, kSkRows) * ceil_div(A.n, tb);
    const int blocks = (int)std::min<int64_t>(tiles, (int64_t)per_sm * sm_count());
    TM_CHECK_CUDA(cudaMemsetAsync(A.ctl, 0, sizeof(SkControl), s));
    void *params[] = {&A};
    TM_CHECK_CUDA(cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(kSkThreads), params, 0, s));
    TM_LAUNCH_CHECK("sk_solve_kernel");
    return TM_OK;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct SkLayout {
    size_t mat, mat_t, su, sv, partial, err, notconv, ctl, cost_part, err_part, total;
};

SkLayout sk_layout(int64_t n, int64_t d, bool log_form, int64_t max_iter, int64_t check_every, bool line) {
    SkLayout L{};
    const size_t dd = (size_t)d * d * sizeof(float), nd = (size_t)n * d * sizeof(float);
    // residual partials: a row per row block of the tile kernel, per CTA of a slab group, two per
    // CTA of a cluster
    size_t rblocks = (size_t)ceil_div(d, kSkRows);
    if (n <= kOneWaveMaxPairs)
        rblocks = std::max(rblocks, std::min((size_t)kSlabMaxCtas, std::max((size_t)ceil_div(d, kSlabRows),
                                                                            (size_t)(log_form ? 0 : 2 * kClMaxCtas))));
    if (check_every <= 0) rblocks = 0;
    const size_t checks = check_every > 0 ? (size_t)(max_iter / check_every) + 1 : 1;
    size_t off = 0;
    L.mat = off;
    off += (log_form || line) ? 0 : align256(dd);  // K (the log form reads C itself)
    L.mat_t = off;
    off += line ? 0 : align256(dd);  // the line cost is computed where it is used
    L.su = off;
    off += align256(nd);  // u (scaling) or log a
    L.sv = off;
    off += align256(nd);  // v (scaling) or log b
    L.partial = off;
    off += align256(rblocks * n * sizeof(double));
    L.err = off;
    off += align256(n * sizeof(double));
    L.notconv = off;
    off += align256(checks * sizeof(int));
    L.ctl = off;
    off += align256(sizeof(SkControl));
    // (sized for the cost kernel with the more blocks where either may run: the SM count is a
    // property of the device, not of the problem)
    const size_t cblocks = cost_by_rows(n, d, kSlabMaxCtas) ? (size_t)ceil_div(d, kCostRows)
                                                            : (size_t)ceil_div(d, kSkRows);
    L.cost_part = off;
    off += align256(cblocks * n * sizeof(double));
    L.err_part = off;
    off += align256(cblocks * n * sizeof(double));
    L.total = off;
    return L;
}

template <typename T>
T *ws_at(void *ws, size_t off) {
    return reinterpret_cast<T *>(static_cast<unsigned char *>(ws) + off);
}

unsigned grid_for(size_t count) {
    return (unsigned)std::min<size_t>((count + 255) / 256, (size_t)sm_count() * 8);
}

int sk_cost(const float *lu, const float *lv, const float *C, const float *a, int64_t n, int64_t d, double epsilon,
            double *cost_part, double *err_part, double *cost, double *err, cudaStream_t s) {
    int64_t rblocks;
    const float inv_eps = 1.0f / (float)epsilon;
    if (cost_by_rows(n, d, std::min(sm_count(), kSlabMaxCtas))) {
        rblocks = ceil_div(d, kCostRows);
        const bool vec = (d % 4) == 0 && aligned16(lv) && aligned16(C);
        sk_cost_rows_kernel<<<(unsigned)(rblocks * ceil_div(n, kCostPairs)), kSkThreads, 0, s>>>(
            lu, lv, C, a, (int)n, (int)d, inv_eps, vec, cost_part, err_part);
        TM_LAUNCH_CHECK("sk_cost_rows_kernel");
    } else {
        rblocks = ceil_div(d, kSkRows);
        sk_cost_kernel<<<(unsigned)(rblocks * ceil_div(n, 16)), kSkThreads, 0, s>>>(lu, lv, C, a, (int)n, (int)d,
                                                                                    inv_eps, cost_part, err_part);
        TM_LAUNCH_CHECK("sk_cost_kernel");
    }
    sk_cost_reduce_kernel<<<(unsigned)ceil_div(n, 8), 256, 0, s>>>(cost_part, err_part, (int)n, (int)rblocks, cost, err);
    TM_LAUNCH_CHECK("sk_cost_reduce_kernel");
    return TM_OK;
}

}  // namespace
}  // namespace tmc

// ----------------------------------------------------------------- C ABI
extern "C" size_t tm_sinkhorn_iter_workspace_size(void) { return sizeof(tmc::SkControl); }

// The reference's fixed-count fused iterations, in place, on the caller's
// matrices: one persistent launch for all n_iter iterations.
static int sk_fixed(bool log_form, const float *num_u, const float *num_v, const float *mat, const float *mat_t,
                    float *u, float *v, int64_t n, int64_t d, int64_t n_iter, double epsilon, void *workspace,
                    size_t workspace_bytes, cudaStream_t s) {
    using namespace tmc;
    const void *ptrs[] = {num_u, num_v, mat, mat_t, u, v};
    const char *names[] = {"a", "b", "matrix", "transposed matrix", "u", "v"};
    for (int k = 0; k < 6; k++)
        if (check_ptr(ptrs[k], names[k]) != TM_OK) return TM_ERR_INVALID_ARGUMENT;
    int st = check_nd(n, d);
    if (st != TM_OK) return st;
    if (n_iter < 0) return fail(TM_ERR_INVALID_ARGUMENT, "n_iter must be >= 0");
    if (n_iter > (1LL << 30)) return fail(TM_ERR_TOO_LARGE, "n_iter too large");
    if (!workspace || workspace_bytes < sizeof(SkControl) || !aligned16(workspace))
        return fail(TM_ERR_WORKSPACE, "Sinkhorn iterations need a 16-byte aligned workspace of %zu bytes",
                    sizeof(SkControl));
    if (n_iter == 0) return TM_OK;
    SkArgs A{};
    A.num_u = num_u;
    A.num_v = num_v;
    A.mat = mat;
    A.mat_t = mat_t;
    A.u = u;
    A.v = v;
    A.n = (int)n;
    A.d = (int)d;
    A.mscale = log_form ? (float)(-1.4426950408889634 / epsilon) : 0.0f;
    A.max_iter = (int)n_iter;
    A.check_every = 0;
    A.ctl = static_cast<SkControl *>(workspace);
    A.vec = (d % 4) == 0 && aligned16(mat) && aligned16(mat_t) && aligned16(u) && aligned16(v);
    return sk_launch(log_form, A, s);
}

extern "C" int tm_sinkhorn_fastiter(const float *a, const float *b, const float *K, const float *K_T, float *u,
                                    float *v, int64_t n, int64_t d, int64_t n_iter, void *workspace,
                                    size_t workspace_bytes, tm_stream_t stream) {
    return sk_fixed(false, a, b, K, K_T, u, v, n, d, n_iter, 1.0, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int tm_sinkhorn_logiter(const float *log_a, const float *log_b, const float *M, const float *M_T,
                                   float *log_u, float *log_v, int64_t n, int64_t d, int64_t n_iter, double epsilon,
                                   void *workspace, size_t workspace_bytes, tm_stream_t stream) {
    if (!(epsilon > 0)) return tmc::fail(TM_ERR_INVALID_ARGUMENT, "epsilon must be positive, got %g", epsilon);
    return sk_fixed(true, log_a, log_b, M, M_T, log_u, log_v, n, d, n_iter, epsilon, workspace, workspace_bytes,
                    (cudaStream_t)stream);
}

extern "C" size_t tm_sinkhorn_f32_workspace_size(int64_t n, int64_t d, int log_space, int64_t max_iter,
                                                 int64_t check_every, int line_cost) {
    if (n < 1 || d < 1 || max_iter < 0) return 0;
    return tmc::sk_layout(n, d, log_space != 0, max_iter, check_every, line_cost != 0).total;
}

extern "C" int tm_sinkhorn_f32_solve(const float *a, const float *b, const float *C, int64_t n, int64_t d,
                                     double epsilon, int log_space, int64_t max_iter, double threshold,
                                     int64_t check_every, float *log_u, float *log_v, double *cost, double *row_err,
                                     int32_t *iterations, void *workspace, size_t workspace_bytes,
                                     tm_stream_t stream) {
    using namespace tmc;
    const void *ptrs[] = {a, b, log_u, log_v};
    const char *names[] = {"a", "b", "log_u", "log_v"};
    for (int k = 0; k < 4; k++)
        if (check_ptr(ptrs[k], names[k]) != TM_OK) return TM_ERR_INVALID_ARGUMENT;
    int st = check_nd(n, d);
    if (st != TM_OK) return st;
    if (!(epsilon > 0)) return fail(TM_ERR_INVALID_ARGUMENT, "epsilon must be positive, got %g", epsilon);
    if (max_iter < 1 || max_iter > (1LL << 30)) return fail(TM_ERR_INVALID_ARGUMENT, "max_iter must be in [1, 2^30]");
    const bool line = C == nullptr;  // the cost of d points on a line, computed where used
    if (threshold < 0) return fail(TM_ERR_INVALID_ARGUMENT, "threshold must be >= 0");
    if (threshold > 0 && check_every < 1) return fail(TM_ERR_INVALID_ARGUMENT, "check_every must be >= 1");
    if (threshold == 0) check_every = 0;
    const bool log_form = log_space != 0;
    const SkLayout L = sk_layout(n, d, log_form, max_iter, check_every, line);
    if (!workspace || workspace_bytes < L.total || ((uintptr_t)workspace & 255))
        return fail(TM_ERR_WORKSPACE, "workspace must be 256-byte aligned and hold %zu bytes", L.total);
    cudaStream_t s = (cudaStream_t)stream;
    const size_t nd = (size_t)n * d;
    float *su = ws_at<float>(workspace, L.su), *sv = ws_at<float>(workspace, L.sv);
    float *mat_t = line ? nullptr : ws_at<float>(workspace, L.mat_t);
    const dim3 tgrid((unsigned)ceil_div(d, 32), (unsigned)ceil_div(d, 32)), tblock(32, 8);
    SkArgs A{};
    A.inv_eps = 1.0f / (float)epsilon;
    if (log_form) {
        if (!line) {
            sk_prepare_kernel<false><<<tgrid, tblock, 0, s>>>(C, nullptr, mat_t, (int)d, 0.0f);
            TM_LAUNCH_CHECK("sk_prepare_kernel");
        }
        sk_log_kernel<<<grid_for(nd), 256, 0, s>>>(a, su, b, sv, nd);  // log a, log b
        TM_LAUNCH_CHECK("sk_log_kernel");
        sk_fill_kernel<<<grid_for(nd), 256, 0, s>>>(log_u, log_v, nd, 0.0f);
        TM_LAUNCH_CHECK("sk_fill_kernel");
        A.num_u = su;
        A.num_v = sv;
        A.mat = C;
        A.u = log_u;
        A.v = log_v;
        A.mscale = (float)(-1.4426950408889634 / epsilon);
    } else {
        float *K = line ? nullptr : ws_at<float>(workspace, L.mat);
        if (!line) {
            sk_prepare_kernel<true><<<tgrid, tblock, 0, s>>>(C, K, mat_t, (int)d, 1.0f / (float)epsilon);
            TM_LAUNCH_CHECK("sk_prepare_kernel");
        }
        sk_fill_kernel<<<grid_for(nd), 256, 0, s>>>(su, sv, nd, 1.0f);
        TM_LAUNCH_CHECK("sk_fill_kernel");
        A.num_u = a;
        A.num_v = b;
        A.mat = K;
        A.u = su;
        A.v = sv;
    }
    A.mat_t = mat_t;
    A.paired = true;
    A.n = (int)n;
    A.d = (int)d;
    A.max_iter = (int)max_iter;
    A.check_every = (int)check_every;
    A.threshold = (float)threshold;
    A.partial = ws_at<double>(workspace, L.partial);
    A.err = ws_at<double>(workspace, L.err);
    A.notconv = ws_at<int>(workspace, L.notconv);
    A.ctl = ws_at<SkControl>(workspace, L.ctl);
    A.vec = (d % 4) == 0 && aligned16(A.mat) && aligned16(A.u) && aligned16(A.v) && aligned16(A.num_u) &&
            aligned16(A.num_v);
    if (check_every > 0)
        TM_CHECK_CUDA(cudaMemsetAsync(A.notconv, 0, (size_t)(max_iter / check_every + 1) * sizeof(int), s));
    if ((st = sk_launch(log_form, A, s)) != TM_OK) return st;
    if (!log_form) {
        sk_log_kernel<<<grid_for(nd), 256, 0, s>>>(su, log_u, sv, log_v, nd);
        TM_LAUNCH_CHECK("sk_log_kernel");
    }
    if (iterations)
        TM_CHECK_CUDA(cudaMemcpyAsync(iterations, &A.ctl->iterations, sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    if (cost || row_err)
        return sk_cost(log_u, log_v, C, a, n, d, epsilon, ws_at<double>(workspace, L.cost_part),
                       ws_at<double>(workspace, L.err_part), cost, row_err, s);
    return TM_OK;
}

extern "C" int tm_sinkhorn_plan(const float *log_u, const float *log_v, const float *C, int64_t n, int64_t d,
                                double epsilon, float *plan, tm_stream_t stream) {
    using namespace tmc;
    const void *ptrs[] = {log_u, log_v, plan};
    const char *names[] = {"log_u", "log_v", "plan"};
    for (int k = 0; k < 3; k++)
        if (check_ptr(ptrs[k], names[k]) != TM_OK) return TM_ERR_INVALID_ARGUMENT;
    int st = check_nd(n, d);
    if (st != TM_OK) return st;
    if (!(epsilon > 0)) return fail(TM_ERR_INVALID_ARGUMENT, "epsilon must be positive, got %g", epsilon);
    const bool vec = (d % 4) == 0 && aligned16(log_v) && aligned16(C) && aligned16(plan);
    const unsigned blocks = (unsigned)std::min<int64_t>(n * d, (int64_t)sm_count() * 32);
    const float inv_eps = 1.0f / (float)epsilon;  // torch: tensor / scalar = tensor * (1 / scalar) on CUDA
    sk_plan_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(log_u, log_v, C, (int)n, (int)d, inv_eps, vec, plan);
    TM_LAUNCH_CHECK("sk_plan_kernel");
    return TM_OK;
}

extern "C" int tm_sinkhorn_cost_grad(const float *log_u, const float *log_v, const float *C,
                                     const float *grad_distance, int64_t n, int64_t d, double epsilon,
                                     float *grad_C, tm_stream_t stream) {
    using namespace tmc;
    const void *ptrs[] = {log_u, log_v, grad_distance, grad_C};
    const char *names[] = {"log_u", "log_v", "grad_distance", "grad_C"};
    for (int k = 0; k < 4; k++)
        if (check_ptr(ptrs[k], names[k]) != TM_OK) return TM_ERR_INVALID_ARGUMENT;
    int st = check_nd(n, d);
    if (st != TM_OK) return st;
    if (!(epsilon > 0)) return fail(TM_ERR_INVALID_ARGUMENT, "epsilon must be positive, got %g", epsilon);
    const dim3 grid((unsigned)ceil_div(d, kGradTile), (unsigned)ceil_div(d, kGradTile));
    if (grid.y > 65535) return fail(TM_ERR_TOO_LARGE, "d too large for the gradient kernel");
    sk_cost_grad_kernel<<<grid, kSkThreads, 0, (cudaStream_t)stream>>>(
        log_u, log_v, C, grad_distance, (int)n, (int)d, (float)(-1.4426950408889634 / epsilon), grad_C);
    TM_LAUNCH_CHECK("sk_cost_grad_kernel");
    return TM_OK;
}
