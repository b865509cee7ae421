// Ragged point-cloud Sinkhorn: many OT problems of uneven sizes (n_p source
// and m_p target points in R^3, squared-Euclidean cost) solved together in
// ONE cooperative persistent launch, and the gradient of the regularised
// cost w.r.t. the points.
//
// Per problem, log-domain Sinkhorn iterations (the form of
// torchmorph/optimal_transport.py:96-125, with the cost recomputed from the
// points instead of read from a matrix):
//
//   f_i = -eps LSE_j( (g_j - C_ij)/eps + log b_j ),
//   g_j = -eps LSE_i( (f_i - C_ij)/eps + log a_i ),   C_ij = |x_i - y_j|^2.
//
// Work: an item is 16 own points of one problem, rows for the f-update, columns for the
// g-update, against all points of the partner cloud.  One warp takes an item by itself: its
// lanes run over the partners, 2 per lane and step, the own points in packed float32 pairs;
// the lanes' sums merge by shuffles.  The partners' records (centred point, exponent term)
// are kept in the workspace, padded per problem to whole steps, and rewritten with the
// potentials, so the loop is loads, FMAs and ex2.  The item lists are sorted by cost
// (partner points, most first) and dealt to the warps of a persistent grid back and forth;
// a grid barrier separates the two updates, nothing else does.  The sums are shifted by the
// previous iteration's value instead of a running maximum.
//
// Bound: per pair 5 operations of the FMA pipe (27 us a half-iteration of the batch below),
// 1 ex2 (22 us) and, with what the loop itself needs, 6 instructions; half of the issue
// slots are used, the rest waits on the 4 warps' dependent FMA-ex2-sum chains.  512 problems
// of 64 .. 2048 points, 185 M pairs, 100 iterations: 12.2 ms; with 64-point tiles per CTA, a
// running maximum per lane, scalar FMAs and a ticket queue 19.3 ms.  One problem of 2048 x
// 2048 points, 200 iterations: 7.9 -> 5.9 ms; 2048 problems of 20 points: 8.2 -> 4.4 ms.
// Packed FMAs alone gave 18.1 ms, without the running maximum 13.8, then records 12.2.  Tried
// at that point: partners staged in shared memory by the CTA 14.2 ms, in a ring of bulk
// copies 16.6, records doubled for the packed operands 13.3, two steps unrolled 12.5; items
// of 8 points 14.2 (3 CTAs an SM); one shift for all 16 own points 11.0, but a pair's error
// grows by half.
//
// Potentials use the dual form f = eps (log u - log a), g = eps (log v -
// log b) of the reference's log_u / log_v and start where log_u = log_v = 0.
//
// Stopping: on check iterations the g-update also accumulates, per problem,
// sum_j b_j |exp((g_old_j - g_new_j)/eps) - 1|, the L1 column-marginal
// error of the plan (f, g_old) whose rows the f-update just made exact;
// problems at or below the threshold stop and their tiles are skipped
// (threshold <= 0: every problem runs max_iter iterations, as the
// reference's threshold = 0).
//
// Every wait in the grid barrier is bounded; a barrier that gives up sets
// the library's device status word and an abort flag that makes every CTA
// leave.  The launch is cooperative, so all CTAs are co-resident.
#include <algorithm>
#include <cmath>
#include <vector>

#include "tm_common.cuh"
#include "tm_tma.cuh"

namespace tmc {
namespace {

constexpr int kPcThreads = 256;
constexpr int kPcWarps = kPcThreads / 32;
constexpr int kPcTile = 64;  // partners per step of a warp; problems are padded to whole tiles
constexpr int kPcOwn = 16;   // own points per item
constexpr int kPcPairs = kPcOwn / 2, kPcShare = 32 / kPcOwn;  // packed pairs; lanes that finish one own point
// gradient kernel
constexpr int kPcLanes = 16;                      // threads sharing one group of own points
constexpr int kPcRep = 4;                         // own points per thread
constexpr int kPcGroups = kPcThreads / kPcLanes;  // 16 groups
constexpr int kPcGradChunk = 256;                 // partner points staged per pass
static_assert(kPcTile == kPcGroups * kPcRep, "the gradient walks the same tiles");
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

struct PcProblem {
    int64_t x0, y0;  // first source / target point (packed arrays)
    int n, m;
    int row_tile0, col_tile0;  // first row tile / column tile of the problem
    float ox, oy, oz;          // centroid of both clouds (the kernels work in centred coordinates)
    int row_item0, col_item0;  // first row item / column item
    int pad;
};

// 2^x with the hardware approximation (MUFU.EX2, ~2 ulp, subnormal results
// flushed: they are below 2^-126 of the running maximum and cannot change a
// float32 sum).
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct PcControl {
    unsigned barrier_count;
    unsigned barrier_gen;
    int n_active;
    int abort;
    int iterations;  // iterations run (all problems)
    int n_row_list, n_col_list;  // items of the still-active problems
    int pad[57];
};
static_assert(sizeof(PcControl) == 256, "control block is 256 bytes");

// One side (sources or targets) of all problems.
struct PcSide {
    const float *pts;  // (N, 3)
    const float *lw;   // log weights (N)
    float *pot;        // potentials (N)
    // Records of the points, every problem padded to whole tiles, 5 arrays of `stride`
    // floats: centred x, y, z; w = k (pot - |x|^2) + log weight log2(e) (-inf on padding);
    // shift = k (pot - |x|^2), minus the last log-sum-exp.  k = log2(e) / eps.
    float *rec;
    int64_t stride;
};

struct __align__(16) PcItem {
    int64_t own0, own_rec;  // first own point, its record
    int n_own;              // own points
    int other;              // first tile of the partner cloud
    int rounds;             // its tiles
    int prob;
};
static_assert(sizeof(PcItem) == 32, "descriptor layout");

struct PcArgs {
    PcSide side[2];  // rows (x, a, f), columns (y, b, g)
    const PcProblem *prob;
    int nprob, row_tiles, row_items;
    float *err;       // per problem: marginal error being accumulated
    int *active;      // per problem: 1 while iterating
    int *iters;       // per problem: iterations when it stopped
    const PcItem *items;  // every row item, then every column item
    const int *row_order, *col_order;  // the problems by cost of their row / column items, most first
    int *row_list, *col_list;  // items of the active problems in that order (rebuilt on check iterations)
    PcControl *ctl;
    int *status;
    float eps, threshold;
    int max_iter, check_every;
    long long spin_limit;  // polls a barrier wait may take (tm_set_grid_wait_budget)
};

__device__ __forceinline__ int find_problem(const PcProblem *prob, int nprob, int tile, bool rows) {
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((rows ? prob[mid].row_tile0 : prob[mid].col_tile0) <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Two floats in one 64-bit register pair: the packed operations round each half as the
// scalar ones do.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// A record's w and shift for a potential, and what rounding took from the shift.  Potential
// and |x|^2 cancel before they are scaled, and both are scaled by the same k: a rounding of
// k changes an exponent (f + g - C) k by that much of itself, not of its terms.  The steps of
// `rest` are kept apart (no contraction) so that it is what it says.
__device__ __forceinline__ float record_w(float pot, float lw, float r2, float k) {
    return fmaf(k, pot - r2, lw * kLog2e);
}
__device__ __forceinline__ float record_shift(float pot, float r2, float k, float *rest) {
    const float d = __fsub_rn(pot, r2), t = __fsub_rn(d, pot), sh = __fmul_rn(k, d);
    const float lost = __fsub_rn(__fsub_rn(pot, __fsub_rn(d, t)), __fadd_rn(r2, t));
    *rest = fmaf(k, lost, fmaf(k, d, -sh));
    return sh;
}

// log2 sum_j 2^z_ij of this lane's own point (of kPcOwn, 32 / kPcOwn lanes to a point; records
// at `own`), with a running maximum per lane: any exponents.
__device__ __noinline__ float running_lse(const float *own, int64_t own_stride, const float *other,
                                          int64_t other_stride, int points, float k) {
    const int lane = threadIdx.x & 31;
    float res = 0.f;
    for (int q0 = 0; q0 < kPcOwn; q0 += 4) {
        float qx[4], qy[4], qz[4], mx[4], sum[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            qx[q] = 2.f * k * own[q0 + q];
            qy[q] = 2.f * k * own[own_stride + q0 + q];
            qz[q] = 2.f * k * own[2 * own_stride + q0 + q];
            mx[q] = -1e30f;
            sum[q] = 0.f;
        }
        for (int j = lane; j < points; j += 32) {
            const float yx = other[j], yy = other[other_stride + j], yz = other[2 * other_stride + j];
            const float w = __ldcg(other + 3 * other_stride + j);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float z = fmaf(qx[q], yx, fmaf(qy[q], yy, fmaf(qz[q], yz, w)));
                if (z > mx[q]) {
                    sum[q] *= fast_exp2(mx[q] - z);
                    mx[q] = z;
                }
                sum[q] += fast_exp2(z - mx[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float m2 = __shfl_xor_sync(0xffffffffu, mx[q], o), s2 = __shfl_xor_sync(0xffffffffu, sum[q], o);
                const float m = fmaxf(mx[q], m2);
                sum[q] = sum[q] * fast_exp2(mx[q] - m) + s2 * fast_exp2(m2 - m);
                mx[q] = m;
            }
            if (lane / kPcShare == q0 + q) res = mx[q] + log2f(sum[q]);
        }
    }
    return res;
}

// One half-iteration: this warp's items of `list` (n of them).
//
// In base 2, with x^ = x - o, y^ = y - o (o the problem's centroid) and
// k = log2(e) / eps, the exponent of a pair is
//   z_ij = w_j - k |x^_i - y^_j|^2 = [w_j - k |y^_j|^2] + (2k x^_i) . y^_j - k |x^_i|^2,
// w_j = k pot_j + log weight_j log2(e): three FMAs per pair on a partner's
// record.  Centring keeps |y^|^2 small, so the expansion loses ~1e-5 relative at most.
//
// The sums are taken of 2^(z_ij - v_i), v_i the value log2 sum_j 2^z_ij had one iteration
// ago, known from the own potential: no maximum to keep, and the new potential is the old
// one plus -eps ln(sum).  A sum that leaves [2^-60, 2^100] (terms below 2^-126 are flushed)
// or is NaN sends its warp through running_lse, as the first iteration, which has no
// value to shift by, does.
__device__ __forceinline__ void half_iteration(const PcArgs &a, const PcSide &own, const PcSide &other,
                                               const int *list, int n, bool first, bool check) {
    constexpr int H = kPcPairs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float k = kLog2e / a.eps;
    const int warps = gridDim.x * kPcWarps;
    // neighbours in the list share a CTA's L1, unless there are too few to go round
    const int self = n >= warps ? blockIdx.x * kPcWarps + warp : warp * gridDim.x + blockIdx.x;
    auto number = [&](int i) {  // this warp's i-th item: dealt back and forth
        const int64_t at = (int64_t)i * warps + ((i & 1) ? warps - 1 - self : self);
        return at < n ? __ldcg(list + at) : -1;  // (the lists are rewritten on check iterations: L2 loads)
    };
    int id = number(0), id1 = number(1);
    if (id < 0) return;
    PcItem T = a.items[id];
    for (int i = 0;; i++) {
        PcItem N = T;
        if (id1 >= 0) N = a.items[id1];
        id = id1;
        id1 = number(i + 2);
        const int mine = lane / kPcShare;
        const bool valid = mine < T.n_own;
        const float old = valid ? __ldcg(own.pot + T.own0 + mine) : 0.f;
        const float lw = valid ? own.lw[T.own0 + mine] : 0.f;
        const float *orec = own.rec + T.own_rec;
        const float *px = other.rec + (int64_t)T.other * kPcTile + 2 * lane, *py = px + other.stride,
                    *pz = py + other.stride, *pw = pz + other.stride;
        const float mx = orec[mine], my = orec[own.stride + mine], mz = orec[2 * own.stride + mine];
        const float r2 = fmaf(mx, mx, fmaf(my, my, mz * mz));
        float rest, pot = 0.f;
        bool ok = false;
        if (!first) {
            // records of a side are written only while the other side's are read
            auto xyz2 = [](const float *p) { return __ldg(reinterpret_cast<const float2 *>(p)); };
            float2 nx = xyz2(px), ny = xyz2(py), nz = xyz2(pz), nw = __ldcg(reinterpret_cast<const float2 *>(pw));
            f32x2 qx[H], qy[H], qz[H], shift[H], sum[H];
            const f32x2 k2 = pack2(2.f * k, 2.f * k);
#pragma unroll
            for (int h = 0; h < H; h += 2) {
                auto quad = [&](int c) { return *reinterpret_cast<const ulonglong2 *>(orec + c * own.stride + 2 * h); };
                const ulonglong2 ox = quad(0), oy = quad(1), oz = quad(2);
                const float4 os = __ldcg(reinterpret_cast<const float4 *>(orec + 4 * own.stride + 2 * h));
                qx[h] = mul2(k2, ox.x);
                qx[h + 1] = mul2(k2, ox.y);
                qy[h] = mul2(k2, oy.x);
                qy[h + 1] = mul2(k2, oy.y);
                qz[h] = mul2(k2, oz.x);
                qz[h + 1] = mul2(k2, oz.y);
                shift[h] = pack2(os.x, os.y);
                shift[h + 1] = pack2(os.z, os.w);
                sum[h] = sum[h + 1] = pack2(0.f, 0.f);
            }
#pragma unroll 1
            for (int r = T.rounds; r > 0; r--) {
                const float2 cx = nx, cy = ny, cz = nz, cw = nw;
                if (r > 1) {
                    px += kPcTile;
                    py += kPcTile;
                    pz += kPcTile;
                    pw += kPcTile;
                    nx = xyz2(px);
                    ny = xyz2(py);
                    nz = xyz2(pz);
                    nw = __ldcg(reinterpret_cast<const float2 *>(pw));
                }
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const f32x2 yx = j ? pack2(cx.y, cx.y) : pack2(cx.x, cx.x), yy = j ? pack2(cy.y, cy.y) : pack2(cy.x, cy.x);
                    const f32x2 yz = j ? pack2(cz.y, cz.y) : pack2(cz.x, cz.x), w = j ? pack2(cw.y, cw.y) : pack2(cw.x, cw.x);
#pragma unroll
                    for (int h = 0; h < H; h++) {
                        // (the shift before the last product: the sum it leaves is near 0)
                        const float2 z = unpack2(fma2(qx[h], yx, add2(fma2(qy[h], yy, fma2(qz[h], yz, w)), shift[h])));
                        sum[h] = add2(sum[h], pack2(fast_exp2(z.x), fast_exp2(z.y)));
                    }
                }
            }
            // 32 lanes x kPcOwn sums -> lane l the total of own point l / kPcShare
            float s[kPcOwn];
#pragma unroll
            for (int h = 0; h < H; h++) {
                const float2 v = unpack2(sum[h]);
                s[2 * h] = v.x;
                s[2 * h + 1] = v.y;
            }
#pragma unroll
            for (int half = kPcOwn / 2; half; half >>= 1) {
                const bool up = lane & (kPcShare * half);
#pragma unroll
                for (int q = 0; q < half; q++) {
                    const float give = up ? s[q] : s[q + half], keep = up ? s[q + half] : s[q];
                    s[q] = keep + __shfl_xor_sync(0xffffffffu, give, kPcShare * half);
                }
            }
            float tot = s[0];
#pragma unroll
            for (int o = kPcShare / 2; o; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
            record_shift(old, r2, k, &rest);
            pot = fmaf(-a.eps * kLn2, log2f(tot) + rest, old);
            ok = !valid || (tot >= 0x1p-60f && tot <= 0x1p100f);
        }
        if (!__all_sync(0xffffffffu, ok)) {
            const float lse = running_lse(orec, own.stride, other.rec + (int64_t)T.other * kPcTile, other.stride,
                                               T.rounds * kPcTile, k);
            pot = r2 - lse / k;
        }
        float e = 0.f;
        if (valid && lane % kPcShare == 0) {
            float *rec = own.rec + T.own_rec + mine;
            own.pot[T.own0 + mine] = pot;
            rec[3 * own.stride] = record_w(pot, lw, r2, k);
            rec[4 * own.stride] = record_shift(pot, r2, k, &rest);
            if (check) e = expf(lw) * fabsf(expm1f((old - pot) / a.eps));
        }
        if (check) {
            for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
            if (lane == 0) atomicAdd(&a.err[T.prob], e);
        }
        if (id < 0) break;
        T = N;
    }
}

// Items and records of the points of every row tile, then of every column tile (one per
// block of 64 threads).  The potentials start where the reference's log_u = log_v = 0 does,
// in dual-potential form f = -eps log a, g = -eps log b.
__global__ void __launch_bounds__(kPcTile) pc_setup_kernel(PcArgs a, const int *tile_prob, PcItem *items) {
    const int t = blockIdx.x, i = threadIdx.x;
    const int p = tile_prob[t];
    const PcProblem P = a.prob[p];
    const bool row = t < a.row_tiles;
    const PcSide S = a.side[row ? 0 : 1];
    const int count = row ? P.n : P.m, at = (row ? t - P.row_tile0 : t - a.row_tiles - P.col_tile0) * kPcTile + i;
    const int64_t point = (row ? P.x0 : P.y0) + at;
    const int64_t rec = (int64_t)(row ? t : t - a.row_tiles) * kPcTile + i;
    float x = 0.f, y = 0.f, z = 0.f, w = -INFINITY, shift = 0.f;
    if (at < count) {
        if (at % kPcOwn == 0) {
            PcItem T;
            T.own0 = point;
            T.own_rec = rec;
            T.n_own = min(kPcOwn, count - at);
            T.other = row ? P.col_tile0 : P.row_tile0;
            T.rounds = ((row ? P.m : P.n) + kPcTile - 1) / kPcTile;
            T.prob = p;
            items[(row ? P.row_item0 : a.row_items + P.col_item0) + at / kPcOwn] = T;
        }
        const float *q = S.pts + 3 * point;
        x = q[0] - P.ox;
        y = q[1] - P.oy;
        z = q[2] - P.oz;
        const float lw = S.lw[point], pot = -a.eps * lw, r2 = fmaf(x, x, fmaf(y, y, z * z)), k = kLog2e / a.eps;
        float rest;
        S.pot[point] = pot;
        w = record_w(pot, lw, r2, k);
        shift = record_shift(pot, r2, k, &rest);
    }
    float *r = S.rec + rec;
    r[0] = x;
    r[S.stride] = y;
    r[2 * S.stride] = z;
    r[3 * S.stride] = w;
    r[4 * S.stride] = shift;
}

// Block-wide exclusive scan of one int per thread; returns the prefix and
// sets *total.
__device__ int block_exclusive_scan(int v, int *total, int *s_scan) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_scan[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int w = 0; w < kPcThreads / 32; w++) {
            const int t = s_scan[w];
            s_scan[w] = run;
            run += t;
        }
        s_scan[kPcThreads / 32] = run;
    }
    __syncthreads();
    const int res = s_scan[warp] + x - v;
    *total = s_scan[kPcThreads / 32];
    __syncthreads();
    return res;
}

// Rebuild the row/column item lists of the active problems, in the order of the first
// lists (one CTA).
__device__ void rebuild_lists(const PcArgs &a, int *s_scan) {
    int rows_run = 0, cols_run = 0;
    for (int base = 0; base < a.nprob; base += kPcThreads) {
        const int k = base + threadIdx.x;
        int nr = 0, nc = 0, r0 = 0, c0 = 0;
        if (k < a.nprob) {
            const int pr = a.row_order[k], pc = a.col_order[k];
            if (a.active[pr]) {
                nr = (a.prob[pr].n + kPcOwn - 1) / kPcOwn;
                r0 = a.prob[pr].row_item0;
            }
            if (a.active[pc]) {
                nc = (a.prob[pc].m + kPcOwn - 1) / kPcOwn;
                c0 = a.row_items + a.prob[pc].col_item0;
            }
        }
        int tr = 0, tc = 0;
        const int orr = block_exclusive_scan(nr, &tr, s_scan);
        const int oc = block_exclusive_scan(nc, &tc, s_scan);
        for (int q = 0; q < nr; q++) a.row_list[rows_run + orr + q] = r0 + q;
        for (int q = 0; q < nc; q++) a.col_list[cols_run + oc + q] = c0 + q;
        rows_run += tr;
        cols_run += tc;
    }
    if (threadIdx.x == 0) {
        a.ctl->n_row_list = rows_run;
        a.ctl->n_col_list = cols_run;
    }
}

__global__ void __launch_bounds__(kPcThreads, 2) pc_sinkhorn_kernel(const __grid_constant__ PcArgs a) {
    __shared__ int s_scan[kPcThreads / 32 + 1];
    const unsigned nblocks = gridDim.x;
    int it = 0;
    while (it < a.max_iter) {
        // without a stopping test only the last iteration has something to note
        const bool check = (a.threshold > 0.f && (it + 1) % a.check_every == 0) || it + 1 == a.max_iter;
        // f-update over the row items of the active problems, then g-update over the column
        // items (+ the column-marginal error on check iterations)
#pragma unroll 1
        for (int ph = 0; ph < 2; ph++) {
            half_iteration(a, a.side[ph], a.side[ph ^ 1], ph ? a.col_list : a.row_list,
                                ph ? *(volatile int *)&a.ctl->n_col_list : *(volatile int *)&a.ctl->n_row_list,
                                it == 0, check && ph);
            if (!grid_barrier_bounded(a.ctl, nblocks, a.status, a.spin_limit)) return;
        }
        it++;
        if (check) {
            if (blockIdx.x == 0) {
                for (int p = threadIdx.x; p < a.nprob; p += kPcThreads) {
                    if (a.active[p] && ((a.threshold > 0.f && a.err[p] <= a.threshold) || it == a.max_iter)) {
                        a.active[p] = 0;
                        a.iters[p] = it;
                        atomicSub(&a.ctl->n_active, 1);
                    }
                    a.err[p] = 0.f;
                }
                __syncthreads();
                rebuild_lists(a, s_scan);
                __threadfence();
            }
            if (!grid_barrier_bounded(a.ctl, nblocks, a.status, a.spin_limit)) return;
            if (*(volatile int *)&a.ctl->n_active <= 0) break;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->iterations = it;
}

// Centroid of both clouds of every problem (one CTA per problem).
__global__ void __launch_bounds__(kPcThreads) pc_center_kernel(const float *x, const float *y, PcProblem *prob) {
    __shared__ float red[3][kPcThreads / 32];
    PcProblem &P = prob[blockIdx.x];
    float s[3] = {0.f, 0.f, 0.f};
    for (int i = threadIdx.x; i < P.n; i += kPcThreads)
        for (int d = 0; d < 3; d++) s[d] += x[3 * (P.x0 + i) + d];
    for (int j = threadIdx.x; j < P.m; j += kPcThreads)
        for (int d = 0; d < 3; d++) s[d] += y[3 * (P.y0 + j) + d];
    for (int d = 0; d < 3; d++) {
        for (int o = 16; o; o >>= 1) s[d] += __shfl_xor_sync(0xffffffffu, s[d], o);
        if ((threadIdx.x & 31) == 0) red[d][threadIdx.x >> 5] = s[d];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float t[3] = {0.f, 0.f, 0.f};
        for (int w = 0; w < kPcThreads / 32; w++)
            for (int d = 0; d < 3; d++) t[d] += red[d][w];
        const float inv = 1.f / (float)(P.n + P.m);
        P.ox = t[0] * inv;
        P.oy = t[1] * inv;
        P.oz = t[2] * inv;
    }
}

// Regularised cost per problem: sum_i a_i f_i + sum_j b_j g_j (fp64 sums).
__global__ void __launch_bounds__(kPcThreads) pc_cost_kernel(const float *f, const float *g, const float *la,
                                                             const float *lb, const PcProblem *prob, double *cost) {
    __shared__ double red[kPcThreads / 32];
    const PcProblem P = prob[blockIdx.x];
    double s = 0.0;
    for (int i = threadIdx.x; i < P.n; i += kPcThreads) s += exp((double)la[P.x0 + i]) * f[P.x0 + i];
    for (int j = threadIdx.x; j < P.m; j += kPcThreads) s += exp((double)lb[P.y0 + j]) * g[P.y0 + j];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kPcThreads / 32; w++) t += red[w];
        cost[blockIdx.x] = t;
    }
}

// Gradient of the regularised cost w.r.t. one cloud (envelope theorem):
// d/dp_i = scale_p * 2 sum_j P_ij (p_i - q_j), P_ij = exp((f_i + g_j - C_ij)/eps
// + log a_i + log b_j) recomputed per pair.  The same 64-point tiles, 16 lanes to 4
// points, partner points staged in shared memory.
__global__ void __launch_bounds__(kPcThreads) pc_grad_kernel(const float *own_pts, const float *other_pts,
                                                             const float *own_pot, const float *other_pot,
                                                             const float *own_lw, const float *other_lw,
                                                             const PcProblem *prob, int nprob, int tiles, bool rows,
                                                             float eps, const float *scale, float *grad) {
    __shared__ float4 s_part[kPcGradChunk];
    __shared__ float s_lw[kPcGradChunk];
    const float k = kLog2e / eps;
    const int grp = threadIdx.x / kPcLanes, lane = threadIdx.x % kPcLanes;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int p = find_problem(prob, nprob, tile, rows);
        const PcProblem P = prob[p];
        const int64_t o0 = rows ? P.x0 : P.y0, q0 = rows ? P.y0 : P.x0;
        const int n_own = rows ? P.n : P.m, n_other = rows ? P.m : P.n;
        const int first = (tile - (rows ? P.row_tile0 : P.col_tile0)) * kPcTile;
        float px[kPcRep], py[kPcRep], pz[kPcRep], pot[kPcRep], lw[kPcRep], ax[kPcRep], ay[kPcRep], az[kPcRep];
#pragma unroll
        for (int q = 0; q < kPcRep; q++) {
            const int i = first + grp + kPcGroups * q;
            const bool v = i < n_own;
            px[q] = v ? own_pts[3 * (o0 + i)] : 0.f;
            py[q] = v ? own_pts[3 * (o0 + i) + 1] : 0.f;
            pz[q] = v ? own_pts[3 * (o0 + i) + 2] : 0.f;
            pot[q] = v ? own_pot[o0 + i] : 0.f;
            lw[q] = v ? own_lw[o0 + i] * kLog2e : -INFINITY;
            ax[q] = ay[q] = az[q] = 0.f;
        }
        for (int j0 = 0; j0 < n_other; j0 += kPcGradChunk) {
            const int cnt = min(kPcGradChunk, n_other - j0);
            for (int t = threadIdx.x; t < cnt; t += kPcThreads) {
                const int64_t j = q0 + j0 + t;
                s_part[t] = make_float4(other_pts[3 * j], other_pts[3 * j + 1], other_pts[3 * j + 2], other_pot[j]);
                s_lw[t] = other_lw[j] * kLog2e;
            }
            __syncthreads();
            for (int t = lane; t < cnt; t += kPcLanes) {
                const float4 pt = s_part[t];
                const float plw = s_lw[t];
#pragma unroll
                for (int q = 0; q < kPcRep; q++) {
                    const float dx = px[q] - pt.x, dy = py[q] - pt.y, dz = pz[q] - pt.z;
                    const float c = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                    // f + g - C first: the potentials and the cost nearly cancel where P is not tiny
                    const float pij = exp2f(fmaf(k, (pot[q] + pt.w) - c, lw[q] + plw));
                    ax[q] = fmaf(pij, dx, ax[q]);
                    ay[q] = fmaf(pij, dy, ay[q]);
                    az[q] = fmaf(pij, dz, az[q]);
                }
            }
            __syncthreads();
        }
        const float sc = 2.f * scale[p];
#pragma unroll
        for (int q = 0; q < kPcRep; q++) {
#pragma unroll
            for (int o = 1; o < kPcLanes; o <<= 1) {
                ax[q] += __shfl_xor_sync(0xffffffffu, ax[q], o);
                ay[q] += __shfl_xor_sync(0xffffffffu, ay[q], o);
                az[q] += __shfl_xor_sync(0xffffffffu, az[q], o);
            }
            const int i = first + grp + kPcGroups * q;
            if (lane == 0 && i < n_own) {
                grad[3 * (o0 + i)] = sc * ax[q];
                grad[3 * (o0 + i) + 1] = sc * ay[q];
                grad[3 * (o0 + i) + 2] = sc * az[q];
            }
        }
    }
}

// Tiles (64 points of one problem) and items (16) of a batch.
struct PcCounts {
    int64_t row_tiles = 0, col_tiles = 0, row_items = 0, col_items = 0;
};

PcCounts pc_counts(int64_t nprob, const int64_t *n, const int64_t *m) {
    PcCounts c;
    for (int64_t p = 0; p < nprob; p++) {
        c.row_tiles += ceil_div(n[p] > 0 ? n[p] : 0, kPcTile);
        c.col_tiles += ceil_div(m[p] > 0 ? m[p] : 0, kPcTile);
        c.row_items += ceil_div(n[p] > 0 ? n[p] : 0, kPcOwn);
        c.col_items += ceil_div(m[p] > 0 ? m[p] : 0, kPcOwn);
    }
    return c;
}

struct PcLayout {
    size_t prob, err, active, iters, ctl, tile_prob, order, row_list, col_list, items, rec[2], total;
};

PcLayout pc_layout(int64_t nprob, const PcCounts &c) {
    PcLayout L{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t at = off;
        off += (bytes + 255) / 256 * 256;
        return at;
    };
    // uploaded together: up to the item lists
    L.ctl = take(sizeof(PcControl));
    L.prob = take((size_t)nprob * sizeof(PcProblem));
    L.err = take((size_t)nprob * 4);
    L.active = take((size_t)nprob * 4);
    L.iters = take((size_t)nprob * 4);
    L.tile_prob = take((size_t)(c.row_tiles + c.col_tiles) * 4);
    L.order = take((size_t)nprob * 2 * 4);
    L.row_list = take((size_t)c.row_items * 4);
    L.col_list = take((size_t)c.col_items * 4);
    L.items = take((size_t)(c.row_items + c.col_items) * sizeof(PcItem));
    L.rec[0] = take((size_t)c.row_tiles * kPcTile * 5 * 4);
    L.rec[1] = take((size_t)c.col_tiles * kPcTile * 5 * 4);
    L.total = off;
    return L;
}

template <typename T>
T *ws_at(void *ws, size_t off) {
    return reinterpret_cast<T *>(static_cast<unsigned char *>(ws) + off);
}

int build_problems(int64_t nprob, const int64_t *n, const int64_t *m, std::vector<PcProblem> &out, int *row_tiles,
                   int *col_tiles, int64_t *nx, int64_t *ny) {
    out.resize(nprob);
    int64_t x0 = 0, y0 = 0, rt = 0, ct = 0;
    for (int64_t p = 0; p < nprob; p++) {
        if (n[p] < 1 || m[p] < 1) return fail(TM_ERR_INVALID_ARGUMENT, "problem %lld has an empty cloud", (long long)p);
        if (n[p] > (1 << 24) || m[p] > (1 << 24)) return fail(TM_ERR_TOO_LARGE, "clouds are limited to 2^24 points");
        out[p].x0 = x0;
        out[p].y0 = y0;
        out[p].n = (int)n[p];
        out[p].m = (int)m[p];
        out[p].row_tile0 = (int)rt;
        out[p].col_tile0 = (int)ct;
        x0 += n[p];
        y0 += m[p];
        rt += ceil_div(n[p], kPcTile);
        ct += ceil_div(m[p], kPcTile);
        if (rt >= (1 << 30) || ct >= (1 << 30)) return fail(TM_ERR_TOO_LARGE, "too many tiles");
    }
    *row_tiles = (int)rt;
    *col_tiles = (int)ct;
    *nx = x0;
    *ny = y0;
    return TM_OK;
}

}  // namespace
}  // namespace tmc

extern "C" size_t tm_pointcloud_sinkhorn_workspace_size(int64_t n_problems, const int64_t *n, const int64_t *m,
                                                        int64_t max_iter) {
    using namespace tmc;
    if (n_problems < 1 || max_iter < 1 || !n || !m) return 0;
    return pc_layout(n_problems, pc_counts(n_problems, n, m)).total;
}

extern "C" int tm_pointcloud_sinkhorn(const float *x, const float *y, const float *log_a, const float *log_b,
                                      int64_t n_problems, const int64_t *n, const int64_t *m, double epsilon,
                                      int64_t max_iter, double threshold, int64_t check_every, float *f, float *g,
                                      double *cost, int32_t *iterations, void *workspace, size_t workspace_bytes,
                                      tm_stream_t stream) {
    using namespace tmc;
    if (!x || !y || !log_a || !log_b || !f || !g || !n || !m)
        return fail(TM_ERR_INVALID_ARGUMENT, "NULL argument");
    if (n_problems < 1 || n_problems > (1 << 24)) return fail(TM_ERR_INVALID_ARGUMENT, "n_problems must be 1..2^24");
    if (!(epsilon > 0)) return fail(TM_ERR_INVALID_ARGUMENT, "epsilon must be positive");
    if (max_iter < 1 || max_iter > (1 << 24)) return fail(TM_ERR_INVALID_ARGUMENT, "max_iter must be 1..2^24");
    if (check_every < 1) return fail(TM_ERR_INVALID_ARGUMENT, "check_every must be positive");
    std::vector<PcProblem> probs;
    int row_tiles = 0, col_tiles = 0;
    int64_t nx = 0, ny = 0;
    int st = build_problems(n_problems, n, m, probs, &row_tiles, &col_tiles, &nx, &ny);
    if (st != TM_OK) return st;
    const PcCounts c = pc_counts(n_problems, n, m);
    if (c.row_items + c.col_items >= (1LL << 31)) return fail(TM_ERR_TOO_LARGE, "too many items");
    const PcLayout L = pc_layout(n_problems, c);
    if (!workspace || workspace_bytes < L.total)
        return fail(TM_ERR_WORKSPACE, "point-cloud Sinkhorn workspace of %zu bytes needed", L.total);
    if ((uintptr_t)workspace & 255) return fail(TM_ERR_INVALID_ARGUMENT, "workspace must be 256-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    // control block, problems, zeroed errors and iteration counts, every problem active, tile
    // problems, the problems' orders by item cost and the first lists, in one upload
    std::vector<int64_t> up(L.items / 8, 0);
    auto *ctl = ws_at<PcControl>(up.data(), L.ctl);
    ctl->n_active = (int)n_problems;
    ctl->n_row_list = (int)c.row_items;
    ctl->n_col_list = (int)c.col_items;
    for (int64_t p = 0, r = 0, q = 0; p < n_problems; p++) {
        probs[p].row_item0 = (int)r;
        probs[p].col_item0 = (int)q;
        r += ceil_div(n[p], kPcOwn);
        q += ceil_div(m[p], kPcOwn);
    }
    std::copy(probs.begin(), probs.end(), ws_at<PcProblem>(up.data(), L.prob));
    std::fill_n(ws_at<int>(up.data(), L.active), n_problems, 1);
    int *tile_prob = ws_at<int>(up.data(), L.tile_prob), *order = ws_at<int>(up.data(), L.order);
    int *row_list = ws_at<int>(up.data(), L.row_list), *col_list = ws_at<int>(up.data(), L.col_list);
    for (int64_t p = 0; p < n_problems; p++) {
        std::fill_n(tile_prob + probs[p].row_tile0, ceil_div(n[p], kPcTile), (int)p);
        std::fill_n(tile_prob + row_tiles + probs[p].col_tile0, ceil_div(m[p], kPcTile), (int)p);
        order[p] = order[n_problems + p] = (int)p;
    }
    std::stable_sort(order, order + n_problems, [&](int a, int b) { return m[a] > m[b]; });
    std::stable_sort(order + n_problems, order + 2 * n_problems, [&](int a, int b) { return n[a] > n[b]; });
    for (int64_t k = 0; k < n_problems; k++) {
        const int pr = order[k], pc = order[n_problems + k];
        for (int64_t t = 0; t < ceil_div(n[pr], kPcOwn); t++) *row_list++ = probs[pr].row_item0 + (int)t;
        for (int64_t t = 0; t < ceil_div(m[pc], kPcOwn); t++) *col_list++ = (int)c.row_items + probs[pc].col_item0 + (int)t;
    }
    TM_CHECK_CUDA(cudaMemcpyAsync(workspace, up.data(), L.items, cudaMemcpyHostToDevice, s));
    auto *prob = ws_at<PcProblem>(workspace, L.prob);
    pc_center_kernel<<<(unsigned)n_problems, kPcThreads, 0, s>>>(x, y, prob);
    TM_LAUNCH_CHECK("pc_center_kernel");
    int *status = nullptr;
    if ((st = device_status_word(&status)) != TM_OK) return st;
    int per_sm = 0;
    TM_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pc_sinkhorn_kernel, kPcThreads, 0));
    if (per_sm < 1) return fail(TM_ERR_UNSUPPORTED, "point-cloud kernel does not fit on an SM");
    per_sm = per_sm > 4 ? 4 : per_sm;  // fewer CTAs make the grid barrier cheaper
    const int blocks = per_sm * sm_count();
    PcArgs args;
    args.side[0] = PcSide{x, log_a, f, ws_at<float>(workspace, L.rec[0]), (int64_t)row_tiles * kPcTile};
    args.side[1] = PcSide{y, log_b, g, ws_at<float>(workspace, L.rec[1]), (int64_t)col_tiles * kPcTile};
    args.prob = prob;
    args.nprob = (int)n_problems;
    args.row_tiles = row_tiles;
    args.row_items = (int)c.row_items;
    args.err = ws_at<float>(workspace, L.err);
    args.active = ws_at<int>(workspace, L.active);
    args.iters = ws_at<int>(workspace, L.iters);
    args.items = ws_at<PcItem>(workspace, L.items);
    args.row_order = ws_at<int>(workspace, L.order);
    args.col_order = args.row_order + n_problems;
    args.row_list = ws_at<int>(workspace, L.row_list);
    args.col_list = ws_at<int>(workspace, L.col_list);
    args.ctl = ws_at<PcControl>(workspace, L.ctl);
    args.status = status;
    args.eps = (float)epsilon;
    args.threshold = (float)threshold;
    args.max_iter = (int)max_iter;
    args.check_every = (int)check_every;
    args.spin_limit = grid_wait_budget();
    pc_setup_kernel<<<(unsigned)(row_tiles + col_tiles), kPcTile, 0, s>>>(
        args, ws_at<int>(workspace, L.tile_prob), ws_at<PcItem>(workspace, L.items));
    TM_LAUNCH_CHECK("pc_setup_kernel");
    void *params[] = {&args};
    TM_CHECK_CUDA(cudaLaunchCooperativeKernel((const void *)pc_sinkhorn_kernel, dim3(blocks), dim3(kPcThreads), params,
                                              0, s));
    TM_LAUNCH_CHECK("pc_sinkhorn_kernel");
    if (cost) {
        pc_cost_kernel<<<(unsigned)n_problems, kPcThreads, 0, s>>>(f, g, log_a, log_b, args.prob, cost);
        TM_LAUNCH_CHECK("pc_cost_kernel");
    }
    if (iterations)
        TM_CHECK_CUDA(cudaMemcpyAsync(iterations, args.iters, (size_t)n_problems * sizeof(int32_t),
                                      cudaMemcpyDeviceToDevice, s));
    return TM_OK;
}

extern "C" size_t tm_pointcloud_sinkhorn_grad_workspace_size(int64_t n_problems) {
    return n_problems < 1 ? 0 : (size_t)n_problems * sizeof(tmc::PcProblem);
}

extern "C" int tm_pointcloud_sinkhorn_grad(const float *x, const float *y, const float *log_a, const float *log_b,
                                           const float *f, const float *g, int64_t n_problems, const int64_t *n,
                                           const int64_t *m, double epsilon, const float *grad_cost, float *grad_x,
                                           float *grad_y, void *workspace, size_t workspace_bytes,
                                           tm_stream_t stream) {
    using namespace tmc;
    if (!x || !y || !log_a || !log_b || !f || !g || !n || !m || !grad_cost)
        return fail(TM_ERR_INVALID_ARGUMENT, "NULL argument");
    if (n_problems < 1 || n_problems > (1 << 24)) return fail(TM_ERR_INVALID_ARGUMENT, "n_problems must be 1..2^24");
    if (!(epsilon > 0)) return fail(TM_ERR_INVALID_ARGUMENT, "epsilon must be positive");
    const size_t need = (size_t)n_problems * sizeof(PcProblem);
    if (!workspace || workspace_bytes < need) return fail(TM_ERR_WORKSPACE, "gradient workspace of %zu bytes needed", need);
    std::vector<PcProblem> probs;
    int row_tiles = 0, col_tiles = 0;
    int64_t nx = 0, ny = 0;
    int st = build_problems(n_problems, n, m, probs, &row_tiles, &col_tiles, &nx, &ny);
    if (st != TM_OK) return st;
    cudaStream_t s = (cudaStream_t)stream;
    auto *dprob = static_cast<PcProblem *>(workspace);
    TM_CHECK_CUDA(cudaMemcpyAsync(dprob, probs.data(), need, cudaMemcpyHostToDevice, s));
    const int cap = sm_count() * 8;
    if (grad_x) {
        pc_grad_kernel<<<row_tiles < cap ? row_tiles : cap, kPcThreads, 0, s>>>(
            x, y, f, g, log_a, log_b, dprob, (int)n_problems, row_tiles, true, (float)epsilon, grad_cost, grad_x);
        TM_LAUNCH_CHECK("pc_grad_kernel");
    }
    if (grad_y) {
        pc_grad_kernel<<<col_tiles < cap ? col_tiles : cap, kPcThreads, 0, s>>>(
            y, x, g, f, log_b, log_a, dprob, (int)n_problems, col_tiles, false, (float)epsilon, grad_cost, grad_y);
        TM_LAUNCH_CHECK("pc_grad_kernel");
    }
    return TM_OK;
}
