// Separable EDT passes over tiles of lines (included by edt_compact.cu, inside
// its anonymous namespace).
//
// A squared distance is an exact integer here: axis a contributes w_a times the
// squared voxel offset (w_a = 1 for unit spacing; for spacings that are binary
// fractions n_a / 2^k, w_a = n_a^2 in units of 4^-k).  Pass 0 (axis 0) gives every
// voxel the nearest background along its column; a later pass computes, for every
// position q of every line along its axis,
//     argmin_p  g(p) + w (q - p)^2,   the lowest p on a tie,
// g(p) = the best squared distance of the passes before.
//
//  * Windows first: |q - p| <= 4, and where a warp needs it the rings up to 12 and 28
//    around it.  A window is exact when its best value is below w (K + 1)^2.  A
//    candidate is the 32-bit key value << 6 | position, so it costs one fused add-min
//    and a tie goes to the lowest position; a thread takes 8 adjacent q, so a staged
//    value is read once for up to 8 candidates.
//  * A position left open whose window bounds the answer to less than 64 voxels walks on
//    outwards by itself.  The others (large objects, sparse backgrounds) are halved: the argmin is
//    monotone in q (for p1 < p2, f(q, p1) - f(q, p2) grows with q; ties to the lowest
//    keep it monotone), so once every second position of a grid of stride 2s is known,
//    the ones between only search the interval of their neighbours' positions, cut
//    further to the radius their window's value allows.  A level costs about one
//    candidate per voxel and every voxel of a level is independent: no serial chain
//    per line, whatever the distances are.  (The lower-envelope passes this replaces
//    ran one thread per line.)
//
// Bound: issue (about 190 instructions per voxel and pass on masks) and the latency of
// the list phases, not memory: 8 x 1000 x 1333 masks, distances alone, move 64 MB in
// 98 us.  Before (one thread, or one warp's lane 0, per line's envelope): 1217 us; 2 x 88 x
// 180 x 214 at spacing (2.5, 1, 1) 1152 -> 126 us; 4 x 128^3 with features, masks 748 ->
// 275 us, Bernoulli(0.99) 629 -> 239 us.  Windows decided per warp instead of by lists
// (a warp runs the widest ring any of its lanes needs) took 138 us on the 2-D masks;
// open positions walked inside their group's thread 121 us.
//
// Dense backgrounds take the first window alone, and there the instructions around it count:
// a tile without an open group skips the lists and reads its distances, all below the window's
// bound, from a table.  FLAT tiles (modes 0 and 2) stage and write their lines, adjacent rows,
// as one run of positions, the others in units of 128 positions of a line: the flat form
// divides by the line length for every position, the units idle in a line's last one.
// Bernoulli(0.5), distances alone, one thread or warp per line -> units and lists for all ->
// now: 64 x 256^2 21.3 -> 28.1 -> 25.4 us, 64 x 250 x 512 (3-D) 32.0 -> 48.6 -> 38.1, 4 x 128
// x 128 x 130 91.5 -> 117.7 -> 85.9 (units there 93.6), 8 x 64 x 64 x 63 30.6 -> 32.7 -> 25.9;
// 64 x 128^2 11.1 -> 15.6 -> 12.5 (tiles of 16 lines; of 32: 14.4).
constexpr int kLineQ = 8;        // positions per thread and window step
constexpr int kLineK1 = 4;       // window radii
constexpr int kLineK2 = 12;
constexpr int kLineK3 = 28;      // = padding of a staged line; kLineQ + 2 K3 positions fit 6 bits
constexpr int kLineFar = 64;     // a position whose bound is nearer than this is searched directly
constexpr int kLineShift = 6;    // key = value << 6 | window position
constexpr uint32_t kLineClamp = 1u << 25;  // larger values are unresolved by any window
constexpr uint16_t kLineOpen = 0x8000;     // position not final yet
constexpr int kMaxWeight = 1 << 15;        // largest w: w (K3 + 1)^2 stays below the clamp

// Whether the shell search left any item to the passes (one read of the flags, by all
// threads of the CTA).
__device__ __forceinline__ bool any_todo(const int *todo, int64_t batch) {
    const int tid = threadIdx.x + threadIdx.y * blockDim.x, threads = blockDim.x * blockDim.y;
    bool left = false;
    for (int64_t i = tid; i < batch; i += threads) left |= __ldcg(todo + i) != 0;
    return __syncthreads_or(left);
}

// ------------------------------------------------------------------ pass 0
// Nearest background along axis 0 as its position f0 (-1: none), ties to the lower.
// A warp takes 32 rows of 32 CPL adjacent columns and packs them into a background word
// per column (bit r = row 32 w + r); the words of all rows of the columns meet in
// shared memory, and a voxel finds its neighbours by count-leading-zeros in its word
// or in the nearest non-zero words above and below.  Every input byte is read once,
// every step is parallel over rows as well as columns.  CPL = 4 adjacent columns per
// lane (4-byte loads, 8-byte stores) where rows are aligned and there are enough
// columns to fill the SMs, else 1.
constexpr int kBitsWarps = 16;  // per CTA: a warp per 32 rows, as many column blocks as fit

template <typename In, int CPL>
__global__ void __launch_bounds__(32 * kBitsWarps) edt_bits0_kernel(const In *__restrict__ in,
                                                                    int16_t *__restrict__ c1, CompactParams p,
                                                                    const int *__restrict__ todo) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kCols = 32 * CPL;
    constexpr int kRows = CPL == 1 ? 16 : 8;  // rows loaded at a time
    pdl_wait();     // launched after the shell search: its flags are complete
    pdl_trigger();  // the line passes may be scheduled now: the flags they read are final
    if (todo && !any_todo(todo, p.batch)) return;
    const int L = p.L0, nw = (L + 31) / 32;
    const int64_t inner = p.numel_item / L;
    // blockDim.y column blocks to a CTA, all of one item
    const int64_t cblocks = (inner + kCols * blockDim.y - 1) / (kCols * blockDim.y), nblk = p.batch * cblocks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    uint32_t *words = reinterpret_cast<uint32_t *>(smem_raw) + (size_t)threadIdx.y * nw * kCols;  // [nw][kCols]
    for (int64_t blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        const int64_t item = blk / cblocks;
        if (todo && !todo[item]) continue;  // finished by the shell search
        const int64_t c0 = ((blk - item * cblocks) * blockDim.y + threadIdx.y) * kCols + CPL * lane;
        const bool live = c0 < inner;  // (CPL = 4: inner is a multiple of 4)
        const In *src = in + item * p.numel_item + c0;
        int16_t *out = c1 + item * p.numel_item + c0;
        for (int w = warp; w < nw; w += warps) {
            uint32_t bits[CPL];
#pragma unroll
            for (int k = 0; k < CPL; k++) bits[k] = 0u;
#pragma unroll 1
            for (int r0 = 0; r0 < 32 && 32 * w + r0 < L; r0 += kRows) {
                In v[kRows][CPL];
#pragma unroll
                for (int r = 0; r < kRows; r++) {
                    const int y = 32 * w + r0 + r;
                    const bool ok = live && y < L;
                    const In *row = src + (int64_t)y * inner;
                    if (CPL == 1) {
                        v[r][0] = ok ? row[0] : (In)1;
                    } else if (sizeof(In) == 1) {
                        const uint32_t q = ok ? *reinterpret_cast<const uint32_t *>(row) : 0x01010101u;
#pragma unroll
                        for (int k = 0; k < CPL; k++) v[r][k] = (In)((q >> (8 * k)) & 255u);
                    } else {
                        const float4 q = ok ? *reinterpret_cast<const float4 *>(row) : make_float4(1, 1, 1, 1);
                        const float e[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                        for (int k = 0; k < CPL; k++) v[r][k] = (In)e[k];
                    }
                }
#pragma unroll
                for (int r = 0; r < kRows; r++)
#pragma unroll
                    for (int k = 0; k < CPL; k++) bits[k] |= (uint32_t)(v[r][k] == (In)0) << (r0 + r);
            }
#pragma unroll
            for (int k = 0; k < CPL; k++) words[w * kCols + CPL * lane + k] = bits[k];
        }
        __syncthreads();
        for (int w = warp; w < nw; w += warps) {
            uint32_t bits[CPL];
            int before[CPL], after[CPL];
#pragma unroll
            for (int k = 0; k < CPL; k++) {
                const uint32_t *col = words + CPL * lane + k;
                bits[k] = col[w * kCols];
                before[k] = after[k] = -1;
                for (int u = w - 1; u >= 0; u--) {
                    const uint32_t b = col[u * kCols];
                    if (b) {
                        before[k] = 32 * u + 31 - __clz(b);
                        break;
                    }
                }
                for (int u = w + 1; u < nw; u++) {
                    const uint32_t b = col[u * kCols];
                    if (b) {
                        after[k] = 32 * u + __ffs(b) - 1;
                        break;
                    }
                }
            }
#pragma unroll 8
            for (int r = 0; r < 32; r++) {
                const int y = 32 * w + r;
                if (y >= L) break;
                int16_t f[CPL];
#pragma unroll
                for (int k = 0; k < CPL; k++) {
                    const uint32_t lo = bits[k] << (31 - r), hi = bits[k] >> r;  // rows <= y, rows >= y
                    const int prev = lo ? y - __clz(lo) : before[k], next = hi ? y + __ffs(hi) - 1 : after[k];
                    f[k] = (int16_t)((prev >= 0 && (next < 0 || y - prev <= next - y)) ? prev : next);
                }
                int16_t *row = out + (int64_t)y * inner;
                if (CPL == 4) {
                    if (live) *reinterpret_cast<short4 *>(row) = make_short4(f[0], f[CPL / 4], f[CPL / 2], f[CPL - 1]);
                } else if (live) {
                    row[0] = f[0];
                }
            }
        }
        __syncthreads();  // the words are rewritten by the next block
    }
}

// -------------------------------------------------------------- later passes
// MODE 0: last axis of 2-D items (input f0).  MODE 1: axis 1 of 3-D items (input f0,
// output (f0 | f1 << 16), -1 for none).  MODE 2: last axis of 3-D items (input the
// output of MODE 1).  Modes 0 and 2 write the results (OUT 0: the distances alone).
struct LineTile {
    int lines, pitch, ppitch;  // lines per tile, words of a staged line, entries of its positions
    int blocks;                // groups of kLineQ positions per line
    size_t pos, any, todo, total;
};

// Staged lines are 1 word more than a multiple of 32 apart: the threads of a warp read
// one position of 32 lines, or positions 8 apart of 8 lines, without bank conflicts.
__host__ __device__ inline LineTile line_tile(int lines, int L) {
    LineTile t;
    t.lines = lines;
    t.pitch = (L + 2 * kLineK3 + kLineQ + 31) / 32 * 32 + 1;
    t.ppitch = (L + 63) / 64 * 64 + 8;  // groups of 8 positions of 8 lines: 16 bytes in distinct banks
    t.pos = (size_t)lines * t.pitch * 4;
    t.any = t.pos + ((size_t)lines * t.ppitch * 2 + 15) / 16 * 16;
    t.blocks = (L + kLineQ - 1) / kLineQ;
    t.todo = t.any + ((size_t)lines + 4) * 4;  // (the list counters behind the flags)
    t.total = t.todo + (size_t)2 * lines * t.blocks * 2;
    return t;
}

// Candidates at distance LO < |q - p| <= HI of the 8 positions from q0 on: key[i] of position
// q0 + i; c[k] = (weight k^2) << kLineShift.  Position code: p - q0 + K3.
template <int LO, int HI>
__device__ __forceinline__ void line_ring(const uint32_t *g, const uint32_t *c, uint32_t (&key)[kLineQ]) {
#pragma unroll
    for (int j = -HI; j < kLineQ + HI; j++) {
        bool used = false;
#pragma unroll
        for (int i = 0; i < kLineQ; i++) {
            const int k = j < i ? i - j : j - i;
            used = used || (k > LO && k <= HI);
        }
        if (!used) continue;
        const uint32_t w = (min(g[j], kLineClamp) << kLineShift) + (uint32_t)(j + kLineK3);
#pragma unroll
        for (int i = 0; i < kLineQ; i++) {
            const int k = j < i ? i - j : j - i;
            if (k > LO && k <= HI) key[i] = __viaddmin_u32(w, c[k], key[i]);
        }
    }
}

template <int MODE, int NL, int T, int OUT, bool FLAT>
__global__ void __launch_bounds__(T, 1024 / T) edt_line_kernel(const void *__restrict__ src, int32_t *__restrict__ c2,
                                                                float *__restrict__ dist,
                                                                int32_t *__restrict__ indices,
                                                                int32_t *__restrict__ sqdist, CompactParams p,
                                                                const int *__restrict__ todo) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kSlots = T / NL;
    // list entries: line and group of 8 positions, line and position (32 lines reach 1024
    // positions, 16 reach 2048, 8 reach 4096)
    constexpr int kPosBits = NL == 32 ? 10 : (NL == 16 ? 11 : 12), kPosMask = (1 << kPosBits) - 1;
    constexpr int kTaskBits = kPosBits - 3, kTaskMask = (1 << kTaskBits) - 1;
    const int L = MODE == 2 ? p.L2 : p.L1;
    const LineTile tl = line_tile(NL, L);
    uint32_t *g = reinterpret_cast<uint32_t *>(smem_raw);
    uint16_t *pos = reinterpret_cast<uint16_t *>(smem_raw + tl.pos);
    int *any = reinterpret_cast<int *>(smem_raw + tl.any), *count = any + NL;
    uint16_t *list = reinterpret_cast<uint16_t *>(smem_raw + tl.todo);  // [2][NL * blocks]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int line = tid % NL, slot = tid / NL;
    // lines of an item: rows (modes 0, 2), columns of every plane (mode 1: W per plane,
    // NL adjacent ones to a tile)
    const int W = MODE == 1 ? p.L2 : 1;
    const int tiles_x = MODE == 1 ? (W + NL - 1) / NL : 1;
    const int rows = MODE == 0 ? p.L0 : p.L0 * p.L1;
    const int64_t tiles = MODE == 1 ? (int64_t)p.L0 * tiles_x : (rows + NL - 1) / NL;
    __shared__ float root[kSqrtTab];  // distances of small values (barriers follow)
    __shared__ int at[NL];            // FLAT, mode 2: z << 16 | y of a line
    if (MODE != 1 && tid < kSqrtTab) root[tid] = line_dist(tid, p.unit2);
    const uint32_t weight = MODE == 2 ? p.w2 : p.w1, w0 = p.w0, w1 = p.w1;
    const float inv_weight = 1.0f / (float)weight;
    const uint32_t far_limit = min(weight * (uint32_t)(kLineFar * kLineFar), kBig);
    uint32_t cw[kLineK3 + 1];
#pragma unroll
    for (int k = 0; k <= kLineK3; k++) cw[k] = (weight * (uint32_t)(k * k)) << kLineShift;
    pdl_trigger();
    const bool idle = todo && !any_todo(todo, p.batch);
    pdl_wait();  // the pass before is complete (also when idle: a grid never completes before it)
    if (idle) return;
    for (int64_t blk = blockIdx.x; blk < p.batch * tiles; blk += gridDim.x) {
        const int64_t item = blk / tiles;
        if (todo && !__ldcg(todo + item)) continue;  // finished by the shell search
        const int t = (int)(blk - item * tiles);
        const int z1 = MODE == 1 ? t / tiles_x : 0, x0 = MODE == 1 ? (t - z1 * tiles_x) * NL : 0;  // mode 1
        const int row0 = MODE == 1 ? 0 : t * NL;                                                  // modes 0, 2
        const int nlines = MODE == 1 ? min(NL, W - x0) : min(NL, rows - row0);
        const int64_t base = item * p.numel_item + (MODE == 1 ? (int64_t)z1 * L * W + x0 : (int64_t)row0 * L);
        // g of position q of a line; -1 marks "no site"
        auto value0 = [&](int f0, int z) -> uint32_t {
            return f0 < 0 ? kBig : w0 * (uint32_t)((z - f0) * (z - f0));
        };
        auto value01 = [&](int32_t f, int z, int y) -> uint32_t {
            const int f0 = (int16_t)(f & 0xffff), f1 = f >> 16;
            return f0 < 0 ? kBig : w0 * (uint32_t)((z - f0) * (z - f0)) + w1 * (uint32_t)((y - f1) * (y - f1));
        };
        if (tid < NL) {
            any[tid] = 0;
            if (MODE == 2 && FLAT) {
                const int z = (int)fdiv(row0 + tid, p.d_l1);
                at[tid] = z << 16 | (row0 + tid - z * p.L1);
            }
        }
        if (tid < 3) count[tid] = 0;
        __syncthreads();
        // ---- stage
        if (MODE == 1) {
            bool have = false;
            for (int y0 = slot; y0 < L; y0 += 4 * kSlots) {
                int f[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int y = y0 + r * kSlots;
                    f[r] = y < L && line < nlines
                               ? (int)reinterpret_cast<const int16_t *>(src)[base + (int64_t)y * W + line]
                               : -1;
                }
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int y = y0 + r * kSlots;
                    if (y < L) g[line * tl.pitch + kLineK3 + y] = value0(f[r], z1);
                    have |= f[r] >= 0;
                }
            }
            if (have) any[line] = 1;
        } else if (FLAT) {
            // the tile's lines are adjacent rows: flat positions, 4 loads in flight
            for (int e0 = tid; e0 < nlines * L; e0 += 4 * T) {
                int32_t f[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    f[r] = -1;
                    if (e0 + r * T < nlines * L)
                        f[r] = MODE == 2 ? reinterpret_cast<const int32_t *>(src)[base + (e0 + r * T)]
                                         : (int32_t) reinterpret_cast<const int16_t *>(src)[base + (e0 + r * T)];
                }
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int e = e0 + r * T;
                    if (e >= nlines * L) break;
                    const int l = (int)fdiv(e, p.d_line);
                    const uint32_t v = MODE == 2 ? value01(f[r], at[l] >> 16, at[l] & 0xffff) : value0(f[r], row0 + l);
                    g[e + l * (tl.pitch - L) + kLineK3] = v;
                    if (v < kBig) any[l] = 1;
                }
            }
        } else {
            // units of 128 positions of a line, one warp each
            const int segs = (L + 127) / 128;
            for (int l = 0, seg = warp;; seg += T / 32) {
                while (seg >= segs) seg -= segs, l++;
                if (l >= nlines) break;
                const int q0 = seg * 128 + lane;
                const int row = row0 + l;
                const int z = MODE == 2 ? row / p.L1 : 0, y = MODE == 2 ? row - z * p.L1 : row;
                const int64_t o = base + (int64_t)l * L + q0;
                uint32_t *gr = g + l * tl.pitch + kLineK3 + q0;
                int32_t f[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    f[r] = -1;
                    if (q0 + 32 * r < L)
                        f[r] = MODE == 2 ? reinterpret_cast<const int32_t *>(src)[o + 32 * r]
                                         : (int32_t) reinterpret_cast<const int16_t *>(src)[o + 32 * r];
                }
                bool have = false;
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const uint32_t v = MODE == 2 ? value01(f[r], z, y) : value0(f[r], y);
                    if (q0 + 32 * r < L) gr[32 * r] = v;
                    have |= v < kBig;
                }
                if (have) any[l] = 1;
            }
        }
        for (int i = tid; i < NL * (2 * kLineK3 + kLineQ); i += T) {
            const int l = i % NL, k = i / NL;
            g[l * tl.pitch + (k < kLineK3 ? k : L + k)] = kBig;
        }
        __syncthreads();
        // ---- windows: the first for every group of 8 positions, the wider ones for the
        // groups on a list (full warps whatever the masks look like)
        const uint32_t *gl = g + line * tl.pitch + kLineK3;
        uint16_t *pl = pos + line * tl.ppitch;
        const bool live = line < nlines && any[line];
        // the largest key of the group's positions inside the line
        auto worst = [&](uint32_t(&key)[kLineQ], int q0) {
            if (q0 + kLineQ > L) {
#pragma unroll
                for (int i = 0; i < kLineQ; i++)
                    if (q0 + i >= L) key[i] = 0u;
            }
            return max(max(max(key[0], key[1]), max(key[2], key[3])), max(max(key[4], key[5]), max(key[6], key[7])));
        };
        auto exact = [&](int K) { return (weight * (uint32_t)((K + 1) * (K + 1))) << kLineShift; };
        // positions q0 - K3 + code of the group's 8, one 16-byte store
        auto store = [&](const uint32_t(&key)[kLineQ], uint16_t *to, int q0) {
            const uint32_t base2 = (uint32_t)(q0 - kLineK3) * 0x10001u;  // (a code below K3 - q0 is padding: unused)
            uint4 v;
            uint32_t *o = &v.x;
#pragma unroll
            for (int i = 0; i < kLineQ; i += 2) o[i / 2] = ((key[i] & 63u) | ((key[i + 1] & 63u) << 16)) + base2;
            *reinterpret_cast<uint4 *>(to + q0) = v;
        };
        // appends the tasks of the calling threads (a group of lanes with one atomic)
        auto append = [&](int which, bool wanted, int task) {
            const unsigned active = __activemask(), want = __ballot_sync(active, wanted);
            if (!want) return;
            const int leader = __ffs(want) - 1;
            int at = 0;
            if (lane == leader) at = atomicAdd(&count[which], __popc(want));
            at = __shfl_sync(active, at, leader);
            if (wanted) list[which * NL * tl.blocks + at + __popc(want & ((1u << lane) - 1u))] = (uint16_t)task;
        };
        bool wider = line < nlines && !any[line];
        for (int qb = slot; qb < tl.blocks; qb += kSlots) {
            const int q0 = qb * kLineQ;
            uint32_t key[kLineQ];
#pragma unroll
            for (int i = 0; i < kLineQ; i++) key[i] = 0xffffffffu;
            line_ring<-1, kLineK1>(gl + q0, cw, key);
            const uint32_t most = worst(key, q0);
            store(key, pl, q0);
            const bool wanted = live && most >= exact(kLineK1);
            wider |= wanted;
            append(0, wanted, line << kTaskBits | qb);
        }
        // (most tiles of a dense background end here, every value below the window's bound)
        wider = __syncthreads_or(wider);
        if (wider) {
            for (int t = tid; t < count[0]; t += T) {
                const int task = list[t], l = task >> kTaskBits, q0 = (task & kTaskMask) * kLineQ;
                uint32_t key[kLineQ];
#pragma unroll
                for (int i = 0; i < kLineQ; i++) key[i] = 0xffffffffu;
                line_ring<-1, kLineK2>(g + l * tl.pitch + kLineK3 + q0, cw, key);
                const bool ok = worst(key, q0) < exact(kLineK2);
                if (ok) store(key, pos + l * tl.ppitch, q0);
                append(1, !ok, task);
            }
            __syncthreads();
            // the positions the widest window leaves open: one by one from here on (list 0 again)
            bool open = false;
            for (int t = tid; t < count[1]; t += T) {
                const int task = list[NL * tl.blocks + t], l = task >> kTaskBits, q0 = (task & kTaskMask) * kLineQ;
                const uint32_t *gt = g + l * tl.pitch + kLineK3;
                uint16_t *pt = pos + l * tl.ppitch;
                uint32_t key[kLineQ];
#pragma unroll
                for (int i = 0; i < kLineQ; i++) key[i] = 0xffffffffu;
                line_ring<-1, kLineK3>(gt + q0, cw, key);
                if (worst(key, q0) < exact(kLineK3)) {
                    store(key, pt, q0);
                    continue;
                }
#pragma unroll
                for (int i = 0; i < kLineQ; i++) {
                    if (q0 + i >= L) continue;
                    const int bp = min(max(q0 - kLineK3 + (int)(key[i] & 63u), 0), L - 1);  // (may point at padding)
                    bool done = key[i] < exact(kLineK3);
                    if (!done) {
                        const uint32_t bound = gt[bp] + weight * (uint32_t)((q0 + i - bp) * (q0 + i - bp));
                        const int at = bound < far_limit ? atomicAdd(&count[2], 1) : NL * tl.blocks;
                        if (at < NL * tl.blocks) list[at] = (uint16_t)(l << kPosBits | (q0 + i));
                        else open = true;
                    }
                    pt[q0 + i] = (uint16_t)(bp | (done ? 0 : kLineOpen));
                }
            }
            __syncthreads();
            for (int t = tid; t < min(count[2], NL * tl.blocks); t += T) {
                const int l = list[t] >> kPosBits, q = list[t] & kPosMask;
                const uint32_t *gt = g + l * tl.pitch + kLineK3 + q;
                uint16_t *pt = pos + l * tl.ppitch + q;
                int b = (*pt & (kLineOpen - 1)) - q;
                uint32_t best = gt[b] + weight * (uint32_t)(b * b);
                for (int k = kLineK3 + 1; weight * (uint32_t)(k * k) <= best; k++) {
                    const uint32_t d = weight * (uint32_t)(k * k);
                    const uint32_t left = q - k >= 0 ? gt[-k] + d : kBig;
                    const uint32_t right = q + k < L ? gt[k] + d : kBig;
                    if (left <= best) {  // equal: the lower position
                        best = left;
                        b = -k;
                    }
                    if (right < best) {
                        best = right;
                        b = k;
                    }
                }
                *pt = (uint16_t)(q + b);
            }
            // ---- halving, where a window left a position open
            if (__syncthreads_or(open)) {
                auto search = [&](int q, int lo, int hi) {
                    const int b = pl[q] & (kLineOpen - 1);
                    const uint32_t v0 = gl[b] + weight * (uint32_t)((q - b) * (q - b));
                    if (v0 < kBig) {  // nothing further than this can be better
                        const int r = (int)sqrtf((float)v0 * inv_weight) + 1;
                        lo = max(lo, q - r);
                        hi = min(hi, q + r);
                    }
                    uint32_t best = 0xffffffffu;
                    int bp = lo;
#pragma unroll 4
                    for (int pp = lo; pp <= hi; pp++) {
                        const uint32_t v = gl[pp] + weight * (uint32_t)((q - pp) * (q - pp));
                        if (v < best) {
                            best = v;
                            bp = pp;
                        }
                    }
                    pl[q] = (uint16_t)bp;
                };
                int s = 1;
                while (8 * s <= L) s *= 2;
                if (live)
                    for (int q = slot * s; q < L; q += kSlots * s)
                        if (pl[q] & kLineOpen) search(q, 0, L - 1);
                for (s >>= 1; s > 0; s >>= 1) {
                    __syncthreads();
                    if (live)
                        for (int q = s + 2 * s * slot; q < L; q += 2 * s * kSlots)
                            if (pl[q] & kLineOpen) search(q, pl[q - s], q + s < L ? pl[q + s] : L - 1);
                }
                __syncthreads();
            }
        }
        // ---- outputs
        const bool near = !wider && weight * ((kLineK1 + 1) * (kLineK1 + 1)) <= kSqrtTab;  // root holds every value
        if (MODE == 1) {
            if (line < nlines) {
                const bool site = any[line] != 0;
                for (int y = slot; y < L; y += kSlots) {
                    const int64_t o = base + (int64_t)y * W + line;
                    int32_t f = -1;
                    if (site) {
                        const int b = pl[y];
                        f = (int32_t)(uint16_t) reinterpret_cast<const int16_t *>(src)[base + (int64_t)b * W + line] |
                            (b << 16);
                    }
                    c2[o] = f;
                }
            }
        } else if (FLAT) {
            for (int e0 = tid; e0 < nlines * L; e0 += 4 * T) {
                int l[4], b[4];
                uint32_t v[4];
                bool site[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int e = min(e0 + r * T, nlines * L - 1);
                    l[r] = (int)fdiv(e, p.d_line);
                    b[r] = pos[e + l[r] * (tl.ppitch - L)];
                    site[r] = any[l[r]] != 0;
                    if (!site[r]) b[r] = 0;
                }
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int q = min(e0 + r * T, nlines * L - 1) - l[r] * L, d = q - b[r];
                    v[r] = g[l[r] * tl.pitch + kLineK3 + b[r]] + weight * (uint32_t)(d * d);
                    if (!site[r]) {  // no background in the item: the site (-1, 0, ...)
                        const int z = MODE == 2 ? at[l[r]] >> 16 : 0, y = MODE == 2 ? at[l[r]] & 0xffff : row0 + l[r];
                        v[r] = w0 * (uint32_t)(MODE == 2 ? (z + 1) * (z + 1) : (y + 1) * (y + 1)) +
                               (MODE == 2 ? w1 * (uint32_t)(y * y) : 0u) + weight * (uint32_t)(q * q);
                    }
                }
                if (dist) {
                    float d[4];
                    if (near) {
#pragma unroll
                        for (int r = 0; r < 4; r++) d[r] = root[min(v[r], kSqrtTab - 1u)];  // (beyond the line: any entry)
                    } else {
#pragma unroll
                        for (int r = 0; r < 4; r++) d[r] = line_dist(v[r], p.unit2);
                    }
#pragma unroll
                    for (int r = 0; r < 4; r++)
                        if (e0 + r * T < nlines * L) __stcs(dist + base + (e0 + r * T), d[r]);
                }
                if (OUT == 0) continue;  // distances only
                if (sqdist) {
#pragma unroll
                    for (int r = 0; r < 4; r++)
                        if (e0 + r * T < nlines * L) __stcs(sqdist + base + (e0 + r * T), (int32_t)v[r]);
                }
                if (indices) {
                    int32_t f[4];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int64_t o = base + l[r] * L + b[r];
                        f[r] = MODE == 2 ? reinterpret_cast<const int32_t *>(src)[o]
                                         : (int32_t) reinterpret_cast<const int16_t *>(src)[o];
                    }
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        if (e0 + r * T >= nlines * L) continue;
                        int32_t *o = indices + base + (e0 + r * T);
                        __stcs(o, site[r] ? (MODE == 2 ? (int32_t)(int16_t)(f[r] & 0xffff) : f[r]) : -1);
                        if (MODE == 2) {
                            __stcs(o + p.numel, site[r] ? f[r] >> 16 : 0);
                            __stcs(o + 2 * p.numel, b[r]);
                        } else {
                            __stcs(o + p.numel, b[r]);
                        }
                    }
                }
            }
        } else {
            const int segs = (L + 127) / 128;
            for (int l = 0, seg = warp;; seg += T / 32) {
                while (seg >= segs) seg -= segs, l++;
                if (l >= nlines) break;
                const int q0 = seg * 128 + lane;
                const int row = row0 + l;
                const int z = MODE == 2 ? row / p.L1 : 0, y = MODE == 2 ? row - z * p.L1 : row;
                const uint32_t *gr = g + l * tl.pitch + kLineK3;
                const uint16_t *pr = pos + l * tl.ppitch + q0;
                const int64_t rowbase = base + (int64_t)l * L, gi = rowbase + q0;
                const bool site = any[l] != 0;
                int b[4];
                uint32_t v[4];
#pragma unroll
                for (int r = 0; r < 4; r++) b[r] = site && q0 + 32 * r < L ? pr[32 * r] : 0;
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int d = q0 + 32 * r - b[r];
                    v[r] = gr[b[r]] + weight * (uint32_t)(d * d);
                }
                if (!site) {  // no background in the item: the site (-1, 0, ...)
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int q = q0 + 32 * r;
                        v[r] = w0 * (uint32_t)(MODE == 2 ? (z + 1) * (z + 1) : (y + 1) * (y + 1)) +
                               (MODE == 2 ? w1 * (uint32_t)(y * y) : 0u) + weight * (uint32_t)(q * q);
                    }
                }
                if (dist) {
                    float d[4];
                    if (near) {
#pragma unroll
                        for (int r = 0; r < 4; r++) d[r] = root[min(v[r], kSqrtTab - 1u)];  // (beyond the line: any entry)
                    } else {
#pragma unroll
                        for (int r = 0; r < 4; r++) d[r] = line_dist(v[r], p.unit2);
                    }
#pragma unroll
                    for (int r = 0; r < 4; r++)
                        if (q0 + 32 * r < L) __stcs(dist + gi + 32 * r, d[r]);
                }
                if (OUT == 0) continue;  // distances only
                if (sqdist) {
#pragma unroll
                    for (int r = 0; r < 4; r++)
                        if (q0 + 32 * r < L) __stcs(sqdist + gi + 32 * r, (int32_t)v[r]);
                }
                if (indices) {
                    int32_t f[4];
#pragma unroll
                    for (int r = 0; r < 4; r++)
                        f[r] = MODE == 2 ? reinterpret_cast<const int32_t *>(src)[rowbase + b[r]]
                                         : (int32_t) reinterpret_cast<const int16_t *>(src)[rowbase + b[r]];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        if (q0 + 32 * r >= L) continue;
                        int32_t *o = indices + gi + 32 * r;
                        __stcs(o, site ? (MODE == 2 ? (int32_t)(int16_t)(f[r] & 0xffff) : f[r]) : -1);
                        if (MODE == 2) {
                            __stcs(o + p.numel, site ? f[r] >> 16 : 0);
                            __stcs(o + 2 * p.numel, b[r]);
                        } else {
                            __stcs(o + p.numel, b[r]);
                        }
                    }
                }
            }
        }
        __syncthreads();  // the tile is rewritten by the next one
    }
}
