// All m steps of an FP64 Arnoldi basis in one launch.
//
// The FP64 step is CGS2 (gram_schmidt.cu): product, dots, update and dots,
// update and norm, normalisation -- five launches, three of which end in a
// grid reduction. Up to a few hundred thousand rows those launches and their
// serial tails are what a step costs (about 40 us at 2,000 rows, 50 us at
// 9,216, 100 us at 600,000 with a window of 2) while its FP64 arithmetic,
// 8 n k flops at about two FMAs per clock per SM, would take 1 to 10 us.
// Measured per step now: 13, 15 and 38 us; whole solves 3.0 times faster at
// 2,000 rows, 2.4 at 50,021 with 100 columns, 1.06 at 4,194,304 with 30, where
// FP64 issue in the sweeps is nearly all of a step. Here every thread block owns a
// contiguous range of rows for the whole basis, keeps its part of w in shared
// memory, and the blocks meet three times a step, each time to exchange k (or
// one) partial sums:
//   w = A v_j; partial V^T w                                | meet
//   h1 = sums; w -= V h1; partial V^T w                     | meet
//   h2 = sums; H(:,j) = h1 + h2; w -= V h2; partial |w|^2   | meet
//   H(j+1,j) = |w|, breakdown test, v_{j+1} = w / |w|
// Every block sums the partials for itself, so nothing is broadcast. What
// the next product gathers is the unnormalised w, scaled at the gather (the
// same rounded product that v_{j+1} holds), where that costs less than a
// fourth meeting.
//
// An FP64 warp instruction keeps its quarter of the SM for 64 clocks whether
// or not it depends on the last one, so work is shared out to have every
// lane of every quarter busy: rows over lanes in the update, columns and row
// slices over warps in the dots, eight columns reduced together by a
// transposing butterfly.
//
// Up to EXACT_ROWS rows the sums keep the order of the separate kernels
// (pairs of rows per lane, the warp butterfly of the sweep's width, warps of
// 64 rows eight at a time, then in row order), so for even n and up to 32
// columns the basis is theirs bit for bit; every row sum of the product is
// theirs at any size. The blocks are one cluster of 16 there, which meet at
// hardware barriers (0.8 us) and write their partials into each other's
// shared memory; beyond, a cooperative grid with bounded waits (1.5 us) and
// exact integer sums. A matrix whose products do not suit the kernel (long
// rows, many entries) keeps the context's SpMV and takes one launch per step.
#include "cycle.cuh"

#include <algorithm>
#include <climits>

namespace mexk {

namespace {

constexpr int AC_THREADS = 512;
constexpr int AC_NW = AC_THREADS / 32;
constexpr int AC_SUB = 64;           // rows of a sub-block: one warp's pairs
constexpr int AC_CLUSTER = 16;
// One cluster up to here (16 SMs: heat 64^2 18 us a step; a grid of 144 blocks
// takes 17 us at 9,216 rows, where the cluster's FP64 work has doubled).
constexpr int EXACT_ROWS = 4096;
constexpr int AC_LONG_MAX = 2048;    // longest row (the product's block-wide rows are not built here)
constexpr int AC_PS = EXACT_ROWS / AC_SUB;  // a cluster's partials of one column

// ---- warp reductions ---------------------------------------------------------
// Lane-bit order of the separate sweeps of width 8, 16 or more columns.
__device__ __forceinline__ constexpr int ac_bit(int width, int level) {
    constexpr int order[3][5] = {{4, 2, 1, 8, 16}, {8, 4, 2, 1, 16}, {16, 8, 4, 2, 1}};
    return order[width][level];
}
// Butterfly over the warp of CN columns (1, 2, 4 or 8) in that order: the
// first log2(CN) levels transpose, so a lane ends with the warp total of
// column ac_column (its other bits name one of 32 / CN copies).
template <int WIDTH, int CN>
__device__ __forceinline__ double ac_reduce(double (&a)[CN], int lane) {
    int level = 0;
#pragma unroll
    for (int h = CN / 2; h >= 1; h >>= 1, ++level) {
        const int b = ac_bit(WIDTH, level);
        const bool up = (lane & b) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double send = up ? a[i] : a[i + h];
            const double keep = up ? a[i + h] : a[i];
            a[i] = keep + __shfl_xor_sync(AC_FULL, send, b);
        }
    }
    double v = a[0];
#pragma unroll
    for (; level < 5; ++level) v += __shfl_xor_sync(AC_FULL, v, ac_bit(WIDTH, level));
    return v;
}
// The column a lane ends with, and which copy of it.
template <int WIDTH, int CN>
__device__ __forceinline__ void ac_place(int lane, int* column, int* copy) {
    int c = 0, d = 0, level = 0;
#pragma unroll
    for (int h = CN / 2; h >= 1; h >>= 1, ++level)
        if (lane & ac_bit(WIDTH, level)) c += h;
#pragma unroll
    for (int w = 1; level < 5; ++level, w <<= 1)
        if (lane & ac_bit(WIDTH, level)) d += w;
    *column = c;
    *copy = d;
}

extern __shared__ double ac_smem[];  // w (the block's rows); a cluster: then the exchanges' partials

constexpr int AC_TILE = 2048;  // products staged at a time
constexpr int AC_SMEM_DOUBLES = 22528;  // rows of w that a block keeps in shared memory (176 KB)

struct AcShared {
    double h[MEXK_M_MAX];               // the second pass's coefficients
    double h1[MEXK_M_MAX];              // the first pass's
    double red[AC_NW][MEXK_M_MAX + 1];  // row slices' dots, then the partial sums' slices
    double prod[AC_TILE];
    double inv;
    int ok;   // the meetings' (cycle.cuh)
    int bad;  // the step's breakdown: a word of its own, no barrier follows the last read of ok
    int nlong;
    int rows_long[AC_THREADS];
};

// One exchange: where the partial sums go. EXACT: part (in every block's
// shared memory), column c's sub-block b at part[c * AC_PS + b]. Else the
// dots to words, column c's digits at words[AC_DIGITS c ..] and after the
// last column the count of non-finite partials; the norm to part, one partial
// per block.
struct AcExchange {
    double* part;
    unsigned long long* words;
};

// The dots of CN columns (kc of them real) with w over sub-blocks s0..s1-1. V:
// the block's first row of the first column, in memory or on chip.
template <int WIDTH, bool EXACT, int CN>
__device__ __forceinline__ void ac_dot_task(const double* V, size_t ldv, int c0, int kc, int r0, int s0, int s1, int sl,
                                            const double* wv, const AcExchange& ex, AcShared& sh) {
    constexpr int SU = EXACT ? 1 : (CN == 8 ? 2 : 4);  // sub-blocks whose loads are in flight together
    const int lane = threadIdx.x & 31;
    double acc[CN];
#pragma unroll
    for (int c = 0; c < CN; ++c) acc[c] = 0.0;
    for (int s = s0; s < s1; s += SU) {
        double2 v[SU][CN];
        const int lr = s * AC_SUB + 2 * lane;
        const double* p = V + static_cast<size_t>(c0) * ldv + lr;
#pragma unroll
        for (int u = 0; u < SU; ++u)
#pragma unroll
            for (int c = 0; c < CN; ++c)
                v[u][c] = (c < kc && s + u < s1) ? *reinterpret_cast<const double2*>(p + c * ldv + u * AC_SUB)
                                                 : make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < SU; ++u) {
            if (u > 0 && s + u >= s1) break;
            const double2 w = *reinterpret_cast<const double2*>(wv + lr + u * AC_SUB);
#pragma unroll
            for (int c = 0; c < CN; ++c) {
                acc[c] = fma(v[u][c].x, w.x, acc[c]);
                acc[c] = fma(v[u][c].y, w.y, acc[c]);
            }
        }
    }
    const double tot = ac_reduce<WIDTH, CN>(acc, lane);
    int cc, copy;
    ac_place<WIDTH, CN>(lane, &cc, &copy);
    const int c = c0 + cc;
    if (cc >= kc) return;
    if (EXACT) {
        const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        double* dst = ex.part + c * AC_PS + r0 / AC_SUB + sl;
        for (int p = copy; p < AC_CLUSTER; p += 32 / CN) *cl.map_shared_rank(dst, p) = tot;
    } else if (copy == 0) {
        sh.red[sl][c] = tot;
    }
}

// Dots of columns 0..k-1 of V with w over the block's rows into the exchange.
// Warps take (group of up to eight columns, sub-block or row slice).
template <int WIDTH, bool EXACT>
__device__ __forceinline__ void ac_dots(const CycleArgs& g, const double* V, size_t ldv, int k, int r0, int nsub,
                                        const double* wv, const AcExchange& ex, AcShared& sh) {
    const int warp = threadIdx.x >> 5;
    const int cgs = (k + 7) >> 3;
    const int slices = EXACT ? nsub : max(1, min(nsub, AC_NW / cgs));
    for (int t = warp; t < cgs * slices; t += AC_NW) {
        const int cg = t % cgs, sl = t / cgs;
        const int c0 = cg * 8, kc = min(8, k - c0);
        const int s0 = EXACT ? sl : sl * nsub / slices, s1 = EXACT ? sl + 1 : (sl + 1) * nsub / slices;
        if (kc > 4) ac_dot_task<WIDTH, EXACT, 8>(V, ldv, c0, kc, r0, s0, s1, sl, wv, ex, sh);
        else if (kc > 2) ac_dot_task<WIDTH, EXACT, 4>(V, ldv, c0, kc, r0, s0, s1, sl, wv, ex, sh);
        else if (kc > 1) ac_dot_task<WIDTH, EXACT, 2>(V, ldv, c0, kc, r0, s0, s1, sl, wv, ex, sh);
        else ac_dot_task<WIDTH, EXACT, 1>(V, ldv, c0, kc, r0, s0, s1, sl, wv, ex, sh);
    }
    if (!EXACT) {
        __syncthreads();
        ac_publish<AC_THREADS>(ex.words, &sh.red[0][0], MEXK_M_MAX + 1, k, slices, g.scale);
    }
}

// out[c] = column c's sum over all blocks, c < k, after the meeting; every
// thread calls it. EXACT: np sub-blocks, eight at a time in order, then the
// eights in order.
template <bool EXACT>
__device__ __forceinline__ void ac_sums(const AcExchange& ex, int k, int np, int scale, double* out, AcShared& sh) {
    if (EXACT) {
        const int slices = (np + 7) / 8, kr = (k + 31) & ~31;  // columns over lanes
        for (int t = threadIdx.x; t < kr * slices; t += AC_THREADS) {
            const int c = t % kr, sl = t / kr;
            if (c < k) {
                const double* p = ex.part + c * AC_PS + sl * 8;
                const int nb = min(8, np - sl * 8);
                double s = p[0];
                for (int b = 1; b < nb; ++b) s += p[b];
                sh.red[sl][c] = s;
            }
        }
        __syncthreads();
        for (int c = threadIdx.x; c < k; c += AC_THREADS) {
            double s = sh.red[0][c];
            for (int q = 1; q < slices; ++q) s += sh.red[q][c];
            out[c] = s;
        }
    } else {
        for (int c = threadIdx.x; c < k; c += AC_THREADS) {
            out[c] = ac_collect(ex.words, c, scale);
        }
    }
    __syncthreads();
}

// w -= V h over the block's rows (one FMA chain per row, in column order; not
// the padding after them, which stays zero where h is not finite); RU rows of
// a thread and CH columns in flight.
template <int RU, int CH>
__device__ __forceinline__ void ac_update_rows(const double* V, size_t ldv, int k, int rows, const double* h,
                                               double* w) {
    for (int r = threadIdx.x; r < rows; r += RU * AC_THREADS) {
        double s[RU];
#pragma unroll
        for (int i = 0; i < RU; ++i) s[i] = 0.0;
        const double* p = V + r;
        for (int c = 0; c < k; c += CH, p += CH * ldv) {
            double v[RU][CH];
#pragma unroll
            for (int i = 0; i < RU; ++i)
#pragma unroll
                for (int u = 0; u < CH; ++u)
                    v[i][u] = (c + u < k && r + i * AC_THREADS < rows) ? p[u * ldv + i * AC_THREADS] : 0.0;
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                if (u > 0 && c + u >= k) break;
#pragma unroll
                for (int i = 0; i < RU; ++i) s[i] = fma(v[i][u], h[c + u], s[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < RU; ++i)
            if (r + i * AC_THREADS < rows) w[r + i * AC_THREADS] -= s[i];
    }
}
__device__ __forceinline__ void ac_update(const double* V, size_t ldv, int k, int rows, const double* h, double* w) {
    if (k <= 2 && rows > AC_THREADS) ac_update_rows<4, 2>(V, ldv, k, rows, h, w);
    else ac_update_rows<1, 8>(V, ldv, k, rows, h, w);
}

// ---- one or two columns --------------------------------------------------------
// A short window's step in three passes instead of five, each reading the
// columns once: the dots; the first update with the second dots; the second
// update with the norm (a sweep of its own for each took 38 of a step's 85
// thousand cycles at 777^2 rows, window 2). UPDATE: w -= h0 v0 + h1 v1.
// The thread's sums of v0.w, v1.w (or |w|^2 in sum[0]) over its rows, in
// pairs: past the last row w stays zero, also where h is not finite.
enum AcPass { AC_PASS_DOTS, AC_PASS_NORM };
template <bool UPDATE, AcPass PASS>
__device__ __forceinline__ void ac_narrow_pass(const double* V, size_t ldv, int k, int r0, int rows, const double* h,
                                               double* w, double (&sum)[2]) {
    constexpr int UN = 4;
    const bool two = k == 2;
    const double* const p0 = V + r0;
    const double* const p1 = p0 + ldv;
    const double h0 = UPDATE ? -h[0] : 0.0, h1 = UPDATE && two ? -h[1] : 0.0;
    sum[0] = sum[1] = 0.0;
    for (int r = 2 * static_cast<int>(threadIdx.x); r < rows; r += 2 * UN * AC_THREADS) {
        double2 x[UN], a[UN], b[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int q = r + 2 * u * AC_THREADS;
            a[u] = b[u] = x[u] = make_double2(0.0, 0.0);
            if (q < rows) {
                a[u] = __ldcg(reinterpret_cast<const double2*>(p0 + q));
                if (two) b[u] = __ldcg(reinterpret_cast<const double2*>(p1 + q));
                x[u] = *reinterpret_cast<const double2*>(w + q);
            }
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int q = r + 2 * u * AC_THREADS;
            if (q >= rows) break;
            if (UPDATE) {
                x[u].x = fma(h0, a[u].x, x[u].x);
                x[u].y = fma(h0, a[u].y, x[u].y);
                if (two) {
                    x[u].x = fma(h1, b[u].x, x[u].x);
                    x[u].y = fma(h1, b[u].y, x[u].y);
                }
                if (q + 1 == rows) x[u].y = 0.0;
                *reinterpret_cast<double2*>(w + q) = x[u];
            }
            if (PASS == AC_PASS_DOTS) {
                sum[0] = fma(a[u].x, x[u].x, sum[0]);
                sum[0] = fma(a[u].y, x[u].y, sum[0]);
                if (two) {
                    sum[1] = fma(b[u].x, x[u].x, sum[1]);
                    sum[1] = fma(b[u].y, x[u].y, sum[1]);
                }
            } else {
                sum[0] = fma(x[u].x, x[u].x, sum[0]);
                sum[0] = fma(x[u].y, x[u].y, sum[0]);
            }
        }
    }
}

// The block's sums of two columns into the exchange.
__device__ __forceinline__ void ac_narrow_publish(const CycleArgs& g, int k, double (&sum)[2], const AcExchange& ex,
                                                  AcShared& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // lanes 0..15 go on with column 0, the others with column 1
    double t = (lane & 16) ? sum[1] : sum[0];
    t += __shfl_xor_sync(AC_FULL, (lane & 16) ? sum[0] : sum[1], 16);
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) t += __shfl_xor_sync(AC_FULL, t, o);
    if ((lane & 15) == 0) sh.red[warp][lane >> 4] = t;
    __syncthreads();
    ac_publish<AC_THREADS>(ex.words, &sh.red[0][0], MEXK_M_MAX + 1, k, AC_NW, g.scale);
}

// The block's rows of w = A x in the row-pattern form, patterns of at most LM
// entries: rounded products added in column order (spmv_pattern.cu). Gathered
// entries times inv (scaled) or as they are.
template <int LM>
__device__ __forceinline__ void ac_product_pattern(const CycleArgs& g, const double* gx, double inv, bool scaled,
                                                   int r0, int rows, int n_rows, double* w) {
    const RowPatterns* __restrict__ T = g.T;
    for (int r = threadIdx.x; r < rows; r += AC_THREADS) {
        double s = 0.0;
        if (r < n_rows) {
            const int id = __ldg(g.pid + r0 + r);
            const int len = __ldg(T->len + id);
            const int* off = T->off + id * PAT_LEN;
            const double* av = T->v64 + id * PAT_LEN;
            double x[LM], a[LM];
#pragma unroll
            for (int q = 0; q < LM; ++q) {
                const bool on = q < len;
                a[q] = on ? __ldg(av + q) : 0.0;
                x[q] = on ? __ldcg(gx + (r0 + r + __ldg(off + q))) : 0.0;
            }
#pragma unroll
            for (int q = 0; q < LM; ++q)
                if (q < len) s = __dadd_rn(s, __dmul_rn(a[q], scaled ? __dmul_rn(x[q], inv) : x[q]));
        }
        w[r] = s;
    }
}

// The same from the CSR arrays (spmv.cu's row sums): the block's products in
// shared memory a tile at a time, coalesced; a row of at most SEQ_ROW_MAX
// entries summed in order by its thread, a longer one by a warp, lanes
// strided, from the arrays.
__device__ __forceinline__ void ac_product_csr(const CycleArgs& g, const double* gx, double inv, bool scaled, int r0,
                                               int rows, int n_rows, double* w, AcShared& sh) {
    constexpr int EU = AC_TILE / AC_THREADS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto entry = [&](int e) {
        const double x = __ldcg(gx + __ldg(g.col_idx + e));
        return __dmul_rn(__ldg(g.values + e), scaled ? __dmul_rn(x, inv) : x);
    };
    for (int rb = 0; rb < rows; rb += AC_THREADS) {
        const int r = rb + static_cast<int>(threadIdx.x);
        const int last = min(n_rows, rb + AC_THREADS);
        if (threadIdx.x == 0) sh.nlong = 0;
        __syncthreads();
        int e = 0, e1 = 0;
        if (r < last) {
            e = __ldg(g.row_ptr + r0 + r);
            e1 = __ldg(g.row_ptr + r0 + r + 1);
            if (e1 - e > SEQ_ROW_MAX) {
                sh.rows_long[atomicAdd(&sh.nlong, 1)] = r;
                e1 = e;
            }
        }
        const int t0 = last > rb ? __ldg(g.row_ptr + r0 + rb) : 0, t1 = last > rb ? __ldg(g.row_ptr + r0 + last) : 0;
        double s = 0.0;
        for (int tb = t0; tb < t1; tb += AC_TILE) {
            const int te = min(t1, tb + AC_TILE);
            int c[EU];
            double x[EU], a[EU];
#pragma unroll
            for (int u = 0; u < EU; ++u) {
                const int i = tb + static_cast<int>(threadIdx.x) + u * AC_THREADS;
                c[u] = i < te ? __ldg(g.col_idx + i) : -1;
                a[u] = i < te ? __ldg(g.values + i) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < EU; ++u) x[u] = c[u] >= 0 ? __ldcg(gx + c[u]) : 0.0;
#pragma unroll
            for (int u = 0; u < EU; ++u) {
                if (tb + u * AC_THREADS >= te) break;
                sh.prod[threadIdx.x + u * AC_THREADS] = __dmul_rn(a[u], scaled ? __dmul_rn(x[u], inv) : x[u]);
            }
            __syncthreads();
            for (; e < min(e1, te); ++e) s = __dadd_rn(s, sh.prod[e - tb]);
            __syncthreads();
        }
        if (r < rows) w[r] = s;
        __syncthreads();
        for (int i = warp; i < sh.nlong; i += AC_NW) {
            const int q = sh.rows_long[i];
            const int a0 = __ldg(g.row_ptr + r0 + q), a1 = __ldg(g.row_ptr + r0 + q + 1);
            double t = 0.0;
            for (int i2 = a0 + lane; i2 < a1; i2 += 32) t = __dadd_rn(t, entry(i2));
            t = warp_sum(t);
            if (lane == 0) w[q] = t;
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void ac_product(const CycleArgs& g, const double* gx, double inv, bool scaled, int r0,
                                           int rows, int n_rows, double* w, AcShared& sh) {
    if (g.pid == nullptr) ac_product_csr(g, gx, inv, scaled, r0, rows, n_rows, w, sh);
    else if (g.max_len <= 5) ac_product_pattern<5>(g, gx, inv, scaled, r0, rows, n_rows, w);
    else if (g.max_len <= 7) ac_product_pattern<7>(g, gx, inv, scaled, r0, rows, n_rows, w);
    else ac_product_pattern<PAT_LEN>(g, gx, inv, scaled, r0, rows, n_rows, w);
}

// The block's |w|^2 from the first nw warps' sums into the exchange.
__device__ __forceinline__ void ac_norm_publish(double acc, int nw, const AcExchange& ex, AcShared& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < nw) {
        const double t = warp_sum(acc);
        if (lane == 0) sh.red[warp][0] = t;
    }
    __syncthreads();
    if (warp == 0) {
        double t = lane < nw ? sh.red[lane][0] : 0.0;
        for (int o = 1; o < nw; o <<= 1) t += __shfl_xor_sync(AC_FULL, t, o);
        if (lane == 0) __stcg(ex.part + blockIdx.x, t);
    }
}

// |w|^2 over the block's rows into the exchange. EXACT per sub-block (pairs,
// then the plain butterfly).
template <bool EXACT>
__device__ __forceinline__ void ac_norm(int r0, int nsub, const double* wv, const AcExchange& ex, AcShared& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double acc = 0.0;
    for (int s = warp; s < nsub; s += AC_NW) {
        const double2 w = *reinterpret_cast<const double2*>(wv + s * AC_SUB + 2 * lane);
        if (EXACT) acc = 0.0;
        acc = fma(w.x, w.x, acc);
        acc = fma(w.y, w.y, acc);
        if (EXACT) {
            const double t = warp_sum(acc);
            const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
            if (lane < AC_CLUSTER) *cl.map_shared_rank(ex.part + r0 / AC_SUB + s, lane) = t;
        }
    }
    if (!EXACT) ac_norm_publish(acc, min(AC_NW, nsub), ex, sh);
}

// |w|^2 over all blocks, after the meeting, in thread 0. The dynamic range of
// a square is too wide for the words: one partial per block, summed by warp 0.
template <bool EXACT>
__device__ __forceinline__ double ac_norm_sum(const AcExchange& ex, int np) {
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    if (threadIdx.x < 32) {
        if (EXACT) {  // lane: eight sub-blocks in order, then the lanes in order
            const int slices = (np + 7) / 8;
            if (lane < slices) {
                const double* p = ex.part + lane * 8;
                const int nb = min(8, np - lane * 8);
                s = p[0];
                for (int b = 1; b < nb; ++b) s += p[b];
            }
            double t = s;
            for (int q = 1; q < slices; ++q) t += __shfl_sync(AC_FULL, s, q);
            s = t;
        } else {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = lane + 32 * u < gridDim.x ? __ldcg(ex.part + lane + 32 * u) : 0.0;
            s = v[0];
#pragma unroll
            for (int u = 1; u < 8; ++u) {
                if (32 * u >= gridDim.x) break;
                s += v[u];
            }
            s = warp_sum(s);
        }
    }
    return s;
}

// CLUSTER: one cluster, the separate kernels' sums. WSMEM: the block's rows of
// w fit in shared memory (else they stay in x). NARROW: a window of at most
// two columns. VSMEM: the block's rows of the basis too (they are read four
// times a step, and from L2 each time costs a round trip).
template <bool CLUSTER, bool WSMEM, bool NARROW = false, bool VSMEM = false>
__global__ void __launch_bounds__(AC_THREADS, 1) arnoldi_cycle_kernel(CycleArgs g) {
    constexpr bool EXACT = CLUSTER;
    __shared__ AcShared sh;
    if (CLUSTER) pdl_wait();
    DevState* st = g.st;
    if (st->done || st->breakdown) return;
    const size_t ldv = static_cast<size_t>(g.ldv), ldh = static_cast<size_t>(g.ldh);
    const int r0 = min(static_cast<int>(blockIdx.x) * g.rows, g.n);
    const int n_rows = min(g.rows, g.n - r0);  // real rows; the rest up to a sub-block are zero
    const int nsub = (n_rows + AC_SUB - 1) / AC_SUB;
    const int rows = nsub * AC_SUB;
    const int np = (g.n + AC_SUB - 1) / AC_SUB;
    const bool lead = blockIdx.x == 0;
    unsigned target = 0;
    double inv = 1.0;
    double* const w = WSMEM ? ac_smem : g.x + r0;
    // the exchanges of a step: first dots, second dots, norm; a grid's words
    // alternate by step parity, so that one set is cleared while the other is
    // in use
    AcExchange ex[3];
    auto exchanges = [&](int parity) {
        for (int i = 0; i < 3; ++i) {
            ex[i].part = EXACT ? ac_smem + g.rows + static_cast<size_t>(i) * g.m * AC_PS
                               : reinterpret_cast<double*>(g.words + 4 * CYCLE_EXCHANGE);
            ex[i].words = g.words + static_cast<size_t>(2 * parity + (i & 1)) * CYCLE_EXCHANGE;
        }
    };
    exchanges(0);
    // the block's rows of the columns in shared memory, column c at c * rows
    double* const vs = ac_smem + g.rows + (CLUSTER ? (2 * g.m + 1) * AC_PS : 0);
    if (VSMEM) {
        for (int r = threadIdx.x; r < rows; r += AC_THREADS) vs[r] = r < n_rows ? g.V[r0 + r] : 0.0;
        __syncthreads();
    }
    if (CLUSTER) cooperative_groups::this_cluster().sync();  // every block runs before another writes to its memory
    if (!CLUSTER && lead && g_test_ac_dead_wait != 0) return;
    for (int j = g.j0; j < g.j1; ++j) {
        const int lo = g.window > 0 ? max(0, j + 1 - g.window) : 0;
        const int k = j + 1 - lo;
        const double* V = g.V + static_cast<size_t>(lo) * ldv;
        const double* const Vb = VSMEM ? vs + lo * rows : V + r0;
        const size_t ldb = VSMEM ? static_cast<size_t>(rows) : ldv;
        const bool scaled = j > g.j0 && g.scale_gather;
        if (!EXACT) exchanges(j & 1);
        if (g.product) {
            ac_product(g, scaled ? g.x : g.V + static_cast<size_t>(j) * ldv, inv, scaled, r0, rows, n_rows, w, sh);
        } else if (WSMEM) {
            for (int r = threadIdx.x; r < rows; r += AC_THREADS) w[r] = r < n_rows ? __ldg(g.x + r0 + r) : 0.0;
        }
        __syncthreads();
        auto dots = [&](const AcExchange& e) {
            if (k <= 8) ac_dots<0, EXACT>(g, Vb, ldb, k, r0, nsub, w, e, sh);
            else if (k <= 16) ac_dots<1, EXACT>(g, Vb, ldb, k, r0, nsub, w, e, sh);
            else ac_dots<2, EXACT>(g, Vb, ldb, k, r0, nsub, w, e, sh);
        };
        constexpr bool narrow = NARROW;
        double sum[2];
        if (narrow) {
            ac_narrow_pass<false, AC_PASS_DOTS>(V, ldv, k, r0, n_rows, nullptr, w, sum);
            ac_narrow_publish(g, k, sum, ex[0], sh);
        } else {
            dots(ex[0]);
        }
        if (!ac_meet<CLUSTER>(g.bar, target, &st->status, &sh.ok)) return;
        // every block has read the other parity's sums: clear them for the next step
        if (!EXACT && lead) {
            unsigned long long* w = g.words + static_cast<size_t>(2 * ((j + 1) & 1)) * CYCLE_EXCHANGE;
            for (int i = threadIdx.x; i < 2 * CYCLE_EXCHANGE; i += AC_THREADS) __stcg(w + i, 0ull);
        }
        ac_sums<EXACT>(ex[0], k, np, g.scale, sh.h1, sh);
        if (narrow) {
            if (g.reortho) ac_narrow_pass<true, AC_PASS_DOTS>(V, ldv, k, r0, n_rows, sh.h1, w, sum);
            else ac_narrow_pass<true, AC_PASS_NORM>(V, ldv, k, r0, n_rows, sh.h1, w, sum);
        } else {
            ac_update(Vb, ldb, k, n_rows, sh.h1, w);
            __syncthreads();
        }
        if (g.reortho) {
            if (narrow) ac_narrow_publish(g, k, sum, ex[1], sh);
            else dots(ex[1]);
            if (!ac_meet<CLUSTER>(g.bar, target, &st->status, &sh.ok)) return;
            ac_sums<EXACT>(ex[1], k, np, g.scale, sh.h, sh);
            if (narrow) {
                ac_narrow_pass<true, AC_PASS_NORM>(V, ldv, k, r0, n_rows, sh.h, w, sum);
            } else {
                ac_update(Vb, ldb, k, n_rows, sh.h, w);
            }
        }
        if (lead)
            for (int c = threadIdx.x; c < k; c += AC_THREADS)
                g.H[(lo + c) + j * ldh] = g.reortho ? sh.h1[c] + sh.h[c] : sh.h1[c];
        __syncthreads();
        if (narrow) ac_norm_publish(sum[0], AC_NW, ex[2], sh);
        else ac_norm<EXACT>(r0, nsub, w, ex[2], sh);
        if (WSMEM && g.scale_gather)
            for (int r = threadIdx.x; r < n_rows; r += AC_THREADS) __stcg(g.x + r0 + r, w[r]);
        if (!ac_meet<CLUSTER>(g.bar, target, &st->status, &sh.ok)) return;
        const double w2 = ac_norm_sum<EXACT>(ex[2], np);
        // one thread: a square root and a division by every warp would queue on the FP64 units
        if (threadIdx.x == 0) {
            const double beta = sqrt(w2);
            const bool bad = beta < 1e-14 || isnan(beta) || isinf(beta);
            sh.bad = bad ? 1 : 0;
            if (!bad) sh.inv = 1.0 / beta;
            if (lead) {
                g.H[(j + 1) + j * ldh] = bad ? 0.0 : beta;
                if (bad) {
                    st->breakdown = 1;
                    st->k_used = j + 1;
                }
            }
        }
        __syncthreads();
        if (sh.bad) break;  // the same sums in every block
        inv = sh.inv;
        double* q = g.V + static_cast<size_t>(j + 1) * ldv + r0;
        if (VSMEM && j + 1 < g.j1) {
            double* const vq = vs + (j + 1) * rows;
            for (int r = threadIdx.x; r < rows; r += AC_THREADS) {
                const double v = w[r] * inv;
                vq[r] = v;
                if (r < n_rows) __stcg(q + r, v);
            }
        } else {
            for (int r = threadIdx.x; r < n_rows; r += AC_THREADS) __stcg(q + r, w[r] * inv);
        }
        if (!g.scale_gather && j + 1 < g.j1 && !ac_meet<CLUSTER>(g.bar, target, &st->status, &sh.ok)) return;
        __syncthreads();
    }
    if (CLUSTER) {
        cooperative_groups::this_cluster().sync();  // no block leaves while another writes to its shared memory
    } else {
        // the last block to leave clears the meeting's words and the sums for the next launch
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            sh.ok = atomicAdd(&g.bar[3], 1u) == gridDim.x - 1 ? 1 : 0;
        }
        __syncthreads();
        if (sh.ok) {
            if (threadIdx.x == 0) {
                g.bar[0] = 0u;
                g.bar[3] = 0u;
            }
            for (int i = threadIdx.x; i < 4 * CYCLE_EXCHANGE; i += AC_THREADS) __stcg(g.words + i, 0ull);
        }
    }
}

int sm_total() { return std::min(device_sm_count(), CYCLE_MAX_BLOCKS); }

}  // namespace

// Dynamic shared memory beside the kernel's own.
constexpr int AC_SMEM_TOTAL = 227 * 1024 - static_cast<int>(sizeof(AcShared)) - 64;

// Rows of a grid's blocks.
static int grid_rows(int n) {
    const int subs = (n + AC_SUB - 1) / AC_SUB;
    return (subs + sm_total() - 1) / sm_total() * AC_SUB;
}

// Once w is no longer on chip (3.4 million rows), a window pays by how well it
// fills the separate sweeps, which are 8, 16, 32 ... columns wide whatever of
// them it has, where this kernel pays for the columns there are. One basis of
// 40 columns on heat grids, separate / one launch (ms): 2048^2 window 4 16.2 /
// 13.5, 5 16.2 / 16.0, 8 16.3 / 17.1, 9 23.4 / 19.4, 12 23.5 / 21.5, 16 23.4 /
// 23.8, 20 29.0 / 27.2, 24 29.1 / 28.8; 3500^2 window 4 43.5 / 40.5, 5 43.6 /
// 47.1, 8 43.9 / 49.4, 9 64.2 / 56.7, 12 64.3 / 62.2, 16 64.1 / 68.9, 24 80.5 /
// 83.3. Without a window 2048^2 30 columns 21.8 / 20.8, 3500^2 60.4 / 60.3, 60
// columns 227.8 / 193.4.
bool arnoldi_cycle_fits(int n, int window) {
    if (n > CYCLE_ROWS_MAX) return false;
    return grid_rows(n) <= AC_SMEM_DOUBLES || window <= 4 || (window - 1) % 8 < 4;
}

// Measured on random rows (degree 10, m = 30, one cycle): own product against
// the context's SpMV and a launch per step, 661 / 871 us at 5,000 rows, 997 /
// 1108 at 50,000, 1367 / 1382 at 100,000, 1971 / 1957 at 200,000 (2.2 million
// entries), 3528 / 3101 at 400,000. Rows longer than one thread sums keep a
// warp each for a whole round trip per 32 entries: the SpMV's. The row-pattern
// form is bound by FP64 issue either way.
bool arnoldi_cycle_product(int n, long long nnz, int max_row, bool pattern) {
    if (pattern) return true;
    if (n <= EXACT_ROWS) return max_row <= AC_LONG_MAX;
    return max_row <= SEQ_ROW_MAX && nnz <= 2000000;
}

int arnoldi_cycle_prepare() {
    const int cl = static_cast<int>(sizeof(double)) * (EXACT_ROWS / AC_CLUSTER + (2 * MEXK_M_MAX + 1) * AC_PS);
    const int ws = static_cast<int>(sizeof(double)) * AC_SMEM_DOUBLES;
    MEXK_CK(cudaFuncSetAttribute(arnoldi_cycle_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, cl));
    MEXK_CK(cudaFuncSetAttribute(arnoldi_cycle_kernel<true, true>,
                                 cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    MEXK_CK(cudaFuncSetAttribute(arnoldi_cycle_kernel<true, true, false, true>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, AC_SMEM_TOTAL));
    MEXK_CK(cudaFuncSetAttribute(arnoldi_cycle_kernel<true, true, false, true>,
                                 cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    MEXK_CK(cudaFuncSetAttribute(arnoldi_cycle_kernel<false, true, false, true>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, AC_SMEM_TOTAL));
    MEXK_CK(cudaFuncSetAttribute(arnoldi_cycle_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, ws));
    MEXK_CK(cudaFuncSetAttribute(arnoldi_cycle_kernel<false, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, ws));
    return MEXK_OK;
}

int arnoldi_cycle_test_hook(int enable) {
    const int v = enable ? 1 : 0;
    MEXK_CK(cudaMemcpyToSymbol(g_test_ac_dead_wait, &v, sizeof(int)));
    return MEXK_OK;
}

int launch_arnoldi_cycle(CycleArgs a, cudaStream_t s) {
    const bool cluster = a.n <= EXACT_ROWS;
    if (a.j0 < 0 || a.j1 > a.m || a.j0 >= a.j1 || (!a.product && a.j1 != a.j0 + 1)) return MEXK_ERR_INVALID;
    int grid;
    if (cluster) {
        const int subs = (a.n + AC_SUB - 1) / AC_SUB;
        grid = AC_CLUSTER;
        a.rows = (subs + grid - 1) / grid * AC_SUB;
        a.scale_gather = 1;
    } else {
        a.rows = grid_rows(a.n);
        grid = (a.n + a.rows - 1) / a.rows;
        a.scale_gather = a.product && a.nnz * a.rows <= 6000ll * a.n ? 1 : 0;
    }
    if (!cluster && grid > CYCLE_MAX_BLOCKS) return MEXK_ERR_UNSUPPORTED;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(AC_THREADS);
    // Three passes against five sweeps, heat grids, window 2, one solve: 200^2 (320 rows a block) 2911 / 2890 us,
    // 300^2 3804 / 3302, 777^2 7271 / 6787, 1500^2 18442 / 16838; below 256 rows a block the sweeps share a column's
    // few rows out better (131^2 2695 / 2763).
    const bool narrow = !cluster && a.window > 0 && a.window <= 2 && a.rows >= 256;
    const bool wsmem = a.rows <= AC_SMEM_DOUBLES;
    if (!wsmem) a.scale_gather = 0;  // x holds w
    cfg.dynamicSmemBytes = sizeof(double) * ((wsmem ? static_cast<size_t>(a.rows) : 0) +
                                             (cluster ? (2 * static_cast<size_t>(a.m) + 1) * AC_PS : 0));
    // the basis on chip as well, where all m columns fit and one launch runs all steps. From L2 / on chip, one
    // solve: random 1,500 rows 556 / 528 us, 20,000 753 / 727, 80,000 1222 / 1197; 8,000 rows, 100 columns 18.9 /
    // 17.2 ms; heat 48^2 2854 / 2700 us, 300^2 5226 / 4997.
    const size_t vbytes = sizeof(double) * static_cast<size_t>(a.rows) * a.m;
    const bool vsmem = a.product && wsmem && !narrow &&
                       cfg.dynamicSmemBytes + vbytes <= static_cast<size_t>(AC_SMEM_TOTAL);
    if (vsmem) cfg.dynamicSmemBytes += vbytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    if (cluster) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = AC_CLUSTER;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    } else {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.numAttrs = 1;
    }
    cfg.attrs = attr;
    const cudaError_t e = cluster && vsmem  ? cudaLaunchKernelEx(&cfg, arnoldi_cycle_kernel<true, true, false, true>, a)
                          : cluster         ? cudaLaunchKernelEx(&cfg, arnoldi_cycle_kernel<true, true>, a)
                          : vsmem           ? cudaLaunchKernelEx(&cfg, arnoldi_cycle_kernel<false, true, false, true>, a)
                          : narrow && wsmem ? cudaLaunchKernelEx(&cfg, arnoldi_cycle_kernel<false, true, true>, a)
                          : narrow          ? cudaLaunchKernelEx(&cfg, arnoldi_cycle_kernel<false, false, true>, a)
                          : wsmem           ? cudaLaunchKernelEx(&cfg, arnoldi_cycle_kernel<false, true>, a)
                                            : cudaLaunchKernelEx(&cfg, arnoldi_cycle_kernel<false, false>, a);
    if (e != cudaSuccess) {
        set_cuda_error(e, "arnoldi_cycle_kernel", __FILE__, __LINE__);
        return MEXK_ERR_CUDA;
    }
    return MEXK_OK;
}

}  // namespace mexk
