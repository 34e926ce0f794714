// All steps of an FP32 basis in one launch: the step of gram_mixed.cu (one
// reduction of a = U^T w, b = U^T u_j and |w|^2, the coefficients corrected by
// the Gram matrix) with the block's rows of the basis in shared memory.
//
// Small and ordinary sizes are bound by latency: launches that wait for one
// another, the sums over the row blocks and the scalar chain took 14 us a step
// at 2,000 rows, where the basis is 240 KB. Here a block keeps its rows for
// the whole cycle, so that a column is read from shared memory, and the
// matrix entries of its rows in registers; per step the blocks exchange only
// w's dot products and the new column. What depends on the new column alone
// (b: its norm, the breakdown test, the Gram row) is summed right after the
// update and worked out while the blocks wait for each other's dots with w.
// The pre-scale p is the power of two that brings the new column's norm, from
// |w|^2 - h.c, into [1, 2): any p near it serves (the next step measures
// the norm exactly), and this one costs no root and rounds nothing.
//
// Up to 8,192 rows (gc_cluster) the blocks are one cluster of 16 which meet at hardware
// barriers and write their partial sums into each other's shared memory;
// beyond, a cooperative grid with bounded waits and exact integer sums
// (cycle.cuh). Columns that do not fit on chip are read from L2.
#include "cycle.cuh"

#include <algorithm>
#include <climits>
#include <type_traits>

namespace mexk {

namespace {

constexpr int GC_THREADS = 512;
constexpr int GC_NW = GC_THREADS / 32;
constexpr int GC_SUB = 128;       // rows of a sub-block: one warp's float4s
constexpr int GC_CLUSTER = 16;
constexpr int GC_EPT = 8;         // matrix entries a thread can keep
constexpr int GC_TILE = GC_THREADS * GC_EPT;
constexpr int GC_GROUP = 4;       // columns of a warp's task
constexpr int GC_RUN = 8;         // float4s of a lane summed in plain FP32
constexpr int GC_LONG_MAX = 4096; // longest row
constexpr int GC_MARGIN = 16;     // |u_c| < 2^(GC_MARGIN / 2)

struct GcShared {
    float red[GC_NW][GRAM_M + 2];
    double b[GRAM_M + 1];
    double c[GRAM_M];
    double s[GRAM_M + 1];
    double ip, w2;
    float coef[GRAM_M];
    float part[GC_NW];
    float w2r;  // |A v_j|^2 / 4^half, in [1, 4); 0: no usable norm
    int half;
    int ok, bad;
    int nlong;
    int rows_long[GC_THREADS];
};

__device__ __forceinline__ float gc_dot4(const float4& a, const float4& b) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)));
}

// The kernel's dynamic shared memory, in order.
struct GcLayout {
    int ldE, rs;
    size_t pa, pb, prod, w, u, v;  // byte offsets; E at 0
    __host__ __device__ GcLayout(int m, int rows, bool cluster, bool csr) {
        ldE = m | 1;
        rs = (rows + GC_SUB - 1) / GC_SUB * GC_SUB;
        pa = (sizeof(double) * m * ldE + 15) / 16 * 16;
        pb = pa + (cluster ? sizeof(double) * (m + 1) * GC_CLUSTER : 0);
        prod = pb + (cluster ? sizeof(double) * 2 * m * GC_CLUSTER : 0);
        w = prod + (csr ? sizeof(float) * GC_TILE : 0);
        u = w + sizeof(float) * rs;
        v = u + sizeof(float) * rs;
    }
};

extern __shared__ __align__(16) unsigned char gc_smem[];

// The block's rows of w = A x, x a column of the basis in memory that other
// blocks wrote during this launch: FP32 products added in entry order (rows of
// more than SEQ_ROW_MAX entries: a warp, lanes strided), as the SpMV kernels.
template <int LM>
__device__ __forceinline__ void gc_product_pattern(const GramCycleArgs& g, const float* x, int r0, int n_rows,
                                                   float* w) {
    const RowPatterns* __restrict__ T = g.T;
    for (int r = threadIdx.x; r < n_rows; r += GC_THREADS) {
        const int id = __ldg(g.pid + r0 + r);
        const int len = __ldg(T->len + id);
        const int* off = T->off + id * PAT_LEN;
        const float* av = T->v32 + id * PAT_LEN;
        float xv[LM], a[LM];
#pragma unroll
        for (int q = 0; q < LM; ++q) {
            const bool on = q < len;
            a[q] = on ? __ldg(av + q) : 0.f;
            xv[q] = on ? x[r0 + r + __ldg(off + q)] : 0.f;
        }
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < LM; ++q)
            if (q < len) s = __fadd_rn(s, __fmul_rn(a[q], xv[q]));
        w[r] = s;
    }
}

// What a thread keeps of the matrix for the whole cycle. Rows of at most
// GC_EPT pattern entries, one per thread: the row's columns and values. A
// block of at most GC_TILE CSR entries: every GC_THREADS-th of them, and the
// extent of row threadIdx.x.
struct GcEntries {
    int c[GC_EPT];  // -1: none
    float a[GC_EPT];
    int e0, e1;
};

__device__ __forceinline__ void gc_product_row(const GcEntries& me, const float* x, int n_rows, float* w) {
    if (static_cast<int>(threadIdx.x) < n_rows) {
        float xv[GC_EPT];
#pragma unroll
        for (int u = 0; u < GC_EPT; ++u) xv[u] = me.c[u] >= 0 ? x[me.c[u]] : 0.f;
        float s = 0.f;
#pragma unroll
        for (int u = 0; u < GC_EPT; ++u)
            if (me.c[u] >= 0) s = __fadd_rn(s, __fmul_rn(me.a[u], xv[u]));
        w[threadIdx.x] = s;
    }
}

__device__ __forceinline__ void gc_product_kept(const GramCycleArgs& g, const GcEntries& me, const float* x, int r0,
                                                int n_rows, int e0, float* prod, float* w, GcShared& sh) {
    float xv[GC_EPT];
#pragma unroll
    for (int u = 0; u < GC_EPT; ++u) xv[u] = me.c[u] >= 0 ? x[me.c[u]] : 0.f;
    if (threadIdx.x == 0) sh.nlong = 0;
#pragma unroll
    for (int u = 0; u < GC_EPT; ++u)
        if (me.c[u] >= 0) prod[threadIdx.x + u * GC_THREADS] = __fmul_rn(me.a[u], xv[u]);
    __syncthreads();
    for (int r = threadIdx.x; r < n_rows; r += GC_THREADS) {
        int a = me.e0, z = me.e1;
        if (r != static_cast<int>(threadIdx.x)) {
            a = __ldg(g.row_ptr + r0 + r) - e0;
            z = __ldg(g.row_ptr + r0 + r + 1) - e0;
        }
        if (z - a > SEQ_ROW_MAX) {
            sh.rows_long[atomicAdd(&sh.nlong, 1)] = r;  // at most GC_TILE / SEQ_ROW_MAX of them
        } else {
            float s = 0.f;
            for (int e = a; e < z; e += 8) {
                float p[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) p[u] = e + u < z ? prod[e + u] : 0.f;
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (e + u < z) s = __fadd_rn(s, p[u]);
            }
            w[r] = s;
        }
    }
    if (!g.long_rows) return;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x >> 5; i < sh.nlong; i += GC_NW) {
        const int r = sh.rows_long[i];
        const int a = __ldg(g.row_ptr + r0 + r) - e0, z = __ldg(g.row_ptr + r0 + r + 1) - e0;
        float s = 0.f;
#pragma unroll 4
        for (int e = a + lane; e < z; e += 32) s = __fadd_rn(s, prod[e]);
        s = warp_sum(s);
        if (lane == 0) w[r] = s;
    }
}

// Any number of entries, a tile at a time.
__device__ __forceinline__ void gc_product_tiles(const GramCycleArgs& g, const float* x, int r0, int n_rows,
                                                 float* prod, float* w, GcShared& sh) {
    const int lane = threadIdx.x & 31;
    for (int rb = 0; rb < n_rows; rb += GC_THREADS) {
        const int r = rb + static_cast<int>(threadIdx.x), last = min(n_rows, rb + GC_THREADS);
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
        const int t0 = __ldg(g.row_ptr + r0 + rb), t1 = __ldg(g.row_ptr + r0 + last);
        float s = 0.f;
        for (int tb = t0; tb < t1; tb += GC_TILE) {
            const int te = min(t1, tb + GC_TILE);
            int c[GC_EPT];
            float a[GC_EPT], xv[GC_EPT];
#pragma unroll
            for (int u = 0; u < GC_EPT; ++u) {
                const int i = tb + static_cast<int>(threadIdx.x) + u * GC_THREADS;
                c[u] = i < te ? __ldg(g.col_idx + i) : -1;
                a[u] = i < te ? __ldg(g.values + i) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < GC_EPT; ++u) xv[u] = c[u] >= 0 ? x[c[u]] : 0.f;
#pragma unroll
            for (int u = 0; u < GC_EPT; ++u)
                if (c[u] >= 0) prod[threadIdx.x + u * GC_THREADS] = __fmul_rn(a[u], xv[u]);
            __syncthreads();
            for (; e < min(e1, te); ++e) s = __fadd_rn(s, prod[e - tb]);
            __syncthreads();
        }
        if (r < last) w[r] = s;
        __syncthreads();
        for (int i = threadIdx.x >> 5; i < sh.nlong; i += GC_NW) {
            const int q = sh.rows_long[i];
            const int a0 = __ldg(g.row_ptr + r0 + q), a1 = __ldg(g.row_ptr + r0 + q + 1);
            float t = 0.f;
#pragma unroll 8
            for (int i2 = a0 + lane; i2 < a1; i2 += 32)
                t = __fadd_rn(t, __fmul_rn(__ldg(g.values + i2), x[__ldg(g.col_idx + i2)]));
            t = warp_sum(t);
            if (lane == 0) w[q] = t;
        }
        __syncthreads();
    }
}

// Columns of the basis from column lo on: on chip at float offset vo + column *
// rs while the column is below on, else at far + column * ldv in memory.
struct GcVectors {
    const float* far;
    size_t ldv;
    int lo, on, vo, rs;
};

// Partial dots of k vectors (nb columns of the basis, then the last two or one
// at float offsets x1, x2) with x (shared memory) over the block's rows
// into sh.red[slice][c]; returns the number of slices. A warp's task is
// GC_GROUP vectors over a slice of the sub-blocks, a power of two of slices
// (no divisions): FP32 per lane and across the warp. A lane's sums of GC_RUN
// float4s are added up with their rounding errors carried along, so that more
// rows in a block make no longer chains than the separate sweep's (up to ten):
// heat 1000^2 3539 -> 3596 us a solve, 777^2 2659 -> 2688 (runs of 4: 3881, 2790).
__device__ __forceinline__ int gc_dots(const GcVectors& B, int nb, int x1, int x2, int k, int n4, const float* x,
                                       GcShared& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cgs = (k + GC_GROUP - 1) / GC_GROUP;
    const int nsub = (n4 + 31) / 32;
    int ls = cgs > 8 ? 0 : cgs > 4 ? 1 : cgs > 2 ? 2 : cgs > 1 ? 3 : 4;  // log2 of the slices
    ls = min(ls, 31 - __clz(max(nsub, 1)));
    const int slices = 1 << ls;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const float4* s4 = reinterpret_cast<const float4*>(gc_smem);
    const int sl = warp & (slices - 1);
    const int s0 = (sl * nsub) >> ls, s1 = ((sl + 1) * nsub) >> ls;
    const int i0 = s0 * 32 + lane, i1 = min(n4, s1 * 32);
    for (int cg = warp >> ls; cg < cgs; cg += GC_NW >> ls) {
        const int c0 = cg * GC_GROUP;
        float acc[GC_GROUP];
        int o[GC_GROUP];
#pragma unroll
        for (int c = 0; c < GC_GROUP; ++c) {
            o[c] = B.vo + (B.lo + c0 + c) * B.rs;
            if (c0 + c >= nb) o[c] = x1;
            if (c0 + c >= k - 1) o[c] = x2;
            o[c] >>= 2;
            acc[c] = 0.f;
        }
        auto sweep = [&](auto at) {
            auto add = [&](int i) {
                const float4 xv = x4[i];
                float4 v[GC_GROUP];
#pragma unroll
                for (int c = 0; c < GC_GROUP; ++c) v[c] = at(c, i);
#pragma unroll
                for (int c = 0; c < GC_GROUP; ++c) acc[c] += gc_dot4(v[c], xv);
            };
            if (s1 - s0 <= GC_RUN) {
#pragma unroll 2
                for (int i = i0; i < i1; i += 32) add(i);
                return;
            }
            float tot[GC_GROUP], rest[GC_GROUP];
#pragma unroll
            for (int c = 0; c < GC_GROUP; ++c) tot[c] = rest[c] = 0.f;
            for (int ib = i0; ib < i1;) {
                const int ie = min(i1, ib + 32 * GC_RUN);
#pragma unroll 2
                for (; ib < ie; ib += 32) add(ib);
#pragma unroll
                for (int c = 0; c < GC_GROUP; ++c) {
                    const float t = __fadd_rn(tot[c], acc[c]), b = __fsub_rn(t, tot[c]);
                    rest[c] += __fadd_rn(__fsub_rn(tot[c], __fsub_rn(t, b)), __fsub_rn(acc[c], b));
                    tot[c] = t;
                    acc[c] = 0.f;
                }
            }
#pragma unroll
            for (int c = 0; c < GC_GROUP; ++c) acc[c] = tot[c] + rest[c];
        };
        if (B.lo + min(c0 + GC_GROUP, nb) <= B.on) {
            sweep([&](int c, int i) { return s4[o[c] + i]; });
        } else {
            const float4* p[GC_GROUP];
#pragma unroll
            for (int c = 0; c < GC_GROUP; ++c)
                p[c] = c0 + c >= nb || B.lo + c0 + c < B.on
                           ? s4 + o[c]
                           : reinterpret_cast<const float4*>(B.far + (B.lo + c0 + c) * B.ldv);
            sweep([&](int c, int i) { return p[c][i]; });
        }
        // transposed over the lanes: lane l ends with vector (l >> 3) & 3
        const bool hi = (lane & 16) != 0, lo = (lane & 8) != 0;
        const float f0 = (hi ? acc[2] : acc[0]) + __shfl_xor_sync(AC_FULL, hi ? acc[0] : acc[2], 16);
        const float f1 = (hi ? acc[3] : acc[1]) + __shfl_xor_sync(AC_FULL, hi ? acc[1] : acc[3], 16);
        float f = (lo ? f1 : f0) + __shfl_xor_sync(AC_FULL, lo ? f0 : f1, 8);
#pragma unroll
        for (int o2 = 4; o2 >= 1; o2 >>= 1) f += __shfl_xor_sync(AC_FULL, f, o2);
        const int c = c0 + (hi ? 2 : 0) + (lo ? 1 : 0);
        if ((lane & 7) == 0 && c < k) sh.red[sl][c] = f;
    }
    return slices;
}

// VW rows (from row VW * i) of u_{j+1} = psc * (wsc * w - sum_c coef_c u_c), the
// kw columns from B.lo on, eight loaded together (past the end the last one,
// times zero).
template <int VW>
__device__ __forceinline__ void gc_update(const GcVectors& B, int kw, int i, const float* fs, int wo, float wsc,
                                          float psc, const float* coef, float (&out)[VW]) {
    using Vec = typename std::conditional<VW == 4, float4, typename std::conditional<VW == 2, float2, float>::type>::type;
    float s[VW];
#pragma unroll
    for (int e = 0; e < VW; ++e) s[e] = 0.f;
    const int onk = min(max(B.on - B.lo, 0), kw);  // the columns on chip come first
    auto add8 = [&](int c, int end, auto load) {
        Vec v[8];
        float h[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            v[u] = load(min(c + u, end - 1));
            h[u] = c + u < end ? coef[c + u] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int e = 0; e < VW; ++e) s[e] = fmaf(reinterpret_cast<const float*>(&v[u])[e], h[u], s[e]);
    };
    const float* p = fs + B.vo + B.lo * B.rs + VW * i;
    for (int c = 0; c < onk; c += 8) add8(c, onk, [&](int q) { return *reinterpret_cast<const Vec*>(p + q * B.rs); });
    const float* pg = B.far + B.lo * B.ldv + VW * i;
    for (int c = onk; c < kw; c += 8)
        add8(c, kw, [&](int q) { return *reinterpret_cast<const Vec*>(pg + q * B.ldv); });
    const Vec w = *reinterpret_cast<const Vec*>(fs + wo + VW * i);
#pragma unroll
    for (int e = 0; e < VW; ++e) out[e] = fmaf(reinterpret_cast<const float*>(&w)[e], wsc, -s[e]) * psc;
}

// The k totals over the slices to every block: a cluster's to part[c * 16 +
// this block] of each block's shared memory; a grid's to the words of column
// c, of range 2^scale(c) (the last one: column GRAM_M when `extra`). Four
// lanes per value.
template <bool CLUSTER, typename Scale>
__device__ __forceinline__ void gc_publish(int k, int slices, bool extra, double* part, unsigned long long* words,
                                           Scale scale, GcShared& sh) {
    for (int t = threadIdx.x; t < ((4 * k + 31) & ~31); t += GC_THREADS) {
        const int c = min(t >> 2, k - 1), q = t & 3;
        double s = q < slices ? static_cast<double>(sh.red[q][c]) : 0.0;
        for (int i = q + 4; i < slices; i += 4) s += static_cast<double>(sh.red[i][c]);
        if (slices > 1) {
            s += __shfl_xor_sync(AC_FULL, s, 1);
            if (slices > 2) s += __shfl_xor_sync(AC_FULL, s, 2);
            else s = __shfl_sync(AC_FULL, s, threadIdx.x & 28);
        } else {
            s = __shfl_sync(AC_FULL, s, threadIdx.x & 28);
        }
        if ((t >> 2) < k) {
            if constexpr (CLUSTER) {
                const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
                double* const p = part + c * GC_CLUSTER + blockIdx.x;
#pragma unroll
                for (int i = 0; i < GC_CLUSTER / 4; ++i) *cl.map_shared_rank(p, q * (GC_CLUSTER / 4) + i) = s;
            } else {
                const int sc = scale(c);
                const int ex = (__double2hiint(s) >> 20) & 0x7ff;
                const bool fits = ex == 0 || (ex < 1023 + sc && ex != 0x7ff);
                if (q < 3 && fits) {
                    int i;
                    const long long d = ac_digit(s, sc, q, &i);
                    const int slot = extra && c == k - 1 ? GRAM_M : c;
                    if (d != 0) atomicAdd(words + AC_DIGITS * slot + i, static_cast<unsigned long long>(d));
                } else if (q == 3 && !fits) {
                    atomicAdd(words + AC_DIGITS * MEXK_M_MAX, 1ull);
                }
            }
        }
    }
}

// The totals over the blocks, after the meeting: use(c, total) for c < k in
// one lane each (a grid's extra value in a warp of its own).
template <bool CLUSTER, typename Scale, typename Use>
__device__ __forceinline__ void gc_collect(int k, bool extra, const double* part, const unsigned long long* words,
                                           Scale scale, Use use) {
    if constexpr (CLUSTER) {
        const int t = threadIdx.x;
        if (t < ((4 * k + 31) & ~31)) {
            const int c = min(t >> 2, k - 1);
            const double2* p = reinterpret_cast<const double2*>(part + c * GC_CLUSTER + 4 * (t & 3));
            const double2 x = p[0], y = p[1];
            double s = (x.x + x.y) + (y.x + y.y);
            s += __shfl_xor_sync(AC_FULL, s, 1);
            s += __shfl_xor_sync(AC_FULL, s, 2);
            if ((t & 3) == 0 && (t >> 2) < k) use(c, s);
        }
    } else {
        const int t = threadIdx.x, plain = extra ? k - 1 : k;
        if (t < plain) use(t, ac_collect(words, t, scale(t)));
        else if (extra && t == GRAM_M) use(k - 1, ac_collect(words, GRAM_M, scale(k - 1)));
    }
}

template <bool CLUSTER>
__global__ void __launch_bounds__(GC_THREADS, 1) gram_cycle_kernel(GramCycleArgs g) {
    __shared__ GcShared sh;
    if (CLUSTER) pdl_wait();
    DevState* st = g.st;
    if (st->done || st->breakdown) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = g.m;
    const size_t ldv = static_cast<size_t>(g.ldv), ldh = static_cast<size_t>(g.ldh);
    const GcLayout L(m, g.rows, CLUSTER, g.pid == nullptr);
    double* const E = reinterpret_cast<double*>(gc_smem);  // G - I
    double* const pa = reinterpret_cast<double*>(gc_smem + L.pa);
    double* const pb = reinterpret_cast<double*>(gc_smem + L.pb);
    float* const prod = reinterpret_cast<float*>(gc_smem + L.prod);
    float* const w = reinterpret_cast<float*>(gc_smem + L.w);
    const int r0 = min(static_cast<int>(blockIdx.x) * g.rows, g.n);
    const int n_rows = min(g.rows, g.n - r0);
    const int n4 = (n_rows + 3) / 4;
    const int rp = 4 * n4;  // rows with the padding of the last float4
    const bool lead = blockIdx.x == 0;
    GramState* gs = g.gs;
    unsigned target = 0;
    GcVectors B{g.V + r0, ldv, 0, g.on, static_cast<int>(L.v / sizeof(float)), L.rs};
    const int on = g.on, vo = static_cast<int>(L.v / sizeof(float)), uo = static_cast<int>(L.u / sizeof(float));
    // the newest column's: always on chip
    auto own = [&](int c) { return c < on ? vo + c * L.rs : uo; };
    float* const fs = reinterpret_cast<float*>(gc_smem);
    const int wo = static_cast<int>(L.w / sizeof(float));
    auto wa = [&](int p) { return g.words + static_cast<size_t>(2 * p) * CYCLE_EXCHANGE; };
    auto wb = [&](int p) { return g.words + static_cast<size_t>(2 * p + 1) * CYCLE_EXCHANGE; };
    const auto scale_b = [](int) { return GC_MARGIN; };

    GcEntries me;
    me.e0 = me.e1 = 0;
    int e0 = 0;
    bool kept = false;
    if (g.pid == nullptr) {
        e0 = __ldg(g.row_ptr + r0);
        const int cnt = __ldg(g.row_ptr + r0 + n_rows) - e0;
        kept = cnt <= GC_TILE;
#pragma unroll
        for (int u = 0; u < GC_EPT; ++u) {
            const int i = tid + u * GC_THREADS;
            const bool have = kept && i < cnt;
            me.c[u] = have ? __ldg(g.col_idx + e0 + i) : -1;
            me.a[u] = have ? __ldg(g.values + e0 + i) : 0.f;
        }
        if (tid < n_rows) {
            me.e0 = __ldg(g.row_ptr + r0 + tid) - e0;
            me.e1 = __ldg(g.row_ptr + r0 + tid + 1) - e0;
        }
    } else {
        kept = g.max_len <= GC_EPT && g.rows <= GC_THREADS;
        const bool have = kept && tid < n_rows;
        const int id = have ? __ldg(g.pid + r0 + tid) : 0;
        const int len = have ? __ldg(g.T->len + id) : 0;
#pragma unroll
        for (int u = 0; u < GC_EPT; ++u) {
            me.c[u] = u < len ? r0 + tid + __ldg(g.T->off + id * PAT_LEN + u) : -1;
            me.a[u] = u < len ? __ldg(g.T->v32 + id * PAT_LEN + u) : 0.f;
        }
    }
    for (int r = tid; r < rp; r += GC_THREADS) {
        w[r] = 0.f;
        fs[own(0) + r] = r < n_rows ? __ldcg(g.V + r0 + r) : 0.f;
    }
    if (tid == 0) sh.ip = gs->ip[0];
    if (CLUSTER) cooperative_groups::this_cluster().sync();  // every block runs before another writes to its memory
    else __syncthreads();
    if (!CLUSTER && lead && g_test_ac_dead_wait != 0) return;
    {
        const int slices = gc_dots(B, 0, 0, own(0), 1, n4, fs + own(0), sh);
        __syncthreads();
        gc_publish<CLUSTER>(1, slices, false, pb, wb(0), scale_b, sh);
    }
    if (!ac_meet<CLUSTER>(g.bar, target, &st->status, &sh.ok)) return;

    bool broke = false;
    for (int j = 0; j < m; ++j) {
        const int lo = g.window > 0 ? max(0, j + 1 - g.window) : 0;
        const int kw = j + 1 - lo;
        const int par = j & 1;
        const auto scale_a = [&](int c) { return c < kw ? g.scale + GC_MARGIN : 2 * (g.scale + GC_MARGIN); };
        // the last block clears the sums of step j - 1, which every block has read
        if (!CLUSTER && blockIdx.x == gridDim.x - 1 && j > 0) {
            unsigned long long* const z = wa(par ^ 1);
            for (int i = tid; i < 2 * CYCLE_EXCHANGE; i += GC_THREADS) __stcg(z + i, 0ull);
        }
        B.lo = lo;
        // w = A u_j
        const float* x = g.V + static_cast<size_t>(j) * ldv;
        if (g.pid != nullptr) {
            if (kept) gc_product_row(me, x, n_rows, w);
            else if (g.max_len <= 5) gc_product_pattern<5>(g, x, r0, n_rows, w);
            else if (g.max_len <= 7) gc_product_pattern<7>(g, x, r0, n_rows, w);
            else gc_product_pattern<PAT_LEN>(g, x, r0, n_rows, w);
        } else if (kept) {
            gc_product_kept(g, me, x, r0, n_rows, e0, prod, w, sh);
        } else {
            gc_product_tiles(g, x, r0, n_rows, prod, w, sh);
        }
        __syncthreads();
        // a = U^T w and |w|^2
        {
            const int slices =
                gc_dots(B, kw - 1, own(j), wo, kw + 1, n4, w, sh);
            __syncthreads();
            gc_publish<CLUSTER>(kw + 1, slices, true, pa, wa(par), scale_a, sh);
        }
        ac_arrive<CLUSTER>(g.bar, target);
        // meanwhile what b gives: s_j, H(j, j-1) and the breakdown test of
        // main.cu:1911, the Gram row
        gc_collect<CLUSTER>(kw, false, pb + par * m * GC_CLUSTER, wb(par), scale_b,
                            [&](int c, double v) { sh.b[c] = v; });
        __syncthreads();
        if (tid < kw) {
            const double bj = sh.b[kw - 1];
            const double sj = (bj > 0.0 && !isinf(bj)) ? rsqrt(bj) : 0.0;
            double gv = 1.0;
            if (tid < kw - 1) {
                gv = (sh.s[lo + tid] * sh.b[tid]) * sj;
                E[(lo + tid) * L.ldE + j] = gv;
                E[j * L.ldE + lo + tid] = gv;
            } else {
                sh.s[j] = sj;
                E[j * L.ldE + j] = 0.0;
                if (lead) gs->s[j] = sj;
            }
            if (lead) {
                gs->G[(lo + tid) + static_cast<size_t>(j) * GRAM_LD] = gv;
                gs->G[j + static_cast<size_t>(lo + tid) * GRAM_LD] = gv;
            }
        }
        if (tid == GC_THREADS - 1) {
            int bad = 0;
            if (j >= 1) {
                const double beta = sqrt(sh.b[kw - 1]) * sh.ip;
                bad = !(beta >= 1e-14) || isinf(beta) ? 1 : 0;
                if (lead) {
                    g.H[j + (j - 1) * ldh] = bad ? 0.0 : beta;
                    if (bad) {
                        st->breakdown = 1;
                        st->k_used = j;
                    }
                }
            }
            sh.bad = bad;
        }
        if (!ac_wait<CLUSTER>(g.bar, target, &st->status, &sh.ok)) return;
        if (CLUSTER) __syncthreads();
        if (sh.bad) {  // the same sums in every block
            broke = true;
            break;
        }
        // c = s s_j a, |A v_j|^2
        gc_collect<CLUSTER>(kw + 1, true, pa, wa(par), scale_a, [&](int c, double v) {
            const double sj = sh.s[j];
            if (c < kw) {
                sh.c[c] = (sh.s[lo + c] * v) * sj;
            } else {
                const double w2 = (sj * sj) * v;
                const int ex = (__double2hiint(w2) >> 20) & 0x7ff;
                const bool usable = w2 > 0.0 && ex > 0 && ex < 0x7ff;
                const int half = usable ? (ex - 1023) >> 1 : 0;
                const double q = __hiloint2double((1023 - half) << 20, 0);  // 2^-half
                sh.half = half;
                sh.w2r = usable ? static_cast<float>((w2 * q) * q) : 0.f;
            }
        });
        __syncthreads();
        // h = c - (G - I) c: four lanes per row
        if (tid < ((4 * kw + 31) & ~31)) {
            const int r = min(tid >> 2, kw - 1), q = tid & 3;
            double h = sh.c[r], e = 0.0;
            const double cr = h;
            if (g.reortho) {
                const double* Er = E + (lo + r) * L.ldE + lo;
                double f = 0.0;
                int i = q;
                for (; i + 4 < kw; i += 8) {
                    e = fma(Er[i], sh.c[i], e);
                    f = fma(Er[i + 4], sh.c[i + 4], f);
                }
                if (i < kw) e = fma(Er[i], sh.c[i], e);
                e += f;
                e += __shfl_xor_sync(AC_FULL, e, 1);
                e += __shfl_xor_sync(AC_FULL, e, 2);
                h -= e;
            }
            const bool mine = (tid >> 2) < kw;
            if (lead && mine && q == 0) g.H[(lo + r) + j * ldh] = h;
            // lane 0: s h; lanes 1 and 2: h and c over 2^half
            const double f = q == 0 ? sh.s[lo + r] : __hiloint2double((1023 - sh.half) << 20, 0);
            const float v = static_cast<float>((q == 2 ? cr : h) * f);
            if (mine && q == 0) sh.coef[r] = v;
            float pr = __shfl_down_sync(AC_FULL, v, 1);
            pr = mine && q == 1 ? v * pr : 0.f;
            pr = warp_sum(pr);
            if (lane == 0) sh.part[warp] = pr;
        }
        if (lead)
            for (int r = tid; r < lo; r += GC_THREADS) g.H[r + j * ldh] = 0.0;  // outside the window
        __syncthreads();
        // the pre-scale from |w - V h|^2 = |w|^2 - h.c (to first order in G - I)
        int pe = 0;
        {
            const float w2r = sh.w2r;
            float t = 0.f;
            for (int i = 0; i < (4 * kw + 31) / 32; ++i) t += sh.part[i];
            float u2 = w2r - t;
            if (!(u2 > 1e-6f * w2r)) u2 = w2r;
            if (w2r > 0.f) pe = min(max(sh.half + (((__float_as_int(u2) >> 23) - 127) >> 1), -120), 120);
        }
        const float psc = __int_as_float((127 - pe) << 23);
        const float wsc = static_cast<float>(sh.s[j]);
        // u_{j+1} = p (s_j w - sum_c s_c h_c u_c)
        const int no = j + 1 < m ? own(j + 1) : uo;
        float* const nx = fs + no;
        float* const out = g.V + static_cast<size_t>(j + 1) * ldv + r0;
        if (rp > 2 * GC_THREADS) {
            for (int i = tid; i < n4; i += GC_THREADS) {
                float v[4];
                gc_update<4>(B, kw, i, fs, wo, wsc, psc, sh.coef, v);
                *reinterpret_cast<float4*>(nx + 4 * i) = make_float4(v[0], v[1], v[2], v[3]);
                __stcg(reinterpret_cast<float4*>(out) + i, make_float4(v[0], v[1], v[2], v[3]));
            }
        } else {
            for (int i = tid; 2 * i < rp; i += GC_THREADS) {
                float v[2];
                gc_update<2>(B, kw, i, fs, wo, wsc, psc, sh.coef, v);
                *reinterpret_cast<float2*>(nx + 2 * i) = make_float2(v[0], v[1]);
                __stcg(reinterpret_cast<float2*>(out) + i, make_float2(v[0], v[1]));
            }
        }
        __syncthreads();
        if (tid == 0) sh.ip = __hiloint2double((1023 + pe) << 20, 0);
        if (lead && tid == 0) {
            gs->ip[j + 1] = __hiloint2double((1023 + pe) << 20, 0);
            gs->wsc = wsc;
            gs->psc = psc;
        }
        // b = U^T u_{j+1} (after the last step: its norm alone)
        {
            const int nlo = j + 1 == m ? m : g.window > 0 ? max(0, j + 2 - g.window) : 0;
            const int nk = j + 2 - nlo;
            B.lo = nlo;
            // column j from memory when it is off chip (its copy on chip is u_{j+1}'s place now)
            const int slices = gc_dots(B, nk - 1, 0, no, nk, n4, nx, sh);
            __syncthreads();
            gc_publish<CLUSTER>(nk, slices, false, pb + (par ^ 1) * m * GC_CLUSTER, wb(par ^ 1), scale_b, sh);
        }
        if (!ac_meet<CLUSTER>(g.bar, target, &st->status, &sh.ok)) return;
    }
    if (!broke && lead) {  // |u_m|: H(m, m-1), s_m
        gc_collect<CLUSTER>(1, false, pb + (m & 1) * m * GC_CLUSTER, wb(m & 1), scale_b, [&](int, double b) {
            const double beta = sqrt(b) * sh.ip;
            const bool bad = !(beta >= 1e-14) || isinf(beta);
            if (m < g.ldh) g.H[m + (m - 1) * ldh] = bad ? 0.0 : beta;
            gs->s[m] = (b > 0.0 && !isinf(b)) ? rsqrt(b) : 0.0;
            gs->G[m + static_cast<size_t>(m) * GRAM_LD] = 1.0;
            if (bad) {
                st->breakdown = 1;
                st->k_used = m;
            }
        });
    }
    if (!CLUSTER) {
        // the last block to leave clears the meeting's words and the sums for the next launch
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            sh.ok = atomicAdd(&g.bar[3], 1u) == gridDim.x - 1 ? 1 : 0;
        }
        __syncthreads();
        if (sh.ok) {
            if (tid == 0) {
                g.bar[0] = 0u;
                g.bar[3] = 0u;
            }
            for (int i = tid; i < 4 * CYCLE_EXCHANGE; i += GC_THREADS) __stcg(g.words + i, 0ull);
        }
    }
}

constexpr int GC_SMEM = 227 * 1024 - static_cast<int>(sizeof(GcShared)) - 1024;

// Whether the blocks are one cluster. Up to 4,096 rows always; to 8,192, whose
// rows are a thread's at most, where a block's entries stay few. Grid /
// cluster, one solve: heat 66^2 1093 / 911 us, 90^2 1081 / 925 (110^2 1086 /
// 1022, its window 2 889 / 868, 126^2 1080 / 1061); random rows of 11: 4,500
// 417 / 365, 8,000 424 / 412, 10,000 420 / 461; power law 8,000 1664 / 1996.
bool gc_cluster(int n, long long nnz, bool long_rows, bool csr) {
    if (n <= 4096) return true;
    return n <= GRAM_CLUSTER_ROWS && (!csr || (!long_rows && nnz <= 90000));
}

struct GcShape {
    int grid, rows, on;
    size_t smem;
};
GcShape gc_shape(int n, int m, bool cluster, bool csr) {
    GcShape s;
    const int blocks = cluster ? GC_CLUSTER : std::min(device_sm_count(), CYCLE_MAX_BLOCKS);
    s.rows = ((n + blocks - 1) / blocks + 31) / 32 * 32;
    s.grid = cluster ? GC_CLUSTER : (n + s.rows - 1) / s.rows;
    const GcLayout L(m, s.rows, cluster, csr);
    const long long left = GC_SMEM - static_cast<long long>(L.v);
    s.on = left <= 0 ? 0 : static_cast<int>(std::min<long long>(m, left / (static_cast<long long>(sizeof(float)) * L.rs)));
    s.smem = L.v + sizeof(float) * static_cast<size_t>(s.on) * L.rs;
    return s;
}

}  // namespace

// One solve, separate kernels / one launch (us). The basis: an eighth of its
// columns on chip is enough, the rest costs three sweeps of L2 instead of two
// (30 columns, heat grid of 48^2 1607 / 913, 400^2 2184 / 1367, 777^2 3613 /
// 2691, 1000^2 4721 / 3727, 1100^2 5418 / 4688; 3D 61^3 862 / 538, 90^3 2304 /
// 1643, 110^3 3301 / 2985). CSR products gather at L2's rate in both, but keep
// less of x in L1 here (random rows of 11: 2,000 584 / 359, 50,000 664 / 499,
// 150,000 896 / 719, 200,000 988 / 1021, 300,000 1193 / 1341); long rows leave
// blocks waiting for one another (power law: 5,000 1608 / 1147, 20,000 3363 /
// 2475, 50,000 3917 / 3730, 100,000 4857 / 5929). A window of two or so columns
// has next to no sweeps (heat 400^2 1445 / 1244, 600^2 1991 / 1907, 777^2
// 2169 / 2224). A few columns are on chip at any size, but above 1.8 million
// rows a block's own rows outlast the launches saved (5 columns: 1300^2 276 /
// 272, 1400^2 283 / 297, 1500^2 285 / 331; 8: 377 / 371, 384 / 404, 390 / 433),
// and up to three are over before they have paid for the start (2: 600^2 254 /
// 262, 1000^2 270 / 284; 3: 281 / 286 at 777^2).
bool gram_cycle_fits(int n, long long nnz, int m, int max_row, bool pattern, int window) {
    if (m < 1 || m > GRAM_M) return false;
    if (window > 0 && window <= 4 && n > 400000) return false;
    if (n > 1800000 || (m <= 3 && n > 300000)) return false;
    if (!pattern && (max_row > GC_LONG_MAX || nnz > (max_row > SEQ_ROW_MAX ? 600000 : 2000000))) return false;
    return 8 * gc_shape(n, m, gc_cluster(n, nnz, max_row > SEQ_ROW_MAX, !pattern), !pattern).on >= m;
}

int gram_cycle_prepare() {
    MEXK_CK(cudaFuncSetAttribute(gram_cycle_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GC_SMEM));
    MEXK_CK(cudaFuncSetAttribute(gram_cycle_kernel<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    MEXK_CK(cudaFuncSetAttribute(gram_cycle_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, GC_SMEM));
    return MEXK_OK;
}

int gram_cycle_test_hook(int enable) {
    const int v = enable ? 1 : 0;
    MEXK_CK(cudaMemcpyToSymbol(g_test_ac_dead_wait, &v, sizeof(int)));
    return MEXK_OK;
}

int launch_gram_cycle(GramCycleArgs a, cudaStream_t s) {
    if (a.m < 1 || a.m > GRAM_M || a.scale == INT_MAX) return MEXK_ERR_INVALID;
    const bool cluster = gc_cluster(a.n, a.nnz, a.long_rows != 0, a.pid == nullptr);
    const GcShape sp = gc_shape(a.n, a.m, cluster, a.pid == nullptr);
    if (sp.on < 1) return MEXK_ERR_UNSUPPORTED;
    a.rows = sp.rows;
    a.on = sp.on;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sp.grid);
    cfg.blockDim = dim3(GC_THREADS);
    cfg.dynamicSmemBytes = sp.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    if (cluster) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = GC_CLUSTER;
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
    const cudaError_t e = cluster ? cudaLaunchKernelEx(&cfg, gram_cycle_kernel<true>, a)
                                  : cudaLaunchKernelEx(&cfg, gram_cycle_kernel<false>, a);
    if (e != cudaSuccess) {
        set_cuda_error(e, "gram_cycle_kernel", __FILE__, __LINE__);
        return MEXK_ERR_CUDA;
    }
    return MEXK_OK;
}

}  // namespace mexk
