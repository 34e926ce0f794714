// All steps of a short-recurrence basis (window 2, symmetric A in the
// row-pattern form, FP32 basis) in one launch, the recurrence on chip.
//
// A step as separate kernels reads u_j and u_{j-1} twice and writes and reads
// w = A u_j: at 2048^2 rows (16.8 MB a column) 28 us, in two launches that
// wait for each other. The recurrence needs three vectors only. Here a block
// keeps its rows of all three for the whole cycle: u_j in shared memory, with
// the neighbouring rows its stencil reaches, w and u_{j-1}, which only their
// own row reads, in tensor memory (a row group's place there may depend on a
// loop counter; in registers the loops had to be unrolled over all 54 groups
// of a block and ran at the rate of instruction fetches, 1200 cycles for 4
// groups). A step reads nothing from memory but the neighbours' rows and
// writes u_{j+1} once, for the lift: the first and last rows of a block, which
// its neighbours read, before it arrives at the meeting, the others after it.
// Per step two meetings (cycle.cuh), the sums as exact integers; what the new
// column alone determines (its norm, the breakdown test, a_{j-1} and the Gram
// entry, by symmetry from the update) is worked out while the blocks wait for
// u_j.w and |w|^2. The pre-scale is the power of two of gram_cycle.cu.
#include "cycle.cuh"

#include <algorithm>
#include <climits>

namespace mexk {

namespace {

constexpr int SC_THREADS = 512;                      // the threads with rows
constexpr int SC_NW = SC_THREADS / 32;
constexpr int SC_BLOCK = SC_THREADS + 32;            // and one warp for the scalar chain
constexpr int SC_CHUNK = 4;                          // row groups (of SC_THREADS rows) handled together
constexpr int SC_CHUNK_ROWS = SC_CHUNK * SC_THREADS;
constexpr int SC_GROUPS = 64;                        // at most: 2 tensor-memory columns each of a warp's 128
constexpr int SC_MARGIN = 16;                        // |u_c| < 2^(SC_MARGIN / 2)
constexpr int SC_TMEM = 512;                         // tensor-memory columns: all of them
constexpr int SC_OTHER = 0xff;                       // mask of a row that is no part of the major pattern
static_assert(STENCIL_LEN < 8, "a row's mask is a byte, SC_OTHER not among them");

struct ScShared {
    float red[3][SC_NW];
    double pre[5];  // s_j, s_j^2, G(j-1, j), c_{j-1}, G(j-1, j) c_{j-1}
    double ip, sp;  // 1 / pre-scale of column j, s_{j-1}
    double b[3], a[2];
    float cp, cj, wsc, psc;
    int ok, bad;
    unsigned tmem;
    unsigned char mask[PAT_MAX];  // a pattern's entries among the major one's
};

extern __shared__ __align__(16) float sc_smem[];

// Four consecutive columns of the warp's lanes of tensor memory.
__device__ __forceinline__ void sc_tst(unsigned at, const float (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(v[0]), "f"(v[1]),
                 "f"(v[2]), "f"(v[3])
                 : "memory");
}
__device__ __forceinline__ void sc_tld(unsigned at, float (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "r"(at)
                 : "memory");
}
__device__ __forceinline__ void sc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The wait names the registers, so that no use of them moves before it.
__device__ __forceinline__ void sc_wait_ld(float (&a)[4], float (&b)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(a[0]), "+f"(a[1]), "+f"(a[2]), "+f"(a[3]), "+f"(b[0]), "+f"(b[1]), "+f"(b[2]), "+f"(b[3])
                 :
                 : "memory");
}

// A barrier of the threads with rows: the scalar warp has work of its own.
__device__ __forceinline__ void sc_rows_sync() { asm volatile("bar.sync 1, %0;" ::"n"(SC_THREADS) : "memory"); }

// The block's sums of NV values (FP32 per thread with rows) to the words of
// columns 0..NV-1, of range 2^scale(v), and the block's arrival at the meeting
// whose target the caller has moved on. The threads with rows call it.
template <int NV, typename Scale>
__device__ __forceinline__ void sc_publish(const float (&v)[NV], unsigned long long* words, unsigned* bar, Scale scale,
                                           ScShared& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const float r = warp_sum(v[q]);
        if (lane == 0) sh.red[q][warp] = r;
    }
    sc_rows_sync();
    if (warp < NV) {
        double s = lane < SC_NW ? static_cast<double>(sh.red[warp][lane]) : 0.0;
#pragma unroll
        for (int o = 1; o < SC_NW; o <<= 1) s += __shfl_xor_sync(AC_FULL, s, o);
        s = __shfl_sync(AC_FULL, s, 0);
        const int sc = scale(warp);
        const int ex = (__double2hiint(s) >> 20) & 0x7ff;
        const bool fits = ex == 0 || (ex < 1023 + sc && ex != 0x7ff);
        if (lane < 3 && fits) {
            int i;
            const long long d = ac_digit(s, sc, lane, &i);
            if (d != 0) atomicAdd(words + AC_DIGITS * warp + i, static_cast<unsigned long long>(d));
        } else if (lane == 3 && !fits) {
            atomicAdd(words + AC_DIGITS * MEXK_M_MAX, 1ull);
        }
    }
    sc_rows_sync();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}

// Dynamic shared memory: reach rows of the blocks before, the block's rows
// (whole chunks), reach rows of those after; then a mask byte per row.
__host__ __device__ inline int sc_chunks(int rows) { return (rows + SC_CHUNK_ROWS - 1) / SC_CHUNK_ROWS; }
__host__ __device__ inline int sc_halo(int reach) { return (reach + 3) / 4 * 4; }

// L: entries of the major pattern, those past its length zero.
template <int L>
__global__ void __launch_bounds__(SC_BLOCK, 1) stencil_cycle_kernel(StencilArgs g) {
    __shared__ ScShared sh;
    DevState* st = g.st;
    if (st->done || st->breakdown) return;
    const int tid = threadIdx.x, warp = tid >> 5;
    const bool scalar = warp == SC_NW;
    const int m = g.m;
    const size_t ldv = static_cast<size_t>(g.ldv), ldh = static_cast<size_t>(g.ldh);
    const int r0 = blockIdx.x * g.rows;
    const int nr = min(g.rows, g.n - r0);
    const bool lead = blockIdx.x == 0;
    GramState* gs = g.gs;
    const RowPatterns* __restrict__ T = g.T;
    const int nc = sc_chunks(nr);
    const int halo = sc_halo(g.reach);
    float* const u = sc_smem + halo;  // u_j, rows -reach .. nr + reach - 1
    unsigned char* const rmask = reinterpret_cast<unsigned char*>(u + sc_chunks(g.rows) * SC_CHUNK_ROWS + halo);
    unsigned target = 0;
    auto wa = [&](int p) { return g.words + static_cast<size_t>(2 * p) * CYCLE_EXCHANGE; };
    auto wb = [&](int p) { return g.words + static_cast<size_t>(2 * p + 1) * CYCLE_EXCHANGE; };
    const auto scale_a = [&](int c) { return c == 0 ? g.scale + SC_MARGIN : 2 * (g.scale + SC_MARGIN); };
    const auto scale_b = [&](int c) { return c == 2 ? g.scale + SC_MARGIN : SC_MARGIN; };
    if (warp == 0) {  // the only block on its SM (SC_SMEM_MIN): nobody it waits for waits for this
        const unsigned p = static_cast<unsigned>(__cvta_generic_to_shared(&sh.tmem));
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(p), "n"(SC_TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    // what a pattern takes of the major one
    const int len = g.len;
    for (int p = tid; p < PAT_MAX; p += SC_BLOCK) {
        // each entry another one of the major pattern's, in its order: a row may store a column twice
        int mask = 0, next = 0;
        const int pl = p < T->count ? __ldg(T->len + p) : 0;
        for (int e = 0; e < pl && mask != SC_OTHER; ++e) {
            const int o = __ldg(T->off + p * PAT_LEN + e);
            const float v = __ldg(T->v32 + p * PAT_LEN + e);
            int hit = -1;
#pragma unroll
            for (int q = L - 1; q >= 0; --q)
                if (q >= next && q < len && g.off[q] == o && __float_as_int(g.val[q]) == __float_as_int(v)) hit = q;
            mask = hit < 0 ? SC_OTHER : mask | 1 << hit;
            next = hit + 1;
        }
        sh.mask[p] = static_cast<unsigned char>(mask);
    }
    const int full = (1 << len) - 1;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tw = sh.tmem + (static_cast<unsigned>(warp & 3) << 21) + (warp >> 2) * 128;  // lane 32 (warp % 4)
    const unsigned tp = tw + SC_GROUPS;
    // chunks whose rows, of this warp, all have the major pattern; all are parts of it
    unsigned plain = 0u, part = 0u;
    if (!scalar) {
        const float zero[4] = {0.f, 0.f, 0.f, 0.f};
        for (int c = 0; c < nc; ++c) {
            bool all = true, sub = true;
            for (int e = 0; e < SC_CHUNK; ++e) {
                const int r = c * SC_CHUNK_ROWS + e * SC_THREADS + tid;
                const int mk = r < nr ? sh.mask[__ldg(g.pid + r0 + r)] : 0;
                rmask[r] = static_cast<unsigned char>(mk);
                all = all && mk == full;
                sub = sub && mk != SC_OTHER;
                u[r] = r < nr ? __ldcg(g.V + r0 + r) : 0.f;
            }
            if (__all_sync(AC_FULL, all)) plain |= 1u << c;
            if (__all_sync(AC_FULL, sub)) part |= 1u << c;
            sc_tst(tp + SC_CHUNK * c, zero);
        }
        sc_wait_st();
    }
    if (tid == 0) {
        sh.ip = gs->ip[0];
        sh.sp = 0.0;
    }
    __syncthreads();
    auto leave = [&]() {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (warp == 0)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem), "n"(SC_TMEM));
    };
    if (lead && g_test_ac_dead_wait != 0) {
        leave();
        return;
    }
    {
        float s[3] = {0.f, 0.f, 0.f};
        target += gridDim.x;
        if (!scalar) {
            for (int r = tid; r < nr; r += SC_THREADS) s[1] = fmaf(u[r], u[r], s[1]);
            sc_publish<3>(s, wb(0), g.bar, scale_b, sh);
        }
    }
    if (!ac_wait<false>(g.bar, target, &st->status, &sh.ok)) {
        leave();
        return;
    }
    // chunks c1..c2-1 gather inside the block; the order of a step's product
    // starts with them, that of its update with the rows the neighbours read
    const int c1 = min(nc, sc_chunks(g.reach)), c2 = max(c1, (nr - g.reach) / SC_CHUNK_ROWS);
    const int hi0 = nr - g.reach;  // rows below reach or from hi0 on are the neighbours' halo
    const int cz = max(0, min(nc - 1, hi0 / SC_CHUNK_ROWS));

    bool broke = false;
    for (int j = 0; j < m; ++j) {
        const int par = j & 1;
        // the last block clears the sums of step j - 1, which every block has read
        // (its threads with rows: their arrival publishes the zeros)
        if (blockIdx.x == gridDim.x - 1 && j > 0 && !scalar) {
            unsigned long long* const z = wa(par ^ 1);
            for (int i = tid; i < 2 * CYCLE_EXCHANGE; i += SC_THREADS) __stcg(z + i, 0ull);
        }
        // the neighbours' rows: requested now, stored after the chunks that need none
        const float* x = g.V + static_cast<size_t>(j) * ldv + r0;
        float hl[SC_CHUNK], hh[SC_CHUNK];
        auto halo_load = [&](int k) {
#pragma unroll
            for (int e = 0; e < SC_CHUNK; ++e) {
                const int i = k + e * SC_THREADS + tid, lo = i - g.reach, hi = nr + i;
                hl[e] = hh[e] = 0.f;
                if (i < g.reach && r0 + lo >= 0) hl[e] = __ldcg(x + lo);
                if (i < g.reach && r0 + hi < g.n) hh[e] = __ldcg(x + hi);
            }
        };
        auto halo_store = [&](int k) {
#pragma unroll
            for (int e = 0; e < SC_CHUNK; ++e) {
                const int i = k + e * SC_THREADS + tid;
                if (i < g.reach) {
                    u[i - g.reach] = hl[e];
                    u[nr + i] = hh[e];
                }
            }
        };
        if (!scalar) halo_load(0);
        // w = A u_j, rounded products added in entry order (the SpMV kernels' sums bit for bit:
        // what a smooth vector's rounding leaves in w is part of what the learned controller was
        // trained on; fused ones cost heat 2048^2 a fifth cycle), u_j.w and |w|^2
        float d0[2] = {0.f, 0.f}, d1[2] = {0.f, 0.f};
        auto product = [&](int c) {
            const int b = c * SC_CHUNK_ROWS + tid;
            float w[SC_CHUNK] = {0.f, 0.f, 0.f, 0.f};
            float xv[SC_CHUNK][L], ur[SC_CHUNK];
            if ((part >> c) & 1u) {
#pragma unroll
                for (int e = 0; e < SC_CHUNK; ++e) {
#pragma unroll
                    for (int q = 0; q < L; ++q) xv[e][q] = u[b + e * SC_THREADS + g.off[q]];
                    ur[e] = u[b + e * SC_THREADS];
                }
                if ((plain >> c) & 1u) {
#pragma unroll
                    for (int e = 0; e < SC_CHUNK; ++e)
#pragma unroll
                        for (int q = 0; q < L; ++q)
                            w[e] = __fadd_rn(w[e], __fmul_rn(g.val[q], xv[e][q]));
                } else {
                    int mk[SC_CHUNK];
#pragma unroll
                    for (int e = 0; e < SC_CHUNK; ++e) mk[e] = rmask[b + e * SC_THREADS];
#pragma unroll
                    for (int e = 0; e < SC_CHUNK; ++e)
#pragma unroll
                        for (int q = 0; q < L; ++q)
                            if ((mk[e] >> q) & 1) w[e] = __fadd_rn(w[e], __fmul_rn(g.val[q], xv[e][q]));
                }
            } else {
                // rows of patterns that are no part of the major one among them: from the table
#pragma unroll
                for (int e = 0; e < SC_CHUNK; ++e) {
                    const int r = b + e * SC_THREADS;
                    ur[e] = u[r];
                    if (r >= nr) continue;
                    const int id = __ldg(g.pid + r0 + r), pl = __ldg(T->len + id);
                    for (int q = 0; q < pl; ++q)
                        w[e] = __fadd_rn(w[e], __fmul_rn(__ldg(T->v32 + id * PAT_LEN + q),
                                                         u[r + __ldg(T->off + id * PAT_LEN + q)]));
                }
            }
            __syncwarp();
            sc_tst(tw + SC_CHUNK * c, w);
            d0[0] += fmaf(ur[0], w[0], ur[1] * w[1]);
            d0[1] += fmaf(ur[2], w[2], ur[3] * w[3]);
            d1[0] += fmaf(w[0], w[0], w[1] * w[1]);
            d1[1] += fmaf(w[2], w[2], w[3] * w[3]);
        };
        target += gridDim.x;
        if (!scalar) {
#pragma unroll 1
            for (int c = c1; c < c2; ++c) product(c);
            halo_store(0);
            for (int k = SC_CHUNK_ROWS; k < g.reach; k += SC_CHUNK_ROWS) {
                halo_load(k);
                halo_store(k);
            }
            sc_rows_sync();
#pragma unroll 1
            for (int i = 0; i < nc - (c2 - c1); ++i) product(i < c1 ? i : i + (c2 - c1));
            sc_wait_st();
            const float s[2] = {d0[0] + d0[1], d1[0] + d1[1]};
            sc_publish<2>(s, wa(par), g.bar, scale_a, sh);
        } else {
            // meanwhile what the last update gave: b_{j-1} = u_{j-1}.u_j, b_j = |u_j|^2,
            // a_{j-1} = w_{j-1}.u_j (A symmetric)
            const int lane = tid & 31;
            if (lane < 3) sh.b[lane] = ac_collect(wb(par), lane, scale_b(lane));
            __syncwarp();
            if (lane == 0) {
                const double bj = sh.b[1], s0 = sh.sp;
                const double sj = (bj > 0.0 && !isinf(bj)) ? rsqrt(bj) : 0.0;
                const double g01 = (s0 * sh.b[0]) * sj, cp = (s0 * sh.b[2]) * sj;
                sh.pre[0] = sj;
                sh.pre[1] = sj * sj;
                sh.pre[2] = g01;
                sh.pre[3] = cp;
                sh.pre[4] = g01 * cp;
                // H(j, j-1) and the breakdown test of main.cu:1911
                int bad = 0;
                if (j >= 1) {
                    const double beta = sqrt(bj) * sh.ip;
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
            __syncwarp();
        }
        if (!ac_wait<false>(g.bar, target, &st->status, &sh.ok)) {
            leave();
            return;
        }
        if (sh.bad) {  // the same sums in every block
            broke = true;
            break;
        }
        if (tid < 2) sh.a[tid] = ac_collect(wa(par), tid, scale_a(tid));
        if (tid < 32) __syncwarp();
        if (tid == 0) {
            // h = c - (G - I) c over the two columns, the update's coefficients,
            // the pre-scale from |w - V h|^2 = |w|^2 - h.c (to first order in G - I)
            const double sj = sh.pre[0], cp = sh.pre[3];
            const double cj = sh.pre[1] * sh.a[0], w2 = sh.pre[1] * sh.a[1];
            double hp = cp, hj = cj;
            if (g.reortho) {
                hp = cp - __dmul_rn(sh.pre[2], cj);
                hj = cj - sh.pre[4];
            }
            double u2 = w2 - hp * cp - hj * cj;
            if (!(u2 > 1e-8 * w2)) u2 = w2;
            const int ex = (__double2hiint(u2) >> 20) & 0x7ff;
            int pe = 0;
            if (u2 > 0.0 && ex > 0 && ex < 0x7ff) pe = min(max((ex - 1023) >> 1, -120), 120);
            sh.cp = static_cast<float>(sh.sp * hp);
            sh.cj = static_cast<float>(sj * hj);
            sh.wsc = static_cast<float>(sj);
            sh.psc = __int_as_float((127 - pe) << 23);
            const double ip = __hiloint2double((1023 + pe) << 20, 0);
            sh.ip = ip;
            if (lead) {
                gs->s[j] = sj;
                gs->ip[j + 1] = ip;
                gs->G[j + static_cast<size_t>(j) * GRAM_LD] = 1.0;
                g.H[j + j * ldh] = hj;
                if (j >= 1) {
                    gs->G[j - 1 + static_cast<size_t>(j) * GRAM_LD] = sh.pre[2];
                    gs->G[j + static_cast<size_t>(j - 1) * GRAM_LD] = sh.pre[2];
                    g.H[(j - 1) + j * ldh] = hp;
                    gs->coef[j - 1] = sh.cp;
                }
                gs->coef[j] = sh.cj;
                gs->wsc = sh.wsc;
                gs->psc = sh.psc;
            }
            sh.sp = sj;
        }
        if (lead)
            for (int r = tid; r < j - 1; r += SC_BLOCK) g.H[r + j * ldh] = 0.0;  // outside the window
        __syncthreads();
        // u_{j+1} = p (s_j w - (c_{j-1} u_{j-1} + c_j u_j)) over u_j, which takes
        // u_{j-1}'s place; the next step's u_j.u_{j+1}, |u_{j+1}|^2 and w.u_{j+1}
        target += gridDim.x;
        if (!scalar) {
            float e0[2] = {0.f, 0.f}, e1[2] = {0.f, 0.f}, e2[2] = {0.f, 0.f};
            float* const out = g.V + static_cast<size_t>(j + 1) * ldv + r0;
            const float cp = sh.cp, cj = sh.cj, wsc = sh.wsc, psc = sh.psc;
#pragma unroll 1
            for (int i = 0; i < nc; ++i) {
                const int c = i + cz < nc ? i + cz : i + cz - nc;
                const int b = c * SC_CHUNK_ROWS + tid;
                float w[4], pv[4], uq[4];
                __syncwarp();
                sc_tld(tw + SC_CHUNK * c, w);
                sc_tld(tp + SC_CHUNK * c, pv);
#pragma unroll
                for (int e = 0; e < SC_CHUNK; ++e) {
                    uq[e] = u[b + e * SC_THREADS];
                    if (b + e * SC_THREADS >= nr) uq[e] = 0.f;  // a halo row's place
                }
                sc_wait_ld(w, pv);
                sc_tst(tp + SC_CHUNK * c, uq);
#pragma unroll
                for (int e = 0; e < SC_CHUNK; ++e) {
                    const int r = b + e * SC_THREADS;
                    const float t = fmaf(w[e], wsc, -fmaf(uq[e], cj, pv[e] * cp)) * psc;
                    if (r < nr) {
                        u[r] = t;
                        if (r < g.reach || r >= hi0) __stcg(out + r, t);
                    }
                    e0[e & 1] = fmaf(uq[e], t, e0[e & 1]);
                    e1[e & 1] = fmaf(t, t, e1[e & 1]);
                    e2[e & 1] = fmaf(w[e], t, e2[e & 1]);
                }
            }
            __syncwarp();
            sc_wait_st();
            const float s[3] = {e0[0] + e0[1], e1[0] + e1[1], e2[0] + e2[1]};
            sc_publish<3>(s, wb(par ^ 1), g.bar, scale_b, sh);
            // the rows no other block reads in this launch
            const int a = sc_halo(g.reach), z = hi0 & ~3;
            for (int i = a + 4 * tid; i < z; i += 4 * SC_THREADS)
                __stcs(reinterpret_cast<float4*>(out + i), *reinterpret_cast<const float4*>(u + i));
            if (tid < 4) {
                if (g.reach + tid < min(a, hi0)) __stcs(out + g.reach + tid, u[g.reach + tid]);
                if (z + tid < hi0 && z + tid >= a) __stcs(out + z + tid, u[z + tid]);
            }
        }
        if (!ac_wait<false>(g.bar, target, &st->status, &sh.ok)) {
            leave();
            return;
        }
    }
    if (!broke && lead && tid == 0) {  // |u_m|: H(m, m-1), s_m
        const double b = ac_collect(wb(m & 1), 1, scale_b(1));
        const double beta = sqrt(b) * sh.ip;
        const bool bad = !(beta >= 1e-14) || isinf(beta);
        if (m < g.ldh) g.H[m + (m - 1) * ldh] = bad ? 0.0 : beta;
        gs->s[m] = (b > 0.0 && !isinf(b)) ? rsqrt(b) : 0.0;
        gs->G[m + static_cast<size_t>(m) * GRAM_LD] = 1.0;
        if (bad) {
            st->breakdown = 1;
            st->k_used = m;
        }
    }
    leave();
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
        for (int i = tid; i < 4 * CYCLE_EXCHANGE; i += SC_BLOCK) __stcg(g.words + i, 0ull);
    }
}

constexpr int SC_SMEM = 227 * 1024 - static_cast<int>(sizeof(ScShared)) - 64;
// More than half an SM's shared memory, whatever a block needs: two blocks of
// different grids on one SM would each wait, the one for tensor memory that
// the other holds, the other at a meeting that the first one's grid delays. A
// cooperative launch does not count tensor memory.
constexpr int SC_SMEM_MIN = 116 * 1024;
static_assert(2 * SC_SMEM_MIN > 228 * 1024, "one block an SM");

int sc_rows(int n) {
    const int blocks = std::min(device_sm_count(), CYCLE_MAX_BLOCKS);
    return ((n + blocks - 1) / blocks + 3) / 4 * 4;
}
size_t sc_bytes(int rows, int reach) {
    const size_t r = static_cast<size_t>(sc_chunks(rows)) * SC_CHUNK_ROWS;
    return sizeof(float) * (r + 2 * static_cast<size_t>(sc_halo(reach))) + r;
}

}  // namespace

bool stencil_cycle_fits(int n, int m, int len, int reach) {
    const int rows = sc_rows(n);
    return m >= 1 && m <= GRAM_M && len >= 1 && len <= STENCIL_LEN && sc_chunks(rows) * SC_CHUNK <= SC_GROUPS &&
           reach < n && sc_bytes(rows, reach) <= static_cast<size_t>(SC_SMEM);
}

int stencil_cycle_prepare() {
    MEXK_CK(cudaFuncSetAttribute(stencil_cycle_kernel<5>, cudaFuncAttributeMaxDynamicSharedMemorySize, SC_SMEM));
    MEXK_CK(cudaFuncSetAttribute(stencil_cycle_kernel<STENCIL_LEN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SC_SMEM));
    return MEXK_OK;
}

int stencil_cycle_test_hook(int enable) {
    const int v = enable ? 1 : 0;
    MEXK_CK(cudaMemcpyToSymbol(g_test_ac_dead_wait, &v, sizeof(int)));
    return MEXK_OK;
}

int launch_stencil_cycle(StencilArgs a, cudaStream_t s) {
    if (a.pid == nullptr || a.scale == INT_MAX || !stencil_cycle_fits(a.n, a.m, a.len, a.reach))
        return MEXK_ERR_INVALID;
    a.rows = sc_rows(a.n);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((a.n + a.rows - 1) / a.rows);
    cfg.blockDim = dim3(SC_BLOCK);
    cfg.dynamicSmemBytes = std::max<size_t>(sc_bytes(a.rows, a.reach), SC_SMEM_MIN);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = a.len <= 5 ? cudaLaunchKernelEx(&cfg, stencil_cycle_kernel<5>, a)
                                     : cudaLaunchKernelEx(&cfg, stencil_cycle_kernel<STENCIL_LEN>, a);
    if (e != cudaSuccess) {
        set_cuda_error(e, "stencil_cycle_kernel", __FILE__, __LINE__);
        return MEXK_ERR_CUDA;
    }
    return MEXK_OK;
}

}  // namespace mexk
