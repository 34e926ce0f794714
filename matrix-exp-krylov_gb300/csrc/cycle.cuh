// Pieces shared by the kernels that run all steps of a basis (arnoldi_cycle.cu,
// gram_cycle.cu): the blocks' meeting and the exact sums over a grid.
#pragma once

#include "gram_step.cuh"

#include <cooperative_groups.h>

namespace mexk {
namespace {

constexpr unsigned AC_FULL = 0xffffffffu;
constexpr unsigned long long AC_WAIT_NS = 1000000000ull;
constexpr unsigned long long AC_TEST_WAIT_NS = 1000000ull;  // the limit under the testing hook

// Testing hook (mexk_test_force_wait_timeout): when set, block 0 of a grid
// leaves before its first meeting, and the others' waits give up after
// AC_TEST_WAIT_NS.
__device__ int g_test_ac_dead_wait = 0;

__device__ __forceinline__ unsigned long long ac_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The blocks' meeting, in two parts. A cluster: the hardware barrier
// (cluster-scope release/acquire). A grid: an arrival counter that only grows
// (bar[0], the next target in `target`), polled with a bounded wait; bar[1] is
// the abort word. Every thread calls both; what is written to shared memory
// between them needs a __syncthreads of its own.
template <bool CLUSTER>
__device__ __forceinline__ void ac_arrive(unsigned* bar, unsigned& target) {
    if constexpr (CLUSTER) {
        cooperative_groups::this_cluster().barrier_arrive();
    } else {
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    }
}
// False when the wait gave up.
template <bool CLUSTER>
__device__ __forceinline__ bool ac_wait(unsigned* bar, unsigned target, int* status, int* s_ok) {
    if constexpr (CLUSTER) {
        cooperative_groups::this_cluster().barrier_wait();
        return true;
    } else {
        if (threadIdx.x == 0) {
            int ok = 1;
            unsigned seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
            if (static_cast<int>(seen - target) < 0) {
                const unsigned long long t0 = ac_ns();
                do {
                    unsigned aborted;
                    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(aborted) : "l"(bar + 1) : "memory");
                    if (aborted != 0u) {
                        ok = 0;
                        break;
                    }
                    const unsigned long long waited = ac_ns() - t0;
                    if (waited > AC_TEST_WAIT_NS) {
                        int hook;  // volatile: not read ahead of the test on every poll
                        asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(hook) : "l"(&g_test_ac_dead_wait) : "memory");
                        if (waited > AC_WAIT_NS || hook != 0) {
                            atomicExch(&bar[1], 1u);
                            atomicOr(status, ST_TIMEOUT);
                            ok = 0;
                            break;
                        }
                    }
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
                } while (static_cast<int>(seen - target) < 0);
            }
            *s_ok = ok;
        }
        __syncthreads();
        return *s_ok != 0;
    }
}
template <bool CLUSTER>
__device__ __forceinline__ bool ac_meet(unsigned* bar, unsigned& target, int* status, int* s_ok) {
    ac_arrive<CLUSTER>(bar, target);
    return ac_wait<CLUSTER>(bar, target, status, s_ok);
}

// ---- exact sums over the blocks of a grid -----------------------------------
// A partial sum x becomes up to three 40-bit digits of the integer
// x / 2^(scale - AC_TOP), added to three of its column's eight 64-bit words
// by integer atomics: the words hold the exact sum of up to 2^23 blocks
// whatever the order of arrival, and every block reads 8 words per column
// instead of one partial per block and column (152 FP64 adds per column cost
// more than the dots themselves). 2^scale bounds every |x|; what lies below
// the last digit, 2^-318 of that bound, rounds off.
constexpr int AC_DIGIT = 40;
constexpr int AC_DIGITS = CYCLE_DIGITS;
constexpr int AC_TOP = AC_DIGIT * AC_DIGITS - 2;
constexpr long long AC_MASK = (1ll << AC_DIGIT) - 1;
// The q-th (0..2) of x's digits, signed; *index its place.
__device__ __forceinline__ long long ac_digit(double x, int scale, int q, int* index) {
    const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(x));
    const int e = static_cast<int>((u >> 52) & 0x7ff);
    *index = 0;
    if (e == 0) return 0;  // zero and subnormals
    unsigned long long m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    int p = e - 1075 - (scale - AC_TOP);  // bit position of m's last bit
    if (p < 0) {
        m = p > -54 ? (m + (1ull << (-p - 1))) >> -p : 0ull;
        p = 0;
    }
    const int base = p / AC_DIGIT, off = p - base * AC_DIGIT;
    *index = min(base + q, AC_DIGITS - 1);
    const unsigned long long v = q == 0   ? (m << off) & AC_MASK
                                 : q == 1 ? (m >> (AC_DIGIT - off)) & AC_MASK
                                          : (off > 2 * AC_DIGIT - 54 ? m >> (2 * AC_DIGIT - off) : 0ull);
    const long long sv = static_cast<long long>(v);
    return (u >> 63) ? -sv : sv;
}
// The double of a column's digits: carries propagated and the sign taken out
// first, then the 64 bits from the highest set one (the next 56 folded into
// the last as a sticky bit) rounded once; integers but for that conversion,
// whose FP64 neighbours would cost 64 cycles each.
__device__ __forceinline__ double ac_value(long long (&d)[AC_DIGITS], int scale) {
#pragma unroll
    for (int i = 0; i + 1 < AC_DIGITS; ++i) {
        d[i + 1] += d[i] >> AC_DIGIT;
        d[i] &= AC_MASK;
    }
    const bool neg = d[AC_DIGITS - 1] < 0;
    if (neg) {
#pragma unroll
        for (int i = 0; i < AC_DIGITS; ++i) d[i] = -d[i];
#pragma unroll
        for (int i = 0; i + 1 < AC_DIGITS; ++i) {
            d[i + 1] += d[i] >> AC_DIGIT;
            d[i] &= AC_MASK;
        }
    }
    unsigned long long h2 = 0, h1 = 0, h0 = 0;
    int top = 0;
#pragma unroll
    for (int i = 0; i < AC_DIGITS; ++i)
        if (d[i] != 0) {
            h2 = static_cast<unsigned long long>(d[i]);
            h1 = i >= 1 ? static_cast<unsigned long long>(d[i >= 1 ? i - 1 : 0]) : 0ull;
            h0 = i >= 2 ? static_cast<unsigned long long>(d[i >= 2 ? i - 2 : 0]) : 0ull;
            top = i;
        }
    if (h2 == 0ull) return 0.0;
    const int lz = __clzll(static_cast<long long>(h2));  // 1..63: the top digit is positive
    const unsigned long long rest = (h1 << (64 - AC_DIGIT)) | (h0 >> (2 * AC_DIGIT - 64));
    unsigned long long bits = (h2 << lz) | (rest >> (64 - lz));
    if ((rest << lz) != 0ull) bits |= 1ull;
    const double r = __ull2double_rn(bits);
    const int e = scale - AC_TOP + AC_DIGIT * top - lz;  // r in [2^63, 2^64]
    double v;
    if (e > -1084 && e < 958) v = __hiloint2double(__double2hiint(r) + (e << 20), __double2loint(r));
    else v = ldexp(r, e);
    return neg ? -v : v;
}

// Adds columns' totals over the row slices (red[q * ld + c], q < slices) to
// the exchange's words: four adjacent lanes per column; every thread calls it.
template <int THREADS>
__device__ __forceinline__ void ac_publish(unsigned long long* words, const double* red, int ld, int k, int slices,
                                           int scale) {
    for (int t = threadIdx.x; t < ((4 * k + 31) & ~31); t += THREADS) {
        const int c = min(t >> 2, k - 1), q = t & 3;
        double s = q < slices ? red[q * ld + c] : 0.0;
        for (int i = q + 4; i < slices; i += 4) s += red[i * ld + c];
        s += __shfl_xor_sync(AC_FULL, s, 1);
        s += __shfl_xor_sync(AC_FULL, s, 2);
        if ((t >> 2) < k) {
            const bool finite = (__double2hiint(s) & 0x7ff00000) != 0x7ff00000;
            if (q < 3 && finite) {
                int i;
                const long long d = ac_digit(s, scale, q, &i);
                if (d != 0) atomicAdd(words + AC_DIGITS * c + i, static_cast<unsigned long long>(d));
            } else if (q == 3 && !finite) {
                atomicAdd(words + AC_DIGITS * MEXK_M_MAX, 1ull);
            }
        }
    }
}
// Column c's sum after the meeting (NaN when a partial was not finite).
__device__ __forceinline__ double ac_collect(const unsigned long long* words, int c, int scale) {
    const ulonglong2* w = reinterpret_cast<const ulonglong2*>(words + AC_DIGITS * c);
    long long d[AC_DIGITS];
#pragma unroll
    for (int i = 0; i < AC_DIGITS; i += 2) {
        const ulonglong2 p = __ldcg(w + i / 2);
        d[i] = static_cast<long long>(p.x);
        d[i + 1] = static_cast<long long>(p.y);
    }
    const bool finite = __ldcg(words + AC_DIGITS * MEXK_M_MAX) == 0ull;
    const double v = ac_value(d, scale);
    return finite ? v : __longlong_as_double(0x7ff8000000000000ll);
}

}  // namespace
}  // namespace mexk
