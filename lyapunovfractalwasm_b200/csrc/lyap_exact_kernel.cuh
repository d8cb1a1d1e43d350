// lyap_exact_kernel.cuh -- the exact lambda kernel (FractalComputer::computeFractal, reference
// src/lyapunov_fractal.hpp:41-86).  Included by lyap_kernels.cu (compiled by nvcc into the library) and, as text,
// by the run-time specialiser (lyap_jit.cu), which compiles one more instance of the same code with the sequence's
// group patterns as compile-time constants.  Keep it free of host-only headers.
#pragma once

#include "lyap_args.h"
#include "lyap_math.h"

namespace lyap {

static __device__ const lyap_logtab_entry g_lyap_logtab[LYAP_LOG_BINS] = {LYAP_LOG_TABLE_INIT};

// ---------------------------------------------------------------------------------------------
// Exact lambda kernel.
//
// One thread owns P pixels of one column, one below another, for their whole orbit: x, the running log sum
// and the parameter values stay in registers.  The per-step A/B(/C) choice is the same for every
// pixel, so steps are taken in groups of U whose pattern (e.g. "AB", "BA") picks, by one warp-uniform
// multiway branch, a straight-line body compiled for exactly that pattern: no per-step select or branch.
// Inside a body the orbit runs ahead and the U*P logarithms that hang off it are independent chains.
//
// The log table (1024 entries x 16 B) sits in shared memory in 8 interleaved copies: entry i of
// copy c is at slot i*8+c and a lane uses copy (lane & 7).  A 16-byte load per lane is served per
// quarter warp, whose 8 lanes then hit 8 different 16-byte bank groups whatever their indices are,
// so the lookups never conflict.
//
// Steps run in chunks of 32 to kMaxChunk (fewer at a region's end) without per-step exit tests.  That is sound because leaving (0,1)
// is permanent for x <- r x (1-x) with r > 0 (x >= 1 gives x <= 0 next, x <= 0 stays <= 0, NaN stays
// NaN), so testing x after the chunk finds every exit, and the only other irregular event, a zero
// derivative (x == 0.5 exactly, skipped and not counted by the reference, :71-74), has exponent field 0,
// for which the exponent table holds -inf: the running sum turns non-finite.  A chunk in which anything irregular
// happened is rolled back and redone by `careful_chunk` / `careful_steps`, which follow the reference step by step.
// ---------------------------------------------------------------------------------------------

constexpr int kTabCopies = 8;
constexpr size_t kTabSmemBytes = (size_t)LYAP_LOG_BINS * kTabCopies * sizeof(lyap_logtab_entry);  // 128 KB
// Second shared table, indexed by the top 12 bits of HALF the derivative (sign + exponent field e - 1, where e is the
// derivative's own field): {e*LN2HI (exact), (e-1023)*LN2LO}.  It replaces an integer->double conversion and one fma per
// logarithm, and it carries the irregular cases: entry 0 (zero or subnormal) is -inf and entries >= 2046 (a derivative
// that is inf or NaN, sign bit) are NaN, so such a step poisons the running sum and the chunk is redone step by step.
constexpr int kExpEntries = 4096;
constexpr size_t kExpSmemBytes = (size_t)kExpEntries * sizeof(double2);                              // 64 KB
constexpr size_t kExactSmemBytes = kTabSmemBytes + kExpSmemBytes;
__device__ __forceinline__ bool in_unit_interval(double x) { return x > 0.0 && x < 1.0; }

// parameter values the chunked fast path may be used with: positive, finite, 2^-500 < r < 2^500
__device__ __forceinline__ bool ordinary_param(double r) {
    const unsigned hw = (unsigned)__double2hiint(r);
    return (hw - 0x20B00000u) < (0x5F300000u - 0x20B00000u);
}

struct PixelState {
    double x, lyap;
    int valid;
};

// Reference semantics, one step at a time, for `n` steps of selector word `word`.
// Returns true when the orbit left (0,1) (the reference's break).  *steps counts executed updates.
template <bool ACC>
__device__ __noinline__ bool careful_chunk(PixelState* ps, double rA, double rB, double rC, unsigned word, int n,
                                           unsigned long long* steps) {
    double x = ps->x, lyap = ps->lyap;
    int valid = ps->valid;
    bool dead = false;
    int j = 0;
    for (; j < n; ++j) {
        const unsigned sel = (word >> (2 * j)) & 3u;
        const double r = sel == 0 ? rA : (sel == 1 ? rB : rC);
        if (ACC) {
            const double deriv = fabs(__dmul_rn(r, __dsub_rn(1.0, __dmul_rn(2.0, x))));   // :69
            if (deriv > 0.0) {                                                              // :71
                lyap = __dadd_rn(lyap, lyap_log_tab(deriv, g_lyap_logtab, 1));              // :72
                ++valid;
            }
        }
        x = __dmul_rn(__dmul_rn(r, x), __dsub_rn(1.0, x));                                  // :58,76
        if (!in_unit_interval(x)) {                                                         // :60,78
            dead = true;
            ++j;
            break;
        }
    }
    *steps += (unsigned long long)j;
    ps->x = x;
    ps->lyap = lyap;
    ps->valid = valid;
    return dead;
}

// |r*(1-2x)| / 2 for r > 0, with the reference's rounding: 1 - 2x = 2*(0.5 - x), and a factor of two changes no rounding
// (the smallest non-zero 0.5 - x is 2^-54, so nothing gets near the subnormals for ordinary r).  The subtraction reads one
// register pair where fma(-2, x, 1) reads two, its second constant being one: the lambda kernel is bound by register reads
// (a 64-bit pair a cycle and scheduler: two-operand fp64 instructions alone use them up, measured 1.98 cycles each, 2.96
// with three distinct registers), and this one read fewer took 4096 x 2048 pixels of
// "AABAB" 200 + 2000 from 16.11 to 15.73 ms.  Together the fp64 pipe (77 % busy on
// the 4096^2 frame), the shared-memory data pipe (80 %, two 16-byte look-ups a logarithm) and the register reads of the seven
// other instructions leave no gap that a change of one of them would fill.
__device__ __forceinline__ double half_derivative(double r, double x) { return __dmul_rn(r, fabs(__dsub_rn(0.5, x))); }

// Constants of the log core in constant memory: fp64 instructions take them as constant-bank
// operands, which costs no instruction (64-bit immediates would each need two moves).
struct LogConsts {
    double c2, c3, c4, ln2hi, ln2lo, klo_bias;
};
static __constant__ LogConsts c_logk = {LYAP_LOG_C2, LYAP_LOG_C3, LYAP_LOG_C4, LYAP_LN2HI, LYAP_LN2LO, LYAP_KLO_BIAS};
static __constant__ int c_minus_2p20 = -(1 << 20);   // read as a constant-bank operand so the product below stays one multiply-add

// lyap_log_core (lyap_math.h) of 2*d for a positive normal d, written against the two shared-memory tables, which start
// at the beginning of the dynamic shared memory: `lane_off` is the byte offset of this lane's copy inside a
// mantissa-table entry group ((lane & 7) * 16; groups are kTabCopies*16 bytes apart), or'ed into the bin offset so
// that the address is one logic operation plus a constant.  Same values in the same order as
// lyap_log_core (e*LN2HI + lp and (e-1023)*LN2LO are tabulated instead of computed), so same bits.
__device__ __forceinline__ double log_fast(double d, unsigned lane_off) {
    const unsigned hw = (unsigned)__double2hiint(d);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // bin index * 128 bytes, or'ed with this lane's copy offset (lane_off = (lane & 7) * 16)
    const unsigned off = ((hw >> 3) & (unsigned)((LYAP_LOG_BINS - 1) * kTabCopies * 16)) | lane_off;
    const double2 me = *reinterpret_cast<const double2*>(smem_raw + off);
    const double lp = me.x, invcb = me.y;
    const unsigned ke = hw >> 20;
    const double2 ee = reinterpret_cast<const double2*>(smem_raw + kTabSmemBytes)[ke];
    const double khi = ee.x, klo = ee.y;
    // The mantissa table holds invc with 0x3FF00000 added to its high word, so subtracting d's exponent field
    // gives invc * 2^-(exponent of d): d * that == mantissa(d) * invc exactly (a power-of-two rescaling),
    // without assembling the mantissa as a separate double.
    int invs_hi;
    asm("mad.lo.s32 %0, %1, %2, %3;" : "=r"(invs_hi) : "r"((int)ke), "r"(c_minus_2p20), "r"(__double2hiint(invcb)));
    const double invs = __hiloint2double(invs_hi, __double2loint(invcb));
    const double r = __fma_rn(d, invs, -1.0);
    double q = __fma_rn(r, c_logk.c4, c_logk.c3);
    q = __fma_rn(r, q, c_logk.c2);
    const double w = __fma_rn(r, q, 1.0);
    const double s = __fma_rn(r, w, klo);
    const double hi = __dadd_rn(khi, lp);      // exact: both on the 2^-42 grid
    return __dadd_rn(hi, s);
}

// The selectors of step j and the 15 behind it, of a region whose words start at `sel` and repeat every `wrap`.
__device__ __forceinline__ unsigned selectors_from(const unsigned* sel, int wrap, int j) {
    const int w = (j / kStepsPerWord) % wrap;
    return __funnelshift_r(sel[w], sel[w + 1 == wrap ? 0 : w + 1], 2 * (j & (kStepsPerWord - 1)));
}

// careful_chunk for steps [first, first + n) of a region whose selector words start at `sel` (n <= kMaxChunk).
// An orbit that has fallen below 2^-740 and whose parameters (positive: the others are sentinels) are at most 256 stays
// below 2^-100 (2^(8 kMaxChunk - 740)) for these steps, where 1 - 2x and 1 - x round to 1: the derivative is the parameter
// itself, with one of at most three logarithms, and a step is a multiplication, an addition and the exit test.  That is how
// nearly every orbit of a frame over [0,4]^2 that ends does end (x runs down to zero where rA*rB < 1), a whole region's after
// one another.  Sixteen such steps at a time are taken without a look at the orbit in between.
// Measured, 800 x 800 over [0.01,3.99]^2, "AB" 100 + 1000: 0.745 -> 0.702 ms (0.645 for a window without exits).
template <bool ACC>
__device__ __noinline__ bool careful_steps(PixelState* ps, double rA, double rB, double rC, const unsigned* sel, int wrap, int first,
                                           int n, unsigned long long* steps) {
    bool dead = false;
    int j = first;
    const int end = first + n;
    if (ps->x < 0x1p-740 && rA <= 256.0 && rB <= 256.0) {
        const unsigned codes = rC > 0.0 && rC <= 256.0 ? 3 : 2;   // parameters that may be used this way
        double x = ps->x, lyap = ps->lyap, zA = 0.0, zB = 0.0, zC = 0.0;
        if (ACC) {
            zA = lyap_log_tab(rA, g_lyap_logtab, 1);
            zB = lyap_log_tab(rB, g_lyap_logtab, 1);
            zC = lyap_log_tab(rC, g_lyap_logtab, 1);
        }
        while (j < end && !dead) {   // leaves at a step that uses another one: the rest is walked below
            const int stop = min(j + kStepsPerWord, end);
            unsigned word = selectors_from(sel, wrap, j);
            // sixteen steps without looking: zero is where the orbit stays, and is looked for at their end
            if (stop - j == kStepsPerWord && (word & 0xAAAAAAAAu) == 0) {
                double y = x, sum = lyap;
#pragma unroll
                for (int k = 0; k < kStepsPerWord; ++k) {
                    const bool is_b = (word >> (2 * k)) & 1u;
                    y = __dmul_rn(is_b ? rB : rA, y);
                    if (ACC) sum = __dadd_rn(sum, is_b ? zB : zA);
                }
                if (y > 0.0) {
                    x = y;
                    lyap = sum;
                    j = stop;
                    continue;
                }
            }
            for (; j < stop && !dead; ++j, word >>= 2) {
                const unsigned code = word & 3u;
                if (code >= codes) break;
                x = __dmul_rn(code == 0 ? rA : (code == 1 ? rB : rC), x);
                if (ACC) lyap = __dadd_rn(lyap, code == 0 ? zA : (code == 1 ? zB : zC));
                dead = !(x > 0.0);
            }
            if (j < stop && !dead) break;
        }
        if (ACC) ps->valid += j - first;
        *steps += (unsigned long long)(j - first);
        ps->x = x;
        ps->lyap = lyap;
    }
    while (j < end && !dead) {
        const int m = min(kStepsPerWord, end - j);
        dead = careful_chunk<ACC>(ps, rA, rB, rC, selectors_from(sel, wrap, j), m, steps);
        j += m;
    }
    return dead;
}

// An orbit whose value at the end of a chunk is, bit for bit, the one a whole number of periods ago goes round the same values
// for good (nothing else enters a step), and a stable one comes to that after some 36/|lambda| steps: on the 4096^2 frame of
// "AABAB" 200 + 2000 41 % of all steps follow in warps all of whose orbits have.  They are not walked.  Measured, together with
// the launch-wide queue of tiles, which such uneven tiles need (without it the first is 20.3 ms and the last 2.44): that frame
// 31.3 -> 19.1 ms, 8192 x 4096 of "BBBBBBAAAAAA" 500 + 4000 over [3.4,4]x[2.5,3.4] 125 -> 69.9, 800 x 600 of "AB" 100 + 10000
// over [0.01,3.99]^2 4.43 -> 1.56; 2048^2 over [3.9,4]^2, where no orbit comes into a cycle, 8.00 -> 8.15.
//
// The longest cycle whose logarithms are kept (640 bytes a thread of local memory), and the chunks after which another value of
// the orbit becomes the reference, at first: cycles that do not go into a chunk are found when they go into up to that many.
// (Rounding makes cycles of nine from cycles of three.)
constexpr int kMaxCycle = 80, kRefChunks = 6;
static_assert(kMaxCycle >= kMaxChunk && kMaxCycle % 4 == 0 && kLeastLeft >= kMaxCycle, "a cycle that goes into a chunk is never too long");

// The last n steps of an orbit that has come back to an earlier value, from step `first` of a region whose selector words start
// at `sel` and repeat every `period` steps: it goes round the same values for good, so the logarithms of one turn are taken and
// the rest of the sum is added up from them.  False (and nothing done) when a turn has more than kMaxCycle steps.
__device__ __noinline__ bool cycle_steps(PixelState* ps, double rA, double rB, double rC, const unsigned* sel, int wrap, int period,
                                         int first, int n, unsigned lane_off) {
    double z[kMaxCycle];
    const double x0 = ps->x;
    double x = x0, sum = 0.0, below = 0.0, above = 0.0;
    int len = 0, zeros = 0, wi = (first / kStepsPerWord) % wrap, in_word = first & (kStepsPerWord - 1);
    unsigned word = sel[wi] >> (2 * in_word);
    do {
        if (len + period > kMaxCycle) return false;
        for (int k = 0; k < period; ++k, ++len) {
            const unsigned code = word & 3u;
            word >>= 2;
            if (++in_word == kStepsPerWord) {
                in_word = 0;
                if (++wi == wrap) wi = 0;
                word = sel[wi];
            }
            const double r = code == 0 ? rA : (code == 1 ? rB : rC);
            const double d = half_derivative(r, x);
            x = __dmul_rn(__dmul_rn(r, x), __dsub_rn(1.0, x));
            double t = -0.0;   // a step whose derivative is zero (:71): adding it changes nothing, and no logarithm is -0
            if (d > 0.0) t = log_fast(d, lane_off);
            else ++zeros;
            z[len] = t;
            sum = __dadd_rn(sum, t);
            below = sum < below ? sum : below;
            above = sum > above ? sum : above;
        }
    } while (x != x0);
    for (int k = len; k & 3; ++k) z[k] = -0.0;
    ps->lyap = lyap_cycle_sum(z, len, below, above, ps->lyap, n);
    ps->valid += n;
    if (zeros) {
        ps->valid -= zeros * (n / len);
        for (int k = 0; k < n % len; ++k) ps->valid -= (unsigned long long)__double_as_longlong(z[k]) == 0x8000000000000000ull;
    }
    return true;
}

// U consecutive logistic steps of all P pixels, selector bits in `word` (step j at bits 2j, 2j+1).
// Written as one straight-line block: the orbit x (3 dependent fp64 operations per step) runs ahead
// and leaves the U derivatives behind, whose logarithms are independent of each other and of the orbit,
// so the scheduler has U*P log chains to interleave.  The sum is still accumulated in step order.
// The warp-uniform parameter choice is a select (no branch, so the block stays one scheduling region).
template <int P, bool ACC, bool HAS_C, int U>
__device__ __forceinline__ void fast_group(double (&x)[P], double (&lyap)[P], double rA, const double (&rB)[P], double rC, unsigned word, unsigned lane_off) {
    double d[U][P];
#pragma unroll
    for (int j = 0; j < U; ++j) {
        const bool not_a = (word >> (2 * j)) & 1u;
        const bool is_c = (word >> (2 * j + 1)) & 1u;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            double r = not_a ? rB[p] : rA;
            if (HAS_C) r = is_c ? rC : r;
            if (ACC) {
                d[j][p] = half_derivative(r, x[p]);
            }
            x[p] = __dmul_rn(__dmul_rn(r, x[p]), __dsub_rn(1.0, x[p]));
        }
    }
    if (ACC) {
        double z[U][P];
#pragma unroll
        for (int j = 0; j < U; ++j)
#pragma unroll
            for (int p = 0; p < P; ++p) z[j][p] = log_fast(d[j][p], lane_off);
#pragma unroll
        for (int p = 0; p < P; ++p) {
#pragma unroll
            for (int j = 0; j < U; ++j) lyap[p] = __dadd_rn(lyap[p], z[j][p]);
        }
    }
}

// U steps whose parameter choices are known at compile time (PAT: 2 bits per step, 0 = A, 1 = B, 2 = C):
// no selects, no per-step branches; every operand is fixed.
template <int P, bool ACC, int U, unsigned PAT>
__device__ __forceinline__ void fixed_group(double (&x)[P], double (&lyap)[P], double rA, const double (&rB)[P], double rC, unsigned lane_off) {
    double d[U][P];
#pragma unroll
    for (int j = 0; j < U; ++j) {
        const unsigned code = (PAT >> (2 * j)) & 3u;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const double r = code == 0 ? rA : (code == 1 ? rB[p] : rC);
            if (ACC) {
                d[j][p] = half_derivative(r, x[p]);
            }
            x[p] = __dmul_rn(__dmul_rn(r, x[p]), __dsub_rn(1.0, x[p]));
        }
    }
    if (ACC) {
        double z[U][P];
#pragma unroll
        for (int j = 0; j < U; ++j)
#pragma unroll
            for (int p = 0; p < P; ++p) z[j][p] = log_fast(d[j][p], lane_off);
#pragma unroll
        for (int p = 0; p < P; ++p) {
#pragma unroll
            for (int j = 0; j < U; ++j) lyap[p] = __dadd_rn(lyap[p], z[j][p]);
        }
    }
}

// 1 bit per step -> 2 bits per step (A/B patterns)
__host__ __device__ constexpr unsigned spread_bits(unsigned m) {
    return (m & 1u) | ((m & 2u) << 1) | ((m & 4u) << 2) | ((m & 8u) << 3);
}

// One group of U steps, dispatched on its pattern index to the matching straight-line body: one
// warp-uniform multiway branch per U steps instead of a choice per step.
//   !HAS_C: idx has one bit per step (0 = A, 1 = B), U is 2 or 4.   HAS_C: idx is the raw 2-bit codes, U is 2.
template <int P, bool ACC, bool HAS_C, int U>
__device__ __forceinline__ void dispatch_group(double (&x)[P], double (&lyap)[P],
                                               double rA, const double (&rB)[P], double rC, unsigned idx,
                                               unsigned lane_off) {
#define LYAP_CASE_AB(N) \
    case N: fixed_group<P, ACC, U, spread_bits(N)>(x, lyap, rA, rB, rC, lane_off); break;
#define LYAP_CASE_RAW(N) \
    case N: fixed_group<P, ACC, U, N>(x, lyap, rA, rB, rC, lane_off); break;
    if (HAS_C) {
        static_assert(!HAS_C || U == 2, "three-parameter groups are two steps long");
        switch (idx) {
            LYAP_CASE_RAW(0x0) LYAP_CASE_RAW(0x1) LYAP_CASE_RAW(0x2) LYAP_CASE_RAW(0x4) LYAP_CASE_RAW(0x5)
            LYAP_CASE_RAW(0x6) LYAP_CASE_RAW(0x8) LYAP_CASE_RAW(0x9) LYAP_CASE_RAW(0xA)
            default: break;   // code 3 is never produced by the host packing
        }
    } else if (U == 2) {
        if (idx & 1u) {
            if (idx & 2u) fixed_group<P, ACC, U, spread_bits(3)>(x, lyap, rA, rB, rC, lane_off);
            else fixed_group<P, ACC, U, spread_bits(1)>(x, lyap, rA, rB, rC, lane_off);
        } else {
            if (idx & 2u) fixed_group<P, ACC, U, spread_bits(2)>(x, lyap, rA, rB, rC, lane_off);
            else fixed_group<P, ACC, U, spread_bits(0)>(x, lyap, rA, rB, rC, lane_off);
        }
    } else {
        switch (idx) {
            LYAP_CASE_AB(0) LYAP_CASE_AB(1) LYAP_CASE_AB(2) LYAP_CASE_AB(3) LYAP_CASE_AB(4) LYAP_CASE_AB(5)
            LYAP_CASE_AB(6) LYAP_CASE_AB(7) LYAP_CASE_AB(8) LYAP_CASE_AB(9) LYAP_CASE_AB(10) LYAP_CASE_AB(11)
            LYAP_CASE_AB(12) LYAP_CASE_AB(13) LYAP_CASE_AB(14) LYAP_CASE_AB(15)
            default: break;
        }
    }
#undef LYAP_CASE_AB
#undef LYAP_CASE_RAW
}

// even bits of w packed into the low 16 bits
__device__ __forceinline__ unsigned compress_even_bits(unsigned w) {
    w &= 0x55555555u;
    w = (w | (w >> 1)) & 0x33333333u;
    w = (w | (w >> 2)) & 0x0F0F0F0Fu;
    w = (w | (w >> 4)) & 0x00FF00FFu;
    w = (w | (w >> 8)) & 0x0000FFFFu;
    return w;
}

// n steps of selector word `word` (2 bits per step: 0 = A, 1 = B, 2 = C).
template <int P, bool ACC, bool HAS_C, int UNROLL>
__device__ __forceinline__ void fast_chunk(double (&x)[P], double (&lyap)[P], double rA, const double (&rB)[P], double rC, unsigned word, int n, unsigned lane_off) {
    constexpr int U = HAS_C ? 2 : UNROLL;
    unsigned pat = HAS_C ? word : compress_even_bits(word);
    constexpr int kBits = HAS_C ? 2 * U : U;
    const int groups = n / U;
#pragma unroll 1
    for (int h = 0; h < groups; ++h) {
        dispatch_group<P, ACC, HAS_C, U>(x, lyap, rA, rB, rC, pat & ((1u << kBits) - 1u), lane_off);
        pat >>= kBits;
    }
    if constexpr (U == 2) {
        if (n % U) fast_group<P, ACC, HAS_C, 1>(x, lyap, rA, rB, rC, word >> (2 * (n - 1)), lane_off);
    } else {
#pragma unroll 1
        for (int j = n & ~(U - 1); j < n; ++j) fast_group<P, ACC, HAS_C, 1>(x, lyap, rA, rB, rC, word >> (2 * j), lane_off);
    }
}

// ---- run-time specialisation -------------------------------------------------------------------
// For a periodic sequence the pattern of every 2-step group repeats every KG groups (KG = lcm(period, 2) / 2).
// With the KG patterns known at compile time (PATS: 4 bits per group = two 2-bit codes) a whole period is one
// straight-line block: no dispatch at all.
template <int P, bool ACC, int KG, unsigned long long PATS, int G = 0>
__device__ __forceinline__ void period_block(double (&x)[P], double (&lyap)[P], double rA, const double (&rB)[P],
                                             double rC, unsigned lane_off) {
    if constexpr (G < KG) {
        fixed_group<P, ACC, 2, (unsigned)((PATS >> (4 * G)) & 15ull)>(x, lyap, rA, rB, rC, lane_off);
        period_block<P, ACC, KG, PATS, G + 1>(x, lyap, rA, rB, rC, lane_off);
    }
}

__host__ __device__ constexpr bool pats_use_c(unsigned long long pats) {
    return (pats & 0xAAAAAAAAAAAAAAAAull) != 0;
}

// The orbits and stores of one warp-tile: this lane's pixels (row + p, col), p < P, of the launch; a lane that is not
// `inside` has none.  The pixels of a thread lie below one another: they share the column's parameter, one register pair
// instead of P, which the instructions of an A step read one after the other; orbits that end do so at much the same time
// in 32 columns, less so in 32 * P; and each store of a warp covers 32 neighbours.
// KG == 0: patterns dispatched at run time; KG > 0: WU_PATS / ACC_PATS are the regions' group patterns.
template <int P, bool HAS_C, int UNROLL, int KG, unsigned long long WU_PATS, unsigned long long ACC_PATS>
__device__ __forceinline__ void exact_tile(const LambdaArgs& a, long long row, int col, bool inside, double* __restrict__ out64,
                                           float* __restrict__ out32, unsigned lane_off, unsigned long long& my_steps) {
    double x[P], lyap[P], rB[P], lam[P];
    const double rA = __dadd_rn(a.min_x, __dmul_rn(a.dx, (double)col));                          // :45
    const double rC = a.c_value;
    int valid[P];
    bool done[P], careful_only[P];
    double ref[P];        // an earlier value of the orbit, from a step that is a multiple of the sequence's period ago
    bool in_cycle[P], no_cycle[P];   // it has come back to one (and at every later test does); its cycle is too long
    int ref_left = 1, ref_chunks = kRefChunks;   // chunks up to the next such value, and from it to the one after
#pragma unroll
    for (int p = 0; p < P; ++p) {
        rB[p] = __dadd_rn(a.min_y, __dmul_rn(a.dy, (double)(int)(a.row_begin + row + p)));       // :42
        x[p] = 0.5;                                                                               // :31,52
        lyap[p] = 0.0;
        valid[p] = 0;
        lam[p] = -5.0;
        done[p] = !inside || rA <= 0.0 || rB[p] <= 0.0;                                           // :47-50
        careful_only[p] = !(ordinary_param(rA) && ordinary_param(rB[p]) && a.fast_ok_c);
        ref[p] = 0.0;
        in_cycle[p] = false;
        no_cycle[p] = careful_only[p];
    }
    // Behind every whole chunk of the accumulation, whose steps are a multiple of the period, while steps enough are left for it
    // to pay: the pixels whose orbit stands where it stood a chunk ago or at the reference value are in a cycle, and when all of
    // the warp's are (or have ended), the `left` steps from `next` on are added up from one turn of each (cycle_steps).  Lanes
    // that are in one before the others go on walking -- refilling them with other pixels costs more in warm-ups run for a part
    // of a warp than it saves --, but for those in `redone`, which had this chunk walked step by step (a derivative of zero) and
    // would have every other.  The generic kernel has no registers left for the reference value (it spills: 1.02 -> 1.07 ms); its
    // chunks hold cycles of three where they can.
    auto cycles = [&](const double (&sx)[P], unsigned redone, const unsigned* sel, int wrap, int period, int next, int left) {
        bool all = true;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            in_cycle[p] = in_cycle[p] || x[p] == sx[p] || (KG > 0 && x[p] == ref[p]);
            all = all && (done[p] || (in_cycle[p] && !no_cycle[p]));
        }
        if (KG > 0 && --ref_left == 0) {
            ref_left = ref_chunks;
            ref_chunks += ref_chunks / 2;
#pragma unroll
            for (int p = 0; p < P; ++p) ref[p] = x[p];
        }
        const bool every = __all_sync(0xFFFFFFFFu, all);
        if (!every && !__any_sync(0xFFFFFFFFu, redone != 0)) return;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            bool ended = false;
            if (!done[p] && in_cycle[p] && !no_cycle[p] && (every || (redone >> p & 1u))) {
                PixelState ps{x[p], lyap[p], valid[p]};
                ended = cycle_steps(&ps, rA, rB[p], rC, sel, wrap, period, next, left, lane_off);
                if (ended) {
                    done[p] = true;
                    lam[p] = ps.valid > 0 ? __ddiv_rn(ps.lyap, __dmul_rn((double)ps.valid, LYAP_LN2)) : -5.0;
                    my_steps += (unsigned long long)left;
                    x[p] = 0.25;
                } else {
                    no_cycle[p] = true;
                }
            }
            const unsigned lanes = __ballot_sync(0xFFFFFFFFu, ended);
            if (a.cycle_steps && lanes && (threadIdx.x & 31) == 0) atomicAdd(a.cycle_steps, (unsigned long long)left * __popc(lanes));
        }
    };

    for (int region = 0; region < 2; ++region) {
        const bool acc = region == 1;
        const int nsteps = acc ? a.iterations : a.warmup;
        const int word0 = acc ? a.acc_word0 : 0;
        const int wrap = acc ? a.acc_wrap : a.wu_wrap;
        if constexpr (KG > 0) {
            // specialised walk: chunks of REP blocks of CB whole periods (>= 16 steps each), then one block, whole periods, single steps
            // REP = 2 blocks between exit tests measured best (1: more tests and state copies; 3 and more: slower code); three of
            // 16 steps hold cycles of three too.  A warp of small tiles that is alone on its scheduler waits some 250 cycles behind
            // every chunk, but replays all of it when an orbit ends there: 128 x 96 of "AABAB" 100 + 4000 over [3.9,4]^2 in chunks of
            // two / three / four blocks 126 / 118 / 113 us, 205 x 165 90 + 478 over [0,4]^2 56 / 55 / 73.
            constexpr int BS = 2 * KG, CB = (kStepsPerWord + BS - 1) / BS, BLOCK = CB * BS;
            constexpr int REP = BLOCK == kStepsPerWord || (P == 1 && BLOCK <= 20) ? 3 : 2, CS = BLOCK * REP;
            static_assert(CS <= kMaxChunk, "an orbit's fall is replayed on the strength of it");
            const unsigned* sel = a.sel + word0;
            int s = 0;
            while (s < nsteps) {
                bool all_done = true;
#pragma unroll
                for (int p = 0; p < P; ++p) all_done = all_done && done[p];
                if (__all_sync(0xFFFFFFFFu, all_done)) break;
                const int left = nsteps - s;
                const int n = left >= CS ? CS : (left >= CB * BS ? CB * BS : (left >= BS ? left / BS * BS : left));
                double sx[P], sl[P];
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    sx[p] = x[p];
                    sl[p] = lyap[p];
                }
                if (left >= CB * BS) {        // CB whole periods, straight-line, REP times (or once)
#pragma unroll 1
                    for (int rep = n / (CB * BS); rep > 0; --rep) {
#pragma unroll
                        for (int b = 0; b < CB; ++b) {
                            if (acc) period_block<P, true, KG, ACC_PATS>(x, lyap, rA, rB, rC, lane_off);
                            else period_block<P, false, KG, WU_PATS>(x, lyap, rA, rB, rC, lane_off);
                        }
                    }
                } else if (left >= BS) {      // the last few whole periods
#pragma unroll 1
                    for (int b = 0; b < n / BS; ++b) {
                        if (acc) period_block<P, true, KG, ACC_PATS>(x, lyap, rA, rB, rC, lane_off);
                        else period_block<P, false, KG, WU_PATS>(x, lyap, rA, rB, rC, lane_off);
                    }
                } else {                      // less than one period: one step at a time
#pragma unroll 1
                    for (int j = s; j < nsteps; ++j) {
                        const unsigned code = (sel[(j / kStepsPerWord) % wrap] >> (2 * (j & (kStepsPerWord - 1)))) & 3u;
                        if (acc) fast_group<P, true, HAS_C, 1>(x, lyap, rA, rB, rC, code, lane_off);
                        else fast_group<P, false, HAS_C, 1>(x, lyap, rA, rB, rC, code, lane_off);
                    }
                }
                unsigned redone = 0;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    if (done[p]) continue;
                    const bool regular = !careful_only[p] && in_unit_interval(x[p]) && isfinite(lyap[p]);
                    if (regular) {
                        if (acc) valid[p] += n;
                        my_steps += (unsigned long long)n;
                    } else {
                        PixelState ps{sx[p], sl[p], valid[p]};
                        const bool dead = acc ? careful_steps<true>(&ps, rA, rB[p], rC, sel, wrap, s, n, &my_steps)
                                              : careful_steps<false>(&ps, rA, rB[p], rC, sel, wrap, s, n, &my_steps);
                        x[p] = ps.x;
                        lyap[p] = ps.lyap;
                        valid[p] = ps.valid;
                        redone |= 1u << p;
                        if (dead) {
                            done[p] = true;
                            lam[p] = ps.valid > 0 ? __ddiv_rn(ps.lyap, __dmul_rn((double)ps.valid, LYAP_LN2)) : -5.0;   // :84-85
                            x[p] = 0.25;
                        }
                    }
                }
                if (acc && n == CS && left >= CS + kLeastLeft) cycles(sx, redone, sel, wrap, BS, s + n, left - n);
                s += n;
            }
            continue;
        }
        // generic walk: exit tests after every second selector word, or after a.acc_chunk steps of the accumulation
        static_assert(2 * kStepsPerWord <= kMaxChunk, "an orbit's fall is replayed on the strength of it");
        const unsigned* sel = a.sel + word0;
        const int chunk = acc ? a.acc_chunk : 2 * kStepsPerWord;
        int s = 0, wi = 0, in_word = 0;   // step s is step in_word of word wi
        while (s < nsteps) {
            bool all_done = true;
#pragma unroll
            for (int p = 0; p < P; ++p) all_done = all_done && done[p];
            if (__all_sync(0xFFFFFFFFu, all_done)) break;

            const int n = min(chunk, nsteps - s);
            // Whole periods lie behind this chunk, it has the selectors of the first: read from its words' beginnings (37 letters
            // 1277 x 719 849 -> 832 us).  With three parameters that makes slower code of the whole loop (1783 x 1722 of "ABC"
            // 172 + 1719, nearly all in cycles, 2.57 -> 2.77 ms), and the words go on through the chunks.
            if (!HAS_C && acc && a.acc_period) wi = 0;
            double sx[P], sl[P];
#pragma unroll
            for (int p = 0; p < P; ++p) {
                sx[p] = x[p];
                sl[p] = lyap[p];
            }
#pragma unroll 1
            for (int k = 0; k < n; k += kStepsPerWord) {
                const int m = min(kStepsPerWord, n - k);
                const int after = wi + 1 == wrap ? 0 : wi + 1;
                const unsigned word = HAS_C ? __funnelshift_r(sel[wi], sel[after], 2 * in_word) : sel[wi];
                in_word += m;
                if (!HAS_C || in_word >= kStepsPerWord) {
                    in_word -= kStepsPerWord;
                    wi = after;
                }
                if (acc) fast_chunk<P, true, HAS_C, UNROLL>(x, lyap, rA, rB, rC, word, m, lane_off);
                else fast_chunk<P, false, HAS_C, UNROLL>(x, lyap, rA, rB, rC, word, m, lane_off);
            }
            unsigned redone = 0;
#pragma unroll
            for (int p = 0; p < P; ++p) {
                if (done[p]) continue;
                // an irregular derivative (zero, subnormal, non-finite) has made the sum non-finite through the exponent table
                const bool regular = !careful_only[p] && in_unit_interval(x[p]) && isfinite(lyap[p]);
                if (regular) {
                    if (acc) valid[p] += n;
                    my_steps += (unsigned long long)n;
                } else {
                    PixelState ps{sx[p], sl[p], valid[p]};
                    const bool dead = acc ? careful_steps<true>(&ps, rA, rB[p], rC, sel, wrap, s, n, &my_steps)
                                          : careful_steps<false>(&ps, rA, rB[p], rC, sel, wrap, s, n, &my_steps);
                    x[p] = ps.x;
                    lyap[p] = ps.lyap;
                    valid[p] = ps.valid;
                    redone |= 1u << p;
                    if (dead) {
                        done[p] = true;
                        lam[p] = ps.valid > 0 ? __ddiv_rn(ps.lyap, __dmul_rn((double)ps.valid, LYAP_LN2)) : -5.0;   // :84-85
                        x[p] = 0.25;   // keep the abandoned lane's arithmetic tame
                    }
                }
            }
            const int left = nsteps - s - n;
            if (acc && a.acc_period && left >= kLeastLeft) cycles(sx, redone, sel, wrap, a.acc_period, s + n, left);
            s += n;
        }
    }

#pragma unroll
    for (int p = 0; p < P; ++p) {
        if (!done[p]) lam[p] = valid[p] > 0 ? __ddiv_rn(lyap[p], __dmul_rn((double)valid[p], LYAP_LN2)) : -5.0;
    }

    if (!inside) return;
    const long long at = row * a.width + col;
#pragma unroll
    for (int p = 0; p < P; ++p) {
        if (out64) out64[at + (long long)p * a.width] = lam[p];
        if (out32) out32[at + (long long)p * a.width] = (float)lam[p];
    }
}

// Body shared by the library's generic kernel (KG == 0) and by a specialised instance (KG > 0).
template <int P, int THREADS, bool HAS_C, int UNROLL, int KG, unsigned long long WU_PATS, unsigned long long ACC_PATS>
__device__ __forceinline__ void lambda_exact_body(const LambdaArgs& a, double* __restrict__ out64, float* __restrict__ out32,
                  unsigned long long* __restrict__ steps_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    lyap_logtab_entry* tab_all = reinterpret_cast<lyap_logtab_entry*>(smem_raw);
    // every entry is read once and written to its copies in an order that differs by lane, so that the 8 lanes of a
    // quarter warp write to 8 bank groups
    for (int e = threadIdx.x; e < LYAP_LOG_BINS; e += THREADS) {
        lyap_logtab_entry t = g_lyap_logtab[e];
        t.invc = __hiloint2double(__double2hiint(t.invc) + 0x3FF00000, __double2loint(t.invc));   // see log_fast
#pragma unroll
        for (int c = 0; c < kTabCopies; ++c) tab_all[e * kTabCopies + ((threadIdx.x + c) & (kTabCopies - 1))] = t;
    }
    const unsigned lane_off = (threadIdx.x & (kTabCopies - 1)) * 16u;
    double2* exp_tab = reinterpret_cast<double2*>(smem_raw + kTabSmemBytes);
    for (int e = threadIdx.x; e < kExpEntries; e += THREADS) {
        double2 v;
        if (e == 0) v = make_double2(__longlong_as_double(0xFFF0000000000000LL), 0.0);                       // zero / subnormal derivative
        else if (e >= 2046) v = make_double2(__longlong_as_double(0x7FF8000000000000LL), 0.0);                // inf, NaN, or a set sign bit
        else v = make_double2(__dmul_rn((double)(e + 1), LYAP_LN2HI), __fma_rn((double)(e + 1), LYAP_LN2LO, LYAP_KLO_BIAS));
        exp_tab[e] = v;
    }
    unsigned long long my_steps = 0;
    // Work is dealt out per warp: first a.wide_tiles warp-tiles of 32*P pixels, then the rest of the frame in tiles of 32 pixels
    // (a scheduler's time is its pixels times a constant whatever its warps' shapes: 2200 steps take 103 / 168 / 238 / 312 us
    // with 1 / 2 / 3 / 4 warps of 2 pixels a thread, 58 / 93 / 123 / 158 us with 1 / 2 / 3 / 4 of one).  A tile whose orbits end
    // or come into cycles soon takes a tenth of another's time, so a warp that is done takes the next tile of the launch from
    // a counter in device memory.  Without one (see a.queue) tile t goes to block t % gridDim, and the block's tiles go round
    // its four schedulers (a warp's scheduler is warp % 4) through counters in shared memory.
    __shared__ unsigned next_unit[4];   // the first units are taken as unit == warp
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < 4) next_unit[threadIdx.x] = THREADS / 32 + threadIdx.x;
    __syncthreads();   // the counters, and both tables, which are read across warps from the first logarithm on
    // Positions are the columns of the rows in groups of P, group by group; a wide tile is 32 consecutive positions.  The
    // small tiles go over the positions that are left, for each of the P rows in turn, and then over the rows behind the
    // last whole group.
    const long long rows = a.n_pixels / a.width, positions = rows / P * a.width;
    const long long first = a.wide_tiles * 32, left = positions - first;
    const long long narrow_pixels = a.n_pixels - first * P;
    for (long long t = (long long)warp * gridDim.x + blockIdx.x;;) {
        if (P > 1 && t < a.wide_tiles) {
            const long long q = t * 32 + lane, group = q / a.width;
            exact_tile<P, HAS_C, UNROLL, KG, WU_PATS, ACC_PATS>(a, group * P, (int)(q - group * a.width), true, out64, out32, lane_off,
                                                                my_steps);
        } else {
            const long long m = (t - a.wide_tiles) * 32 + lane;
            if (m - lane >= narrow_pixels) break;
            long long row, col;
            if (m < left * P) {
                const long long p = m / left, q = first + (m - p * left);
                row = q / a.width * P + p;
                col = q % a.width;
            } else {
                const long long k = m - left * P;
                row = rows / P * P + k / a.width;
                col = k % a.width;
            }
            exact_tile<1, HAS_C, UNROLL, KG, WU_PATS, ACC_PATS>(a, row, (int)col, m < narrow_pixels, out64, out32, lane_off, my_steps);
        }
        unsigned unit = 0;
        if (lane == 0) unit = a.queue ? atomicAdd(a.queue, 1u) : atomicAdd(&next_unit[warp & 3], 4u);
        unit = __shfl_sync(0xFFFFFFFFu, unit, 0);
        t = a.queue ? unit + (long long)gridDim.x * (THREADS / 32) : (long long)unit * gridDim.x + blockIdx.x;
    }
    // the last warp to be done leaves the queue as it was found
    if (a.queue && lane == 0 && atomicAdd(a.queue + 1, 1u) == gridDim.x * (THREADS / 32) - 1) {
        a.queue[0] = 0;
        a.queue[1] = 0;
    }

    if (steps_out) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) my_steps += __shfl_down_sync(0xFFFFFFFFu, my_steps, o);
        if ((threadIdx.x & 31) == 0 && my_steps) atomicAdd(steps_out, my_steps);
    }
}


template <int P, int THREADS, bool HAS_C, int UNROLL>
__global__ void __launch_bounds__(THREADS, 1)
k_lambda_exact(const __grid_constant__ LambdaArgs a, double* __restrict__ out64, float* __restrict__ out32,
               unsigned long long* __restrict__ steps_out) {
    lambda_exact_body<P, THREADS, HAS_C, UNROLL, 0, 0ull, 0ull>(a, out64, out32, steps_out);
}

#if defined(LYAP_SPEC_EXACT)
// The specialised instance; LYAP_SPEC_* are given on the run-time compiler's command line.
extern "C" __global__ void __launch_bounds__(LYAP_SPEC_THREADS, 1)
k_lambda_exact_spec(const __grid_constant__ LambdaArgs a, double* __restrict__ out64, float* __restrict__ out32,
                    unsigned long long* __restrict__ steps_out) {
    lambda_exact_body<LYAP_SPEC_P, LYAP_SPEC_THREADS, pats_use_c(LYAP_SPEC_WU_PATS | LYAP_SPEC_ACC_PATS), 2, LYAP_SPEC_KG,
                      LYAP_SPEC_WU_PATS, LYAP_SPEC_ACC_PATS>(a, out64, out32, steps_out);
}
#endif

}  // namespace lyap
