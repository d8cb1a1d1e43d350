// lyap_kernels_fast.cuh -- fast-mode lambda kernels (included by lyap_kernels.cu after lyap_exact_kernel.cuh, and, as
// text, by the run-time specialiser).
//
// Same sequence handling, sentinel and early-exit rules as the exact kernel; a thread owns P pixels.  The arithmetic is
// rearranged for speed and is NOT bit-compatible with the reference:
//   t = r*x;  deriv = fma(-2,t,r) = r(1-2x);  x' = fma(-t,x,t) = r x (1-x)         (4 fused ops/step)
// and instead of one log per step the |deriv| are multiplied together; the product's exponent is moved into an integer at
// least every 32 (fp64) or 20 (fp32) steps, and one log of the remaining mantissa is taken at the end:
// sum log|deriv| = E*ln2 + log(mantissa product).
// A chunk in which the orbit left (0,1) or a derivative was exactly zero is rolled back and redone step by step with the
// reference's rules (skip zero terms, stop at the exit, keep the partial sum), in a product of its own.  An orbit that
// stands where it stood a chunk ago is in a cycle, and the chunks that are left are added up from the product of one turn.
// What a pixel's sum comes to is decided by its own orbit alone, whichever others are in its warp.
#pragma once

namespace lyap {

template <typename T>
struct FastTraits;

template <>
struct FastTraits<double> {
    static constexpr int kRenorm = 32;
    static __device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double abs_(double a) { return fabs(a); }
    // returns biased exponent; rewrites v's exponent to 0 (mantissa in [1,2)); sign assumed +
    static __device__ __forceinline__ int strip(double& v) {
        const unsigned hw = (unsigned)__double2hiint(v);
        v = __hiloint2double((int)((hw & 0x000FFFFFu) | 0x3FF00000u), __double2loint(v));
        return (int)(hw >> 20);
    }
    static constexpr int kBias = 1023;
    static constexpr int kExpMax = 2047;
};

template <>
struct FastTraits<float> {
    // A product that is subnormal or zero when it is stripped sends the chunk to the step-by-step path.  Falling below
    // 2^-126 from [1,2) within 20 steps takes derivatives that average below 2^-6 (x within a percent of 0.5 step after
    // step); only a product that did so and was multiplied back above 2^-126 before the strip would lose low bits
    // unnoticed.  Where the strips fall does not change a regular pixel's bits (moving the exponent out is exact).
    static constexpr int kRenorm = 20;
    static __device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float abs_(float a) { return fabsf(a); }
    // the sign, which the packed steps leave in, goes too
    static __device__ __forceinline__ int strip(float& v) {
        const unsigned u = __float_as_uint(v);
        v = __uint_as_float((u & 0x007FFFFFu) | 0x3F800000u);
        return (int)((u >> 23) & 0xFFu);
    }
    static constexpr int kBias = 127;
    static constexpr int kExpMax = 255;
};

// The three fast kernels: which type the orbit and the product run in, and whether the orbit and the derivative use the
// reference's own operations (then x and every derivative have the exact kernel's bits and only the accumulation --
// a running product instead of a sum of logarithms -- differs) or the fused ones.
// packed: two pixels a step in the two-wide fp32 instructions; the orbit is then held as -x (see packed_step).
struct FusedF64 { using real = double; static constexpr bool same_orbit = false, packed = false; };
struct FusedF32 { using real = float; static constexpr bool same_orbit = false, packed = true; };
struct OrbitF64 { using real = double; static constexpr bool same_orbit = true, packed = false; };

// One step of one pixel: the derivative at x (times into prod when ACC), then the update.
//   fused:      t = r*x;  deriv = fma(-2,t,r) = r(1-2x);  x' = fma(-t,x,t) = r x (1-x)            4 instructions
//   same orbit: |fma(-2,x,1)| into the product (deriv = r*|1-2x|, :69; the r's are added as n*log r at the end);
//               x' = (r*x)*(1-x) (:76)                                                             5 instructions
template <typename FL, bool ACC>
__device__ __forceinline__ void fast_step_one(typename FL::real& x, typename FL::real& prod, typename FL::real r) {
    using T = typename FL::real;
    using F = FastTraits<T>;
    if (FL::same_orbit) {
        // |r*(1-2x)| = r*|1-2x| for r > 0: only |1-2x| (exact: 2x and 1-2x round nowhere near 0.5) goes into the product;
        // the factors r are accounted for per pixel at the end, from how many steps used which parameter
        if (ACC) prod = F::mul(prod, F::abs_(F::fma_((T)-2, x, (T)1)));
        x = F::mul(F::mul(r, x), F::sub((T)1, x));
    } else {
        const T t = F::mul(r, x);
        if (ACC) prod = F::mul(prod, F::abs_(F::fma_((T)-2, t, r)));
        x = F::fma_(-t, x, t);
    }
}

// One fused step of two pixels, y = -x:  nt = r*y = -t;  deriv = fma(2,nt,r);  y' = fma(nt,y,nt).  The two-wide instructions
// take no sign changes, and with -x none is needed; the derivative's sign stays in the product until it is stripped.  All
// values are the unpacked step's or their exact negatives, so the results have the same bits.
// One-wide, the step's four instructions read two or three registers each, and two of them in one bank cost a cycle more;
// a pair of registers spans the banks.  4096 x 2048 pixels of "AABAB" 200 + 2000: 3.05 ms one-wide, 2.54 two-wide.
template <bool ACC>
__device__ __forceinline__ void packed_step(float& y0, float& y1, float& prod0, float& prod1, float r0, float r1) {
    unsigned long long y, r, nt;
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(y0), "f"(y1));
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(r0), "f"(r1));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(nt) : "l"(r), "l"(y));
    if (ACC) {
        unsigned long long prod, deriv, two;
        asm("mov.b64 %0, {%1, %2};" : "=l"(prod) : "f"(prod0), "f"(prod1));
        asm("mov.b64 %0, {%1, %1};" : "=l"(two) : "f"(2.0f));
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(deriv) : "l"(nt), "l"(two), "l"(r));
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(prod) : "l"(prod), "l"(deriv));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(prod0), "=f"(prod1) : "l"(prod));
    }
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(y) : "l"(nt), "l"(y), "l"(nt));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(y0), "=f"(y1) : "l"(y));
}

template <typename T>
struct FastPixel {
    T x;
    double extra;   // logarithms of what the careful path multiplied up, and of falls
    int esum;       // its powers of two
    int valid;
};

// how many of the first n (<= 16) steps of a selector word use each of the parameters
__device__ __forceinline__ void count_word_codes(unsigned word, int n, int& c0, int& c1, int& c2) {
    const unsigned live = n >= 16 ? 0x55555555u : ((1u << (2 * n)) - 1u) & 0x55555555u;
    const unsigned lo = word & 0x55555555u, hi = (word >> 1) & 0x55555555u;
    c0 = __popc(~lo & ~hi & live);
    c1 = __popc(lo & ~hi & live);
    c2 = __popc(hi & ~lo & live);
}

// Below kFallen, 1 - 2x and 1 - x round to 1 and r - 2rx to r: a step is x <- r*x and its derivative the parameter itself.
// A parameter of at most kFallenParam takes such an x to less than 1/2, so that zero is the only way out of (0,1); the
// comparison is false for NaN, whose derivative is no term of the sum, and for infinity.
constexpr double kFallen = 0x1p-60, kFallenParam = 0x1p59;

// An orbit that runs down to zero (rA*rB < 1: a whole region of a frame over [0,4]^2 does, each orbit at another step) spends
// most of its steps below kFallen, where the logarithm of a step's derivative is one of at most three taken beforehand: the
// same sums, without a table look-up and a polynomial a step.  2048 x 1024 over [0.01,4]^2, "ABAAB" 120 + 1200: fused
// fp64 5.11 -> 2.07 ms, on the exact orbit 3.74 -> 1.82 (over [2.5,4]^2, without exits, 0.67 and 0.88, as before).
template <typename T, bool ACC>
struct Fall {
    T rA, rB, rC;
    int nA = 0, nB = 0, nC = 0;   // steps by the parameter they use

    static __device__ __forceinline__ bool applies(T x, T rA, T rB) {   // fp32 orbits are at zero too soon for it to pay
        return sizeof(T) == 8 && x < (T)kFallen && rA <= (T)kFallenParam && rB <= (T)kFallenParam;
    }
    __device__ __forceinline__ Fall(T a, T b, T c) : rA(a), rB(b), rC(c) {}
    // the first steps of n <= 16 of selector word `word` that are of this kind; their number.  A whole word, far enough down and
    // with small parameters, is walked without looking at it in between: zero is where it stays, and is looked for at the end.
    __device__ __forceinline__ int walk(T& x, unsigned word, int n) {
        int j = 0;
        if (n == kStepsPerWord && (word & 0xAAAAAAAAu) == 0 && x < (T)0x1p-92 && rA <= (T)4 && rB <= (T)4) {
            T y = x;
#pragma unroll
            for (int k = 0; k < kStepsPerWord; ++k) y = FastTraits<T>::mul((word >> (2 * k)) & 1u ? rB : rA, y);
            if (y > (T)0) {
                x = y;
                j = kStepsPerWord;
            }
        }
        for (unsigned w = word; j < n && x > (T)0 && x < (T)kFallen; ++j, w >>= 2) {
            const unsigned code = w & 3u;
            if (code >= 2u && !(rC > (T)0 && rC <= (T)kFallenParam)) break;
            x = FastTraits<T>::mul(code == 0 ? rA : (code == 1 ? rB : rC), x);
        }
        if (ACC) {
            int a, b, c;
            count_word_codes(word, j, a, b, c);
            nA += a;
            nB += b;
            nC += c;
        }
        return j;
    }
    // the logarithms of the parameters, as often as they were used
    __device__ __forceinline__ double sum() const {
        double total = 0.0;
#pragma unroll 1
        for (int k = 0; k < 3; ++k) {   // the code of one logarithm
            const int uses = k == 0 ? nA : (k == 1 ? nB : nC);
            if (uses) total = __fma_rn((double)uses, lyap_log_tab((double)(k == 0 ? rA : (k == 1 ? rB : rC)), g_lyap_logtab, 1), total);
        }
        return total;
    }
};

// A product of an orbit's derivatives as (hi + lo) * 2^e.  fp32 derivatives are multiplied in doubles and need no lo.
template <typename FL>
struct LongProduct {
    using T = typename FL::real;
    using F = FastTraits<T>;
    double hi = 1.0, lo = 0.0;
    int e = 0;
    __device__ __forceinline__ void multiply(double m) {
        const double p = __dmul_rn(hi, m);
        if (sizeof(T) == 8) lo = __fma_rn(lo, m, __fma_rn(hi, m, -p));
        hi = p;
    }
    // one step of the orbit, its derivative (same orbit: the factor |1 - 2x|) into the product
    __device__ __forceinline__ void step(T& x, T r) {
        const T t = F::mul(r, x);
        const double m = (double)F::abs_(FL::same_orbit ? F::fma_((T)-2, x, (T)1) : F::fma_((T)-2, t, r));
        x = FL::same_orbit ? F::mul(t, F::sub((T)1, x)) : F::fma_(-t, x, t);
        multiply(m);
    }
    // after at most kRun factors: a derivative inside a cycle is no smaller than 2^-93 (fp64: a parameter of 2^-40 times 2^-53)
    static constexpr int kRun = 8;
    __device__ __forceinline__ void strip() {
        const int field = (int)((unsigned)__double2hiint(hi) >> 20);
        if (sizeof(T) == 8) lo = __dmul_rn(lo, __hiloint2double((2046 - field) << 20, 0));
        hi = __hiloint2double((__double2hiint(hi) & 0x000FFFFF) | 0x3FF00000, __double2loint(hi));
        e += field - 1023;
    }
    template <int KG, unsigned long long PATS, int J = 0>
    __device__ __forceinline__ void unit(T& x, T rA, T rB, T rC) {
        if constexpr (J < fast_unit(2 * KG)) {
            constexpr unsigned code = (unsigned)(PATS >> (2 * (J % (2 * KG)))) & 3u;
            step(x, code == 0 ? rA : (code == 1 ? rB : rC));
            if (J % kRun == kRun - 1 || J == fast_unit(2 * KG) - 1) strip();
            unit<KG, PATS, J + 1>(x, rA, rB, rC);
        }
    }
    // `times` times its logarithm but for the 2^e, which is had in two doubles: `times` is many and would multiply the
    // rounding of one.  The mantissa is first brought to where the logarithm is smallest.
    __device__ __forceinline__ double log_times(double times) {
        if (hi > 1.41) {
            hi = __dmul_rn(hi, 0.5);
            lo = __dmul_rn(lo, 0.5);
            ++e;
        }
        double h, s;
        lyap_log_core((unsigned)__double2hiint(hi), (unsigned)__double2loint(hi), 0, g_lyap_logtab, 1, &h, &s);
        if (sizeof(T) == 8) s = __fma_rn(lo, (double)__frcp_rn((float)hi), s);
        return __fma_rn(times, h, __dmul_rn(times, s));
    }
};

// The reference's rules, one step at a time, for n <= 16 steps of selector word `word`; true when the orbit left (0,1).  Ordinary
// derivatives are multiplied up in a double's range, which is nearer to their logarithms' sum than adding those one by one, and
// quicker (800 x 800 over [0.01,3.99]^2, "AB" 100 + 1000, fp32: 395 -> 239 us); others give a logarithm each, infinite ones
// with what follows from it.
template <typename FL, bool ACC>
__device__ __forceinline__ bool fast_careful_body(FastPixel<typename FL::real>* ps, typename FL::real rA, typename FL::real rB,
                                                  typename FL::real rC, unsigned word, int n, LongProduct<FL>& product,
                                                  unsigned* steps) {
    using T = typename FL::real;
    using F = FastTraits<T>;
    T x = ps->x;
    int valid = ps->valid;
    bool dead = false;
    int j = 0;
    for (; j < n && !dead; ++j, word >>= 2) {
        const unsigned sel = word & 3u;
        const T r = sel == 0 ? rA : (sel == 1 ? rB : rC);
        const T t = F::mul(r, x);
        if (ACC) {
            const double d = (double)(FL::same_orbit ? F::mul(r, F::abs_(F::fma_((T)-2, x, (T)1))) : F::abs_(F::fma_((T)-2, t, r)));
            if (d > 0x1p-100 && d < 0x1p100) {
                product.multiply(d);
                ++valid;
            } else if (d > 0.0) {
                ps->extra = __dadd_rn(ps->extra, lyap_log_tab(d, g_lyap_logtab, 1));
                ++valid;
            }
            if (j % LongProduct<FL>::kRun == LongProduct<FL>::kRun - 1) product.strip();
        }
        x = FL::same_orbit ? F::mul(t, F::sub((T)1, x)) : F::fma_(-t, x, t);
        dead = !(x > (T)0 && x < (T)1);
    }
    product.strip();
    *steps += j;
    ps->x = x;
    ps->valid = valid;
    return dead;
}

// The steps of a falling orbit from `first` on, of a region whose selector words start at `sel`, up to `end`, to the orbit's own
// end or to a step that is not of this kind; returns the first step not taken.
template <typename FL, bool ACC>
__device__ __forceinline__ int fast_fall(FastPixel<typename FL::real>* ps, typename FL::real rA, typename FL::real rB,
                                         typename FL::real rC, const unsigned* sel, int wrap, int first, int end,
                                         unsigned* steps) {
    using T = typename FL::real;
    Fall<T, ACC> fall(rA, rB, rC);
    T x = ps->x;
    int j = first;
    for (int m = 0, k = 0; k == m && j < end; j += k) {
        m = min(kStepsPerWord, end - j);
        k = fall.walk(x, selectors_from(sel, wrap, j), m);
    }
    if (ACC) {
        ps->valid += j - first;
        ps->extra = __dadd_rn(ps->extra, fall.sum());
    }
    *steps += j - first;
    ps->x = x;
    return j;
}

template <typename FL, int P, bool ACC>
__device__ __forceinline__ void fast_mode_steps(typename FL::real (&x)[P], typename FL::real (&prod)[P],
                                                const typename FL::real (&r)[P]) {
    if constexpr (FL::packed) {
        static_assert(P % 2 == 0, "pixels go in pairs");
#pragma unroll
        for (int p = 0; p < P; p += 2) packed_step<ACC>(x[p], x[p + 1], prod[p], prod[p + 1], r[p], r[p + 1]);
    } else {
#pragma unroll
        for (int p = 0; p < P; ++p) fast_step_one<FL, ACC>(x[p], prod[p], r[p]);
    }
}

// fast_careful_body for steps [first, first + n) of a region whose selector words start at `sel`.  It calls no other function: a
// second level of calls shows in the registers that the kernels' own loops have left.
template <typename FL, bool ACC>
__device__ __noinline__ bool fast_careful_steps(FastPixel<typename FL::real>* ps, typename FL::real rA, typename FL::real rB,
                                                typename FL::real rC, const unsigned* sel, int wrap, int first, int n,
                                                unsigned* steps) {
    using T = typename FL::real;
    LongProduct<FL> product;
    bool dead = false;
    int j = first;
    const int end = first + n;
    while (j < end && !dead) {
        if (Fall<T, ACC>::applies(ps->x, rA, rB)) {
            j = fast_fall<FL, ACC>(ps, rA, rB, rC, sel, wrap, j, end, steps);
            dead = !(ps->x > (T)0);
            if (dead || j == end) break;
        }
        const int m = min(kStepsPerWord, end - j);
        dead = fast_careful_body<FL, ACC>(ps, rA, rB, rC, selectors_from(sel, wrap, j), m, product, steps);
        j += m;
    }
    if (ACC) {
        ps->extra = __dadd_rn(ps->extra, product.log_times(1.0));
        ps->esum += product.e;
    }
    return dead;
}

// Moves the exponent of every pixel's running product into its integer sum and notes the smallest exponent field seen.
// The sum takes the BIASED field; the caller subtracts the bias once per strip when it accepts the chunk.  Only the
// low end needs watching: while x stays inside (0,1) every derivative is below r in magnitude, so a product of at most
// kRenorm of them cannot overflow, and an x that left (0,1) is found by the test on x itself.
template <typename T, int P>
__device__ __forceinline__ void strip_products(T (&prod)[P], int (&esum)[P], int (&emin)[P]) {
    using F = FastTraits<T>;
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const int e = F::strip(prod[p]);
        emin[p] = min(emin[p], e);
        esum[p] += e;
    }
}

// strips fast_fixed_groups makes in NG groups
template <typename T>
__host__ __device__ constexpr int strips_in_groups(int ng) {
    int n = 0;
    for (int gi = 0; gi < ng; ++gi)
        if ((2 * (gi + 1)) % FastTraits<T>::kRenorm == 0 || gi == ng - 1) ++n;
    return n;
}

// Run-time specialisation (see lyap_jit.cu): NG two-step groups whose patterns are compile-time constants
// (PATS: 4 bits per group, repeating every KG groups), as one straight-line block; the products are stripped
// every kRenorm steps and after the last group.
template <typename FL, int P, bool ACC, int KG, unsigned long long PATS, int NG, int GI = 0>
__device__ __forceinline__ void fast_fixed_groups(typename FL::real (&x)[P], typename FL::real (&prod)[P], int (&esum)[P],
                                                  int (&emin)[P], const typename FL::real (&rA)[P],
                                                  const typename FL::real (&rB)[P], const typename FL::real (&rC)[P]) {
    using T = typename FL::real;
    using F = FastTraits<T>;
    if constexpr (GI < NG) {
        constexpr unsigned pat = (unsigned)((PATS >> (4 * (GI % KG))) & 15ull);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            constexpr unsigned code0 = pat & 3u, code1 = (pat >> 2) & 3u;
            const unsigned code = j == 0 ? code0 : code1;
            fast_mode_steps<FL, P, ACC>(x, prod, code == 0 ? rA : (code == 1 ? rB : rC));
        }
        if (ACC && ((2 * (GI + 1)) % F::kRenorm == 0 || GI == NG - 1)) strip_products<T, P>(prod, esum, emin);
        fast_fixed_groups<FL, P, ACC, KG, PATS, NG, GI + 1>(x, prod, esum, emin, rA, rB, rC);
    }
}

template <typename T>
__device__ __forceinline__ bool ordinary_param_t(T r);
template <>
__device__ __forceinline__ bool ordinary_param_t<double>(double r) { return r > 0x1p-40 && r < 0x1p40; }
template <>
__device__ __forceinline__ bool ordinary_param_t<float>(float r) { return r > 0x1p-20f && r < 0x1p5f; }

// how many of the `steps` 2-bit codes in `pats` (step j at bits 2j, 2j+1) equal `code`
__host__ __device__ constexpr int count_code(unsigned long long pats, int steps, unsigned code) {
    int n = 0;
    for (int j = 0; j < steps; ++j) n += ((pats >> (2 * j)) & 3ull) == code ? 1 : 0;
    return n;
}

// n steps of selector word `word`: of A's and B's four at a time, one of 16 straight-line bodies picked by a warp-uniform
// branch; single ones, and words with a third parameter, step by step.  1200 x 900 of "ABBAABA" 100 + 1000 over [2,4]^2 in fp32:
// 486 us step by step, 406 so.
template <typename FL, int P, bool ACC, unsigned PAT>
__device__ __forceinline__ void fast_four(typename FL::real (&x)[P], typename FL::real (&prod)[P], const typename FL::real (&rA)[P],
                                          const typename FL::real (&rB)[P]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) fast_mode_steps<FL, P, ACC>(x, prod, (PAT >> j) & 1u ? rB : rA);
}
template <typename FL, int P, bool ACC>
__device__ __forceinline__ void fast_word(typename FL::real (&x)[P], typename FL::real (&prod)[P], const typename FL::real (&rA)[P],
                                          const typename FL::real (&rB)[P], const typename FL::real (&rC)[P], unsigned word, int n) {
    if ((word & 0xAAAAAAAAu) == 0) {
        unsigned pat = compress_even_bits(word);
#pragma unroll 1
        for (; n >= 4; n -= 4, pat >>= 4) {
            switch (pat & 15u) {
#define LYAP_FOUR(N) case N: fast_four<FL, P, ACC, N>(x, prod, rA, rB); break;
                LYAP_FOUR(0) LYAP_FOUR(1) LYAP_FOUR(2) LYAP_FOUR(3) LYAP_FOUR(4) LYAP_FOUR(5) LYAP_FOUR(6) LYAP_FOUR(7)
                LYAP_FOUR(8) LYAP_FOUR(9) LYAP_FOUR(10) LYAP_FOUR(11) LYAP_FOUR(12) LYAP_FOUR(13) LYAP_FOUR(14)
                default: fast_four<FL, P, ACC, 15>(x, prod, rA, rB);
#undef LYAP_FOUR
            }
        }
        word = spread_bits(pat & 15u);
    }
#pragma unroll 1
    for (int j = 0; j < n; ++j, word >>= 2) {
        const unsigned code = word & 3u;
        if (code == 0) fast_mode_steps<FL, P, ACC>(x, prod, rA);
        else if (code == 1) fast_mode_steps<FL, P, ACC>(x, prod, rB);
        else fast_mode_steps<FL, P, ACC>(x, prod, rC);
    }
}

// Whole chunks that have to be left behind the one in which an orbit is found in a cycle.  Warps in which other orbits are not walk
// on and walk a turn at the end besides: 276 x 283 of "AB" 23 + 238 over [3.9,4]^2 in fp32 takes 31.1 us without such a limit (and
// with one), 20.9 with two or more; 3889 x 4085 of "ABBBBBBABA" 71 + 719 over [2.5,4]^2 in fp64 4.19 ms with two, 4.50 with four.
constexpr int kLeastChunks = 3;

// q times the sum of the logarithms of the derivatives (same orbit: of the factors |1 - 2x|) over n steps, whole periods, of an
// orbit that stands at x again after them, none of them zero: one turn of its cycle, in units of whole periods, is walked.  The
// orbit stands behind a whole chunk, at a period's start, and the generic kernel takes the selectors from the beginning of the
// region's words (`sel`): behind the last chunk there may be fewer than a turn's.  The sum is *exponent * log 2 + the result.
template <typename FL, int KG, unsigned long long PATS>
__device__ __noinline__ double fast_cycle(typename FL::real x, typename FL::real rA, typename FL::real rB, typename FL::real rC,
                                          const unsigned* sel, int wrap, int unit, int n, int q, int* exponent) {
    using T = typename FL::real;
    const T x0 = x;
    LongProduct<FL> product;
    int len = 0;
    if constexpr (KG > 0) {
        do {
            product.template unit<KG, PATS>(x, rA, rB, rC);
            len += fast_unit(2 * KG);
        } while (x != x0 && len < n);
    } else {
        const unsigned head = sel[0];
        do {
            for (int k = 0; k < unit; k += kStepsPerWord) {
                unsigned word = k == 0 ? head : sel[k / kStepsPerWord % wrap];
                const int m = min(kStepsPerWord, unit - k);
                for (int j = 0; j < m; ++j, word >>= 2) {
                    const unsigned code = word & 3u;
                    product.step(x, code == 0 ? rA : (code == 1 ? rB : rC));
                    if (j == LongProduct<FL>::kRun - 1) product.strip();
                }
                product.strip();
            }
            len += unit;
        } while (x != x0 && len < n);
    }
    const int times = q * (n / len);
    const double sum = product.log_times((double)times);
    *exponent = times * product.e;
    return sum;
}

// Body shared by the precompiled kernel (KG == 0) and a run-time specialised instance (KG > 0): one tile a warp.
template <typename FL, int P, int THREADS, int KG, unsigned long long WU_PATS, unsigned long long ACC_PATS>
__device__ __forceinline__ void lambda_fast_body(const LambdaArgs& a, double* __restrict__ out64, float* __restrict__ out32,
                                                 unsigned long long* __restrict__ steps_out) {
    using T = typename FL::real;
    using F = FastTraits<T>;
    constexpr T kSign = FL::packed ? (T)-1 : (T)1;   // x[] holds kSign * x
    unsigned my_steps = 0, cycle_steps = 0;   // of a thread's pixels: no more than P * 2^24, and a warp's 2^30
    // A tile is 32 neighbouring positions.  In a frame of rows enough a position is a column of a group of P rows, whose
    // pixels lie below one another: tiles as high as they are compact come into cycles or leave (0,1) as a whole most often.
    // Where the last group would be mostly empty, the frame is one long row cut into P pieces, a pixel of each a position.
    const long long rows = a.n_pixels / a.width, groups = (rows + P - 1) / P;
    const bool grouped = 32 * (groups * P - rows) <= rows;
    const long long positions = grouped ? groups * a.width : (a.n_pixels + P - 1) / P;
    const long long at = (blockIdx.x * (long long)(THREADS / 32) + (threadIdx.x >> 5)) * 32 + (threadIdx.x & 31);
    if (at - (threadIdx.x & 31) >= positions) return;
    T x[P], prod[P], rA[P], rB[P], rC[P];
    double extra[P];
    int valid[P], esum[P];   // 32 bits are enough: the host admits at most 2^24 steps per pixel in the fast modes
    int nuse[P][3];          // same-orbit flavour: accumulated steps of accepted chunks by the parameter they used (A, B, C)
    // a pixel's state: on its way, on its way but step by step (an odd parameter), ended, or, from 0 on, the accumulated steps
    // after which its orbit stood where it had stood a chunk before
    constexpr int kWalks = -1, kCareful = -2, kDone = -3;
    int state[P];
    // a thread's own places for its sums then: registers for them would be taken from the loop (4096^2 of "AABAB" 200 + 2000
    // in fp32 3.27 -> 3.20 ms)
    __shared__ T kept_prod[P][THREADS];
    __shared__ int kept_esum[P][THREADS];
    // pixel p's place in the launch, or -1 where there is none
    auto place = [&](int p) -> long long {
        const long long group = at / a.width;
        if (at >= positions) return -1;
        if (grouped) return group * P + p < rows ? at + (group * (P - 1) + p) * a.width : -1;
        const long long i = at + p * positions;
        return i < a.n_pixels ? i : -1;
    };
    // a pixel is written when its orbit has ended, one that has none is a sentinel
    auto store = [&](int p, double lam) {
        const long long i = place(p);
        if (out64) out64[i] = lam;
        if (out32) out32[i] = (float)lam;
    };
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const long long i = place(p), row = i / a.width;
        const double rb = __dadd_rn(a.min_y, __dmul_rn(a.dy, (double)(int)(a.row_begin + row)));
        const double ra = __dadd_rn(a.min_x, __dmul_rn(a.dx, (double)(int)(i - row * a.width)));
        rA[p] = (T)ra;
        rB[p] = (T)rb;
        rC[p] = (T)a.c_value;
        x[p] = kSign * (T)0.5;
        prod[p] = (T)1;
        extra[p] = 0.0;
        valid[p] = 0;
        esum[p] = 0;
        if constexpr (FL::same_orbit) nuse[p][0] = nuse[p][1] = nuse[p][2] = 0;
        state[p] = ordinary_param_t<T>(rA[p]) && ordinary_param_t<T>(rB[p]) && a.fast_ok_c ? kWalks : kCareful;
        if (i < 0 || ra <= 0.0 || rb <= 0.0) state[p] = kDone;
        if (i >= 0 && state[p] == kDone) store(p, -5.0);
    }

    // lambda from the partial sums: esum*ln2 + log(mantissa product) + logarithms of falls, redone chunks and turns of a cycle
    // (+ n_A log r_A + n_B log r_B + n_C log r_C where the product left the parameters out)
    auto finish = [&](int p) -> double {
        double lsum = __fma_rn((double)esum[p], LYAP_LN2, __dadd_rn(lyap_log_tab((double)prod[p], g_lyap_logtab, 1), extra[p]));
        if constexpr (FL::same_orbit) {
            double rsum = 0.0;
            if (nuse[p][0] > 0) rsum = __fma_rn((double)nuse[p][0], lyap_log_tab((double)rA[p], g_lyap_logtab, 1), rsum);
            if (nuse[p][1] > 0) rsum = __fma_rn((double)nuse[p][1], lyap_log_tab((double)rB[p], g_lyap_logtab, 1), rsum);
            if (nuse[p][2] > 0) rsum = __fma_rn((double)nuse[p][2], lyap_log_tab((double)rC[p], g_lyap_logtab, 1), rsum);
            lsum = __dadd_rn(lsum, rsum);
        }
        return valid[p] > 0 ? __ddiv_rn(lsum, __dmul_rn((double)valid[p], LYAP_LN2)) : -5.0;
    };

    for (int region = 0; region < 2; ++region) {
        const bool acc = region == 1;
        const int nsteps = acc ? a.iterations : a.warmup;
        const int word0 = acc ? a.acc_word0 : 0;
        const int wrap = acc ? a.acc_wrap : a.wu_wrap;
        const unsigned* sel = a.sel + word0;
        // an instance's chunk: REP straight-line blocks of CB whole periods
        constexpr int BS = KG > 0 ? 2 * KG : 1, CB = fast_block_periods(BS), REP = fast_chunk_blocks(BS);
        const int chunk = KG > 0 ? CB * BS * REP : a.acc_chunk, unit = KG > 0 ? fast_unit(BS) : a.acc_period;
        const int whole = acc && unit > 0 ? nsteps / chunk * chunk : 0;   // the steps in chunks that are a multiple of the period
        int s = 0;
        while (s < nsteps) {
            bool all_done = true;
#pragma unroll
            for (int p = 0; p < P; ++p) all_done = all_done && state[p] == kDone;
            if (__all_sync(0xFFFFFFFFu, all_done)) break;
            const int left = nsteps - s;
            int n = min(left, chunk);
            T sx[P], sp[P];
            int se[P], emin[P];
            int nstrip = 0;   // strips made in this chunk (the same for every pixel): their bias leaves the sums below
            int cuse[3] = {0, 0, 0};   // accumulated steps of this chunk by parameter (same for every pixel)
#pragma unroll
            for (int p = 0; p < P; ++p) {
                sx[p] = x[p];
                sp[p] = prod[p];
                se[p] = esum[p];
                emin[p] = F::kExpMax;
            }
            if constexpr (KG > 0) {
                constexpr int kPer0 = count_code(ACC_PATS, BS, 0), kPer1 = count_code(ACC_PATS, BS, 1), kPer2 = count_code(ACC_PATS, BS, 2);
                if (left >= CB * BS) {          // whole blocks
                    const int blocks = left >= chunk ? REP : 1;
                    n = blocks * CB * BS;
#pragma unroll 1
                    for (int rep = 0; rep < blocks; ++rep) {
                        if (acc) fast_fixed_groups<FL, P, true, KG, ACC_PATS, CB * KG>(x, prod, esum, emin, rA, rB, rC);
                        else fast_fixed_groups<FL, P, false, KG, WU_PATS, CB * KG>(x, prod, esum, emin, rA, rB, rC);
                    }
                    nstrip = blocks * strips_in_groups<T>(CB * KG);
                    if constexpr (FL::same_orbit) cuse[0] = blocks * CB * kPer0, cuse[1] = blocks * CB * kPer1, cuse[2] = blocks * CB * kPer2;
                } else if (left >= BS) {        // the last few whole periods
                    n = left / BS * BS;
#pragma unroll 1
                    for (int b = 0; b < n / BS; ++b) {
                        if (acc) fast_fixed_groups<FL, P, true, KG, ACC_PATS, KG>(x, prod, esum, emin, rA, rB, rC);
                        else fast_fixed_groups<FL, P, false, KG, WU_PATS, KG>(x, prod, esum, emin, rA, rB, rC);
                    }
                    nstrip = (n / BS) * strips_in_groups<T>(KG);
                    if constexpr (FL::same_orbit) cuse[0] = (n / BS) * kPer0, cuse[1] = (n / BS) * kPer1, cuse[2] = (n / BS) * kPer2;
                }
            }
            if (KG == 0 || left < BS) {         // a selector word, or the part of one that the chunk holds, at a time
                n = KG == 0 ? n : left;
                int wi = (s / kStepsPerWord) % wrap;
                const int in_word = s & (kStepsPerWord - 1);
#pragma unroll 1
                for (int k = 0; k < n; k += kStepsPerWord) {
                    const int m = min(kStepsPerWord, n - k), after = wi + 1 == wrap ? 0 : wi + 1;
                    const unsigned word = __funnelshift_r(sel[wi], sel[after], 2 * in_word);
                    wi = after;
                    if (acc) {
                        if constexpr (FL::same_orbit) {
                            int c0, c1, c2;
                            count_word_codes(word, m, c0, c1, c2);
                            cuse[0] += c0, cuse[1] += c1, cuse[2] += c2;
                        }
                        fast_word<FL, P, true>(x, prod, rA, rB, rC, word, m);
                        static_assert(kStepsPerWord <= F::kRenorm, "a word's derivatives fit the product");
                        strip_products<T, P>(prod, esum, emin);
                        ++nstrip;
                    } else {
                        fast_word<FL, P, false>(x, prod, rA, rB, rC, word, m);
                    }
                }
            }
            bool all_cycle = true;
#pragma unroll
            for (int p = 0; p < P; ++p) {
                if (state[p] == kDone) continue;
                if (state[p] >= 0) continue;   // its sums are kept (and run on unused), x comes back by itself
                // a zero derivative (or a product that underflowed) shows as exponent field 0
                const bool regular = state[p] == kWalks && (kSign * x[p] > (T)0 && kSign * x[p] < (T)1) && (!acc || emin[p] != 0);
                if (regular) {
                    if (acc) {
                        valid[p] += n;
                        esum[p] -= F::kBias * nstrip;
                        if constexpr (FL::same_orbit) {
                            nuse[p][0] += cuse[0];
                            nuse[p][1] += cuse[1];
                            nuse[p][2] += cuse[2];
                        }
                        if (s < whole - kLeastChunks * chunk && x[p] == sx[p]) {
                            state[p] = s + n;
                            kept_prod[p][threadIdx.x] = prod[p];
                            kept_esum[p][threadIdx.x] = esum[p];
                        }
                    }
                    my_steps += n;
                } else {
                    prod[p] = sp[p];
                    FastPixel<T> ps{kSign * sx[p], extra[p], se[p], valid[p]};
                    const bool dead = acc ? fast_careful_steps<FL, true>(&ps, rA[p], rB[p], rC[p], sel, wrap, s, n, &my_steps)
                                          : fast_careful_steps<FL, false>(&ps, rA[p], rB[p], rC[p], sel, wrap, s, n, &my_steps);
                    x[p] = kSign * ps.x;
                    extra[p] = ps.extra;
                    esum[p] = ps.esum;
                    valid[p] = ps.valid;
                    if (dead) {
                        // the result stands now: the abandoned lane keeps running on garbage
                        state[p] = kDone;
                        store(p, finish(p));
                        x[p] = kSign * (T)0.25;
                    }
                }
                all_cycle = all_cycle && (state[p] >= 0 || state[p] == kDone);
            }
            s += n;
            // An orbit that has come back to the value it had a chunk before (as it will from then on) keeps its sums as they
            // are there, and the whole chunks that are left are added up from one turn of its cycle: a pixel's bits are its own,
            // whichever others are in its warp, which walks on until all its orbits have, or to the last whole chunk's end.
            // Cycles walked in full / this: 4096^2 of "AABAB" 200 + 2000 fp32 4.76 / 3.20 ms, fp64 8.37 / 5.59, on the exact orbit
            // 10.3 / 6.92; 2731 x 1537 of "ABB" 150 + 1500 over [2,4]^2, fp64: 1.61 / 0.90.
            if (s > whole || (s < whole && !__all_sync(0xFFFFFFFFu, all_cycle))) continue;
#pragma unroll
            for (int p = 0; p < P; ++p) {
                if (state[p] < 0) continue;
                const int q = (whole - state[p]) / chunk;
                int exponent;
                extra[p] = __dadd_rn(extra[p], fast_cycle<FL, KG, ACC_PATS>(kSign * x[p], rA[p], rB[p], rC[p], sel, wrap, unit, chunk, q,
                                                                             &exponent));
                prod[p] = kept_prod[p][threadIdx.x];
                esum[p] = kept_esum[p][threadIdx.x] + exponent;
                valid[p] += q * chunk;
                if constexpr (FL::same_orbit) {
                    nuse[p][0] += q * cuse[0];
                    nuse[p][1] += q * cuse[1];
                    nuse[p][2] += q * cuse[2];
                }
                my_steps += q * chunk;
                cycle_steps += whole - s;
                state[p] = kWalks;
            }
            s = whole;
        }
    }

#pragma unroll
    for (int p = 0; p < P; ++p) {
        if (state[p] != kDone) store(p, finish(p));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        my_steps += __shfl_down_sync(0xFFFFFFFFu, my_steps, o);
        cycle_steps += __shfl_down_sync(0xFFFFFFFFu, cycle_steps, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (steps_out && my_steps) atomicAdd(steps_out, (unsigned long long)my_steps);
        if (a.cycle_steps && cycle_steps) atomicAdd(a.cycle_steps, (unsigned long long)cycle_steps);
    }
}

constexpr int kFastThreads = 128;

template <typename FL, int P, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS)
k_lambda_fast(const __grid_constant__ LambdaArgs a, double* __restrict__ out64, float* __restrict__ out32,
              unsigned long long* __restrict__ steps_out) {
    lambda_fast_body<FL, P, THREADS, 0, 0ull, 0ull>(a, out64, out32, steps_out);
}

#if defined(LYAP_SPEC_FAST)
// The specialised instance; LYAP_SPEC_* are given on the run-time compiler's command line.
// 24 warps an SM in fp32, 20 in fp64: 4096^2 of "AABAB" 200 + 2000 in fp32 with 32 / 24 / 20 warps 3.39 / 3.39 / 3.51 ms (and
// 800 x 800 over [0.01,3.99]^2 422 / 396 / 399 us), in fp64 with 24 / 20 / 16 warps 5.55 / 5.56 / 5.73.
extern "C" __global__ void __launch_bounds__(LYAP_SPEC_THREADS, (sizeof(LYAP_SPEC_FAST::real) == 8 ? 640 : 768) / LYAP_SPEC_THREADS)
k_lambda_fast_spec(const __grid_constant__ LambdaArgs a, double* __restrict__ out64, float* __restrict__ out32,
                   unsigned long long* __restrict__ steps_out) {
    lambda_fast_body<LYAP_SPEC_FAST, LYAP_SPEC_P, LYAP_SPEC_THREADS, LYAP_SPEC_KG, LYAP_SPEC_WU_PATS, LYAP_SPEC_ACC_PATS>(
        a, out64, out32, steps_out);
}
#endif


}  // namespace lyap
