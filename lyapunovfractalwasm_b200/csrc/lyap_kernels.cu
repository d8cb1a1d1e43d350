// lyap_kernels.cu -- sm_100a kernels of the Lyapunov-fractal engine.
//
//   k_lambda_exact   FractalComputer::computeFractal  (reference src/lyapunov_fractal.hpp:41-86)
//   k_minmax         normalizeData pass 1             (src/lyapunov_fractal.hpp:110-120)
//   k_normalize      normalizeData pass 2             (src/lyapunov_fractal.hpp:122-137)
//   k_colorize       box mean + palette + RGBA store  (web/fractal_renderer.js:283-311,207-281,191-198)
//
// Build with -fmad=false: the exact kernels may only fuse where an fma is written out.
#include <algorithm>
#include <cfloat>
#include <math_constants.h>
#include <cstdint>
#include <cstdlib>

#include "lyap_engine.h"
#include "lyap_math.h"

#include "lyap_exact_kernel.cuh"
#include "lyap_kernels_fast.cuh"

namespace lyap {

// The wide tiles' shape.  2048 x 2048 of "AABAB" 200 + 2000 / "BBBBBBAAAAAA" 500 + 4000, frame 0 of the zoom (a third of its
// orbits end) and the 800 x 800 page: 2 pixels a thread 7.92 / 15.75 / 4.48 / 0.676 ms, 3 pixels 7.90 / 15.96 / 4.66 / 0.716,
// 3 pixels side by side in a row 7.84 / 15.80 / 4.90 / 0.705 (128 registers and a few spilled); 4 of 384 threads 8.00 / 16.9
// (all before cycles were cut short).  The generic kernel picks a straight-line body every two steps for all of a thread's
// pixels: 3 pixels 1.02 ms, 2 pixels 1.07 (1277 x 719 over [3.8,4]^2, 37 letters, 100 + 1000).
constexpr int kExactThreads = 512, kExactPixels = 2, kGenericPixels = 3;

template <int P, bool HAS_C, int UNROLL>
static cudaError_t launch_exact_generic(const LambdaArgs& a, double* out64, float* out32, unsigned long long* steps,
                                        unsigned grid, cudaStream_t st) {
    auto kern = k_lambda_exact<P, kExactThreads, HAS_C, UNROLL>;
    constexpr size_t smem = kExactSmemBytes;
    // the attribute is per device and cheap to set; doing it on every launch keeps this thread- and device-safe
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, kExactThreads, smem, st>>>(a, out64, out32, steps);
    note_lambda_kernel(P == 1 ? "k_lambda_exact<1,512> (generic: patterns dispatched every 4 steps)"
                              : "k_lambda_exact<3,512> (generic: patterns dispatched every 2 steps)");
    return cudaGetLastError();
}

// LYAP_JIT: 0 never compile at run time, 1 (default) once enough work with a sequence has been seen, 2 at once.
// LYAP_PREBUILT=0: ignore the instances compiled at build time (with LYAP_JIT=0 that forces the generic kernels).
static int spec_mode() {
    const char* je = getenv("LYAP_JIT");
    const char* pe = getenv("LYAP_PREBUILT");
    const int jit = je ? atoi(je) : 1;
    const int pre = pe ? atoi(pe) : 1;
    return (jit < 0 ? 0 : (jit > 2 ? 2 : jit)) | (pre ? kSpecUsePrebuilt : 0);
}

// Deals a launch out: `wide_tiles` of `pixels` a thread first (as far as the rows' whole groups hold them), then tiles of 32
// pixels, which even out the end.  With `rounds` or fewer tiles a warp the launch does without a queue.  Returns the grid: the
// shared tables allow one CTA per SM.
static unsigned deal_exact(LambdaArgs* a, int pixels, long long wide_tiles, int rounds, int sm_count) {
    const long long groups = a->n_pixels / a->width / pixels * a->width / 32;   // wide tiles in the rows' whole groups
    a->wide_tiles = std::max(0LL, std::min(wide_tiles, groups));
    const long long warp_tiles = a->wide_tiles + (a->n_pixels - a->wide_tiles * 32 * pixels + 31) / 32;
    if (warp_tiles <= (long long)rounds * kExactThreads / 32 * sm_count) a->queue = nullptr;
    return (unsigned)std::min<long long>(warp_tiles, sm_count);
}

cudaError_t launch_lambda_exact(const LambdaArgs& args, double* out64, float* out32, unsigned long long* steps,
                                int sm_count, cudaStream_t st) {
    if (args.n_pixels <= 0) return cudaSuccess;
    LambdaArgs a = args;
    // A periodic sequence can run an instance of this kernel made for its patterns.
    // Frames of up to 40 tiles of 32 a scheduler go in such tiles alone: with 4 / 8 / 16 / 32 / all of them 800 x 800 of "AB"
    // 100 + 1000 over [0.01,3.99]^2 takes 471 / 471 / 471 / 447 / 426 us and 512 x 512 over [2,4]^2 215 / 210 / 202 / 202 / 202;
    // 1920 x 1080 of "ABC" 300 + 3000 3675 / 3694 / 3701 / 3717 / 3758.
    // Orbits of one length end on an SM's 16 warps at once, which then take 16 tiles from the queue where others get none: two
    // rounds of tiles and fewer are dealt out beforehand (315 x 305 of "AB" 82 + 821 over [3.4,4]x[2.5,3.4]: 126 -> 104 us).
    // Runs long enough for cycles to be cut short make uneven tiles, which small ones and the queue even out.  Those of shorter runs
    // end together: whole rounds of wide tiles over the schedulers, all dealt out beforehand (744 x 659 of "ABC" 24 + 213 137 -> 122 us,
    // 1074 x 549 of "AABAB" 25 + 158 132 -> 118; 550 x 530 of "BBBBBBAAAAAA" 20 + 399 over [2,4]^2 is better in small ones, 126 us
    // against 166).
    const long long schedulers = 4LL * sm_count, tiles = (a.n_pixels + 31) / 32;
    const bool uneven = a.acc_period && a.iterations >= 300;
    long long wide = (tiles - 2 * schedulers) / (kExactPixels * schedulers) * schedulers;
    if (uneven) wide = tiles <= 40 * schedulers ? 0 : (tiles - 8 * schedulers) / kExactPixels;
    else a.queue = nullptr;
    unsigned grid = deal_exact(&a, kExactPixels, wide, 2, sm_count);
    bool launched = false;
    const cudaError_t e = launch_lambda_spec(a, out64, out32, steps, grid, st, 0, kExactPixels, kExactThreads, kExactSmemBytes,
                                             spec_mode(), &launched);
    if (e != cudaSuccess || launched) return e;
    bool has_c = false;
    const int words = a.acc_word0 + (a.iterations > 0 ? min(a.acc_wrap, (a.iterations - 1) / kStepsPerWord + 1) : 0);
    for (int i = 0; i < words; ++i) has_c = has_c || (a.sel[i] & 0xAAAAAAAAu);
    // The generic kernel's choice of a body serves all of a thread's pixels, so that its large frames have four small tiles a
    // scheduler only (1277 x 719 of 37 letters with 4 / 8 / 16 / 32 / all 864 / 892 / 930 / 989 / 1028 us).  Frames of few tiles go
    // in small ones alone, through a kernel that has four steps to a body; more, up to what one round of warps holds, in as few
    // wide tiles as fill it.  Short runs' even tiles: there a round begins earlier (454 x 247 of 37 letters 24 + 218 56 us in small
    // tiles, 49 in a round), and a few rounds are dealt out beforehand (685 x 485, 11 + 111: 65 us from the queue, 60).
    // 37 letters in four small tiles a scheduler beyond the wide ones, and small ones alone up to six / this: 64 x 32 100 + 4000 296 /
    // 249 us, 437 x 385 230 + 2304 over [3.9,4]^2 552 / 457, 357 x 213 of "ABBAB" 24 + 1700 over [0,4]^2 219 / 194.
    a.queue = args.queue;
    if (tiles <= (uneven ? 6 : 5) * schedulers) {
        grid = deal_exact(&a, 1, 0, 1, sm_count);
        return has_c ? launch_exact_generic<1, true, 2>(a, out64, out32, steps, grid, st)
                     : launch_exact_generic<1, false, 4>(a, out64, out32, steps, grid, st);
    }
    wide = (tiles - 4 * schedulers) / kGenericPixels;
    if (tiles <= 4 * kGenericPixels * schedulers) wide = (tiles - 2 * schedulers - 1) / (2 * schedulers) * schedulers;
    else if (!uneven && tiles <= 8 * kGenericPixels * schedulers) {
        wide = (tiles - 2 * schedulers) / (kGenericPixels * schedulers) * schedulers;
        a.queue = nullptr;
    }
    grid = deal_exact(&a, kGenericPixels, wide, 1, sm_count);
    return has_c ? launch_exact_generic<kGenericPixels, true, 2>(a, out64, out32, steps, grid, st)
                 : launch_exact_generic<kGenericPixels, false, 2>(a, out64, out32, steps, grid, st);
}

// ---------------------------------------------------------------------------------------------
// normalizeData pass 1: min / max over finite values > -4.
// Results are selections, so any reduction order gives the reference's bits.
// ---------------------------------------------------------------------------------------------
constexpr int kMinmaxThreads = 256;

// N values.  Zeros are ordered by their sign, whichever comes first, as fmin and fmax do; without one among the values a
// comparison and a select, which are shorter, come to the same.
template <int N>
__device__ __forceinline__ void minmax_take(const double (&v)[N], double& lo, double& hi) {
    bool zero = false;
#pragma unroll
    for (int k = 0; k < N; ++k) zero = zero || v[k] == 0.0;
    if (zero) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (v[k] > -4.0 && v[k] <= DBL_MAX) {     // :116
                lo = fmin(lo, v[k]);
                hi = fmax(hi, v[k]);
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (v[k] > -4.0 && v[k] <= DBL_MAX) {
                lo = v[k] < lo ? v[k] : lo;
                hi = v[k] > hi ? v[k] : hi;
            }
        }
    }
}

// 8 blocks an SM at once, as many as are launched (with 34 registers 6 fit, and the others wait for them), and four loads in
// flight a thread.  8.3 million values: 20.4 us with one load, 17.8 so; 2^26 values (6.2 TB/s now): 89 us with one load, 102
// with four and 34 registers, 87 so; the same not 16-byte aligned 140, 230 and 86.
__global__ void __launch_bounds__(kMinmaxThreads, 8)
k_minmax(const double* __restrict__ v, unsigned long long n, double* __restrict__ minmax, double* partial,
         unsigned int* ticket) {
    double lo = DBL_MAX, hi = -DBL_MAX;   // :110-111
    const unsigned long long tid = (unsigned long long)blockIdx.x * kMinmaxThreads + threadIdx.x;
    const unsigned long long nthreads = (unsigned long long)gridDim.x * kMinmaxThreads;
    const bool aligned = (reinterpret_cast<uintptr_t>(v) & 15) == 0;
    unsigned long long i = tid;
    if (aligned) {
        const unsigned long long n2 = n / 2;
        const double2* v2 = reinterpret_cast<const double2*>(v);
        for (; i + 3 * nthreads < n2; i += 4 * nthreads) {
            double q[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double2 pair = v2[i + k * nthreads];
                q[2 * k] = pair.x;
                q[2 * k + 1] = pair.y;
            }
            minmax_take(q, lo, hi);
        }
        for (; i < n2; i += nthreads) {
            const double2 pair = v2[i];
            const double q[2] = {pair.x, pair.y};
            minmax_take(q, lo, hi);
        }
        i = (n & ~1ull) + tid;   // the last of an odd number
    } else {
        for (; i + 3 * nthreads < n; i += 4 * nthreads) {
            double q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k] = v[i + k * nthreads];
            minmax_take(q, lo, hi);
        }
    }
    for (; i < n; i += nthreads) {
        const double q[1] = {v[i]};
        minmax_take(q, lo, hi);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_down_sync(0xFFFFFFFFu, lo, o));
        hi = fmax(hi, __shfl_down_sync(0xFFFFFFFFu, hi, o));
    }
    __shared__ double s_lo[kMinmaxThreads / 32], s_hi[kMinmaxThreads / 32];
    __shared__ bool s_last;
    if ((threadIdx.x & 31) == 0) {
        s_lo[threadIdx.x >> 5] = lo;
        s_hi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kMinmaxThreads / 32; ++w) {
            lo = fmin(lo, s_lo[w]);
            hi = fmax(hi, s_hi[w]);
        }
        partial[2 * blockIdx.x] = lo;
        partial[2 * blockIdx.x + 1] = hi;
        __threadfence();
        const unsigned t = atomicAdd(ticket, 1u);
        s_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        lo = DBL_MAX;
        hi = -DBL_MAX;
        for (unsigned b = threadIdx.x; b < gridDim.x; b += kMinmaxThreads) {
            lo = fmin(lo, __ldcg(&partial[2 * b]));
            hi = fmax(hi, __ldcg(&partial[2 * b + 1]));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fmin(lo, __shfl_down_sync(0xFFFFFFFFu, lo, o));
            hi = fmax(hi, __shfl_down_sync(0xFFFFFFFFu, hi, o));
        }
        __syncthreads();
        if ((threadIdx.x & 31) == 0) {
            s_lo[threadIdx.x >> 5] = lo;
            s_hi[threadIdx.x >> 5] = hi;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < kMinmaxThreads / 32; ++w) {
                lo = fmin(lo, s_lo[w]);
                hi = fmax(hi, s_hi[w]);
            }
            minmax[0] = lo;
            minmax[1] = hi;
            *ticket = 0;   // ready for the next launch
        }
    }
}

cudaError_t launch_minmax(const double* v, unsigned long long n, double* minmax, void* scratch, int sm_count, cudaStream_t st) {
    double* partial = static_cast<double*>(scratch);
    unsigned int* ticket = reinterpret_cast<unsigned int*>(partial + 2 * kMinmaxBlocks);
    unsigned long long want = (n / 2 + kMinmaxThreads - 1) / kMinmaxThreads;
    if (want < 1) want = 1;
    // 8 blocks per SM of this device, never more than the scratch has room for
    const unsigned long long cap = (unsigned long long)(8 * sm_count < kMinmaxBlocks && sm_count > 0 ? 8 * sm_count : kMinmaxBlocks);
    const int grid = (int)(want < cap ? want : cap);
    k_minmax<<<grid, kMinmaxThreads, 0, st>>>(v, n, minmax, partial, ticket);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Min/max without any allocation (lyap_minmax_device_noalloc in the public header).
//
// Same kernel as above; its scratch (per-block partial results and the arrival ticket) is this fixed
// array in the library image instead of memory owned by a context.  In host code the array's name is
// only a handle: the address a kernel can use is obtained once per device with cudaGetSymbolAddress,
// with that device current, and cached.
// ---------------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_minmax_fixed_scratch[(kMinmaxScratchBytes + 255) / 256 * 256];

}  // namespace lyap

#include <mutex>

#include "../../include/lyap_b200.h"

extern "C" int lyap_minmax_device_noalloc(const double* d_values, uint64_t n, double* d_minmax, void* cuda_stream) {
    using namespace lyap;
    if (!d_minmax || (!d_values && n)) return set_error(LYAP_ERR_INVALID, "lyap_minmax_device_noalloc: null pointer");
    if (n > LYAP_NOALLOC_MAX_VALUES)
        return set_error(LYAP_ERR_TOO_LARGE, "lyap_minmax_device_noalloc: n exceeds LYAP_NOALLOC_MAX_VALUES (2^32 values)");
    constexpr int kMaxDevices = LYAP_NOALLOC_MAX_DEVICES;
    static std::mutex mu;
    static void* scratch_of_device[kMaxDevices] = {};
    static int sm_count_of_device[kMaxDevices] = {};
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(LYAP_ERR_CUDA, cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices)
        return set_error(LYAP_ERR_INVALID, "lyap_minmax_device_noalloc: device ordinal beyond LYAP_NOALLOC_MAX_DEVICES");
    void* scratch = nullptr;
    int sm_count = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!scratch_of_device[dev]) {   // one-time set-up for this device (it is the current one)
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_minmax_fixed_scratch);
            if (e != cudaSuccess) return set_error(LYAP_ERR_CUDA, cudaGetErrorString(e));
            int sms = 0;
            e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return set_error(LYAP_ERR_CUDA, cudaGetErrorString(e));
            sm_count_of_device[dev] = sms;
            scratch_of_device[dev] = p;
        }
        scratch = scratch_of_device[dev];
        sm_count = sm_count_of_device[dev];
    }
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    // the arrival ticket must start at zero; the array keeps whatever the last call (or an aborted one) left
    unsigned int* ticket = reinterpret_cast<unsigned int*>(static_cast<double*>(scratch) + 2 * kMinmaxBlocks);
    e = cudaMemsetAsync(ticket, 0, 16, st);
    if (e != cudaSuccess) return set_error(LYAP_ERR_CUDA, cudaGetErrorString(e));
    e = launch_minmax(d_values, n, d_minmax, scratch, sm_count, st);
    if (e != cudaSuccess) return set_error(LYAP_ERR_CUDA, cudaGetErrorString(e));
    return LYAP_OK;
}

namespace lyap {

// ---------------------------------------------------------------------------------------------
// normalizeData pass 2.
// ---------------------------------------------------------------------------------------------
constexpr int kNormThreads = 256;

// Constants of the plain functions below in constant memory, where an fp64 instruction reads them as an operand: as literals
// they are put together in registers by two instructions each, which was more than half of what these kernels issued.
struct ColourConsts {
    double invln2, ln2hi, ln2lo, exp_c[13], log_c2, log_c3, log_c4, klo_bias;
    double two_over_pi, pio2[3], sin_c[7], cos_c[7];
    double pi, third2pi, third4pi, pal[5];   // pal: 0.8, 0.3, 0.9, 0.7, 0.6
    double fifth, tenth, p95, y12;
    double recip[10];                         // of a number of neighbours
};
static __constant__ ColourConsts c_col = {
    LYAP_INVLN2, LYAP_LN2HI, LYAP_LN2LO,
    {LYAP_EXP_C2, LYAP_EXP_C3, LYAP_EXP_C4, LYAP_EXP_C5, LYAP_EXP_C6, LYAP_EXP_C7, LYAP_EXP_C8, LYAP_EXP_C9, LYAP_EXP_C10,
     LYAP_EXP_C11, LYAP_EXP_C12, LYAP_EXP_C13, LYAP_EXP_C14},
    LYAP_LOG_C2, LYAP_LOG_C3, LYAP_LOG_C4, LYAP_KLO_BIAS,
    LYAP_2OVERPI, {LYAP_PIO2_1, LYAP_PIO2_2, LYAP_PIO2_3},
    {LYAP_SIN_C0, LYAP_SIN_C1, LYAP_SIN_C2, LYAP_SIN_C3, LYAP_SIN_C4, LYAP_SIN_C5, LYAP_SIN_C6},
    {LYAP_COS_C0, LYAP_COS_C1, LYAP_COS_C2, LYAP_COS_C3, LYAP_COS_C4, LYAP_COS_C5, LYAP_COS_C6},
    LYAP_PI, 2.0 * LYAP_PI / 3.0, 4.0 * LYAP_PI / 3.0, {0.8, 0.3, 0.9, 0.7, 0.6}, 0.2, 0.1, 0.95, 1.2,
    {0.0, 1.0, 1.0 / 2.0, 1.0 / 3.0, 1.0 / 4.0, 1.0 / 5.0, 1.0 / 6.0, 1.0 / 7.0, 1.0 / 8.0, 1.0 / 9.0}};

// lyap_exp for |x| <= 600: no special values, and the power of two goes in by adding to the exponent field (lyap_exp
// multiplies by it: the same, as nothing leaves the normal range).  The integer is the low word of the shifted sum; a
// conversion costs as much as eight fp64 instructions.
__device__ __forceinline__ double exp_plain(double x) {
    const double magic = 0x1.8p52;
    const double z = __fma_rn(x, c_col.invln2, magic);
    const double nf = __dsub_rn(z, magic);
    double r = __fma_rn(-nf, c_col.ln2hi, x);
    r = __fma_rn(-nf, c_col.ln2lo, r);
    double p = __fma_rn(c_col.exp_c[12], r, c_col.exp_c[11]);
#pragma unroll
    for (int k = 10; k >= 0; --k) p = __fma_rn(p, r, c_col.exp_c[k]);
    const double v = __dadd_rn(1.0, __fma_rn(p, __dmul_rn(r, r), r));
    return __hiloint2double(__double2hiint(v) + (__double2loint(z) << 20), __double2loint(v));
}

// lyap_pow_tab for 2^-300 <= t <= 2 and 1 <= y <= 1.5, without its special cases
__device__ __forceinline__ double pow_plain(double t, double y, const lyap_logtab_entry* tab) {
    const unsigned hw = (unsigned)__double2hiint(t);   // lyap_log_core
    const lyap_logtab_entry ent = tab[(hw >> 10) & (LYAP_LOG_BINS - 1)];
    const double m = __hiloint2double((int)((hw & 0x000FFFFFu) | 0x3FF00000u), __double2loint(t));
    const double kd = __dsub_rn(__hiloint2double(0x43300000, (int)(hw >> 20)), 0x1p52);
    const double r = __fma_rn(m, ent.invc, -1.0);
    double w = __fma_rn(r, c_col.log_c4, c_col.log_c3);
    w = __fma_rn(r, w, c_col.log_c2);
    w = __fma_rn(r, w, 1.0);
    const double s = __fma_rn(r, w, __fma_rn(kd, c_col.ln2lo, c_col.klo_bias));
    const double hi = __fma_rn(kd, c_col.ln2hi, ent.lp);
    const double zh = __dadd_rn(hi, s);
    const double bb = __dsub_rn(zh, hi);
    const double zl = __dadd_rn(__dsub_rn(hi, __dsub_rn(zh, bb)), __dsub_rn(s, bb));
    const double ph = __dmul_rn(y, zh);
    const double pl = __dadd_rn(__fma_rn(y, zh, -ph), __dmul_rn(y, zl));
    const double e = exp_plain(ph);
    return t == 1.0 ? 1.0 : __fma_rn(e, pl, e);
}

// any value, special ones included
__device__ __noinline__ double normalize_any(double val, double t, const lyap_logtab_entry* tab) {
    if (!(isfinite(val) && val > -4.0)) return 0.0;                                      // :130,135
    const double s = lyap_pow_tab(t, 1.2, tab, 1);                                       // :132
    return __ddiv_rn(1.0, __dadd_rn(1.0, lyap_exp(__dmul_rn(-7.0, __dsub_rn(s, 0.5)))));   // :133
}

__device__ __forceinline__ double sigmoid_plain(double s) {                             // :133
    return __drcp_rn(__dadd_rn(1.0, exp_plain(__dmul_rn(-7.0, __dsub_rn(s, 0.5)))));
}

// Bound by the fp64 pipe and its register reads: 71 fp64 instructions a value in two exponentials and a logarithm.  A value
// as a frame has them takes the plain functions; sentinels, the minimum itself, NaN and whatever a caller's own min and max
// make of a value are put right afterwards (same bits), so that a thread's common way has no branch in it; a warp that has
// none but such values leaves it out.
// 3840 x 2160 with the launch (5 us), a branch a value / no way out for a warp and the load at the top of the loop / as here:
// ordinary values 85 / 60 / 58 us (the pipe alone 33), half of them sentinels 85 / 65 / 60, all but a few the minimum
// 48 / 78 / 35; with 4 instead of 8 blocks per SM 3 us more.
template <int N>
__device__ __forceinline__ void normalize_some(const double (&val)[N], double (&out)[N], double mn, double range_inv,
                                               const lyap_logtab_entry* tab) {
    double t[N];
    bool plain[N], any = false, all = true;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        t[k] = __dmul_rn(__dsub_rn(val[k], mn), range_inv);                              // :131
        plain[k] = val[k] > -4.0 && t[k] >= 0x1p-300 && t[k] <= 2.0;                      // then val is finite, :130
        any = any || plain[k];
        all = all && plain[k];
    }
    if (__any_sync(__activemask(), any)) {
#pragma unroll
        for (int k = 0; k < N; ++k)
            out[k] = sigmoid_plain(pow_plain(plain[k] ? t[k] : 1.0, c_col.y12, tab));    // :132, below 2.3
        if (all) return;
    }
    const double least = sigmoid_plain(0.0);                                             // of t = 0
#pragma unroll
    for (int k = 0; k < N; ++k) {
        if (plain[k]) continue;
        if (!(val[k] > -4.0 && val[k] <= DBL_MAX)) out[k] = 0.0;                         // :130,135
        else if (t[k] == 0.0) out[k] = least;
        else out[k] = normalize_any(val[k], t[k], tab);
    }
}

__global__ void __launch_bounds__(kNormThreads, 4)
k_normalize(const double* __restrict__ v, unsigned long long n, const double* __restrict__ minmax,
            double* __restrict__ out) {
    __shared__ lyap_logtab_entry tab[LYAP_LOG_BINS];
    for (int e = threadIdx.x; e < LYAP_LOG_BINS; e += kNormThreads) tab[e] = g_lyap_logtab[e];
    __syncthreads();
    const double mn = minmax[0], mx = minmax[1];
    const double range_inv = __ddiv_rn(1.0, __dsub_rn(mx, mn));                          // :124-125
    const unsigned long long tid = (unsigned long long)blockIdx.x * kNormThreads + threadIdx.x;
    const unsigned long long nthreads = (unsigned long long)gridDim.x * kNormThreads;
    if (mn >= mx) {                                                                      // :122
        for (unsigned long long i = tid; i < n; i += nthreads) out[i] = 0.0;
        return;
    }
    const bool aligned = ((reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    if (aligned) {
        const unsigned long long n2 = n / 2;
        const double2* v2 = reinterpret_cast<const double2*>(v);
        double2* o2 = reinterpret_cast<double2*>(out);
        double2 next = tid < n2 ? v2[tid] : make_double2(0.0, 0.0);   // loaded a turn of the loop ahead: the branches hold loads back
        for (unsigned long long i = tid; i < n2; i += nthreads) {
            const double val[2] = {next.x, next.y};
            if (i + nthreads < n2) next = v2[i + nthreads];
            double r[2];
            normalize_some(val, r, mn, range_inv, tab);
            o2[i] = make_double2(r[0], r[1]);
        }
    }
    // values of a misaligned array, the last of an odd number
    for (unsigned long long i = aligned ? (n & ~1ull) + tid : tid; i < n; i += nthreads) {
        const double val[1] = {v[i]};
        double r[1];
        normalize_some(val, r, mn, range_inv, tab);
        out[i] = r[0];
    }
}

cudaError_t launch_normalize(const double* v, unsigned long long n, const double* minmax, double* out,
                             int sm_count, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    unsigned long long want = (n / 2 + kNormThreads - 1) / kNormThreads;
    if (want < 1) want = 1;
    const unsigned long long cap = (unsigned long long)sm_count * 8;
    const int grid = (int)(want < cap ? want : cap);
    k_normalize<<<grid, kNormThreads, 0, st>>>(v, n, minmax, out);
    return cudaGetLastError();
}

// A block for kernels whose threads each take a column of a strip of rows: the width dealt out evenly over as few blocks as
// cover it, and as many strips on top of one another as there are threads left.  Whole warps of columns where a block has
// one strip; in a narrower frame a warp goes on with the next strip's first columns.
static dim3 column_block(int width, int threads) {
    const long long blocks = ((long long)width + threads - 1) / threads;
    const int columns = (int)((width + blocks - 1) / blocks);
    return columns > threads / 2 ? dim3((unsigned)(columns + 31) / 32 * 32, 1) : dim3((unsigned)columns, (unsigned)(threads / columns));
}

// ---------------------------------------------------------------------------------------------
// Colour stage: 3x3 mean (edge-aware, fixed summation order) -> palette -> clamped bytes, alpha 255.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned clamp_u8(double v) {   // Uint8ClampedArray store of an integer-valued double
    if (!(v > 0.0)) return 0u;                              // negatives and NaN -> 0
    if (v >= 255.0) return 255u;
    return (unsigned)(int)v;
}

__device__ __forceinline__ double hue2rgb(double p, double q, double t) {   // web/fractal_renderer.js:32-39
    if (t < 0) t = __dadd_rn(t, 1.0);
    if (t > 1) t = __dsub_rn(t, 1.0);
    if (t < 1.0 / 6) return __dadd_rn(p, __dmul_rn(__dmul_rn(__dsub_rn(q, p), 6.0), t));
    if (t < 1.0 / 2) return q;
    if (t < 2.0 / 3) return __dadd_rn(p, __dmul_rn(__dmul_rn(__dsub_rn(q, p), __dsub_rn(2.0 / 3, t)), 6.0));
    return p;
}

__device__ __forceinline__ double scale255(double v) { return floor(__dmul_rn(255.0, v)); }

// any t, special values included
__device__ __noinline__ unsigned palette_rgba(double t, int palette, const lyap_logtab_entry* tab) {
    const double PI = LYAP_PI;
    const double mid = __dmul_rn(fabs(__dsub_rn(t, 0.5)), 2.0);
    const double I = __dsub_rn(1.0, mid);
    double r, g, b;
    switch (palette) {
        default:
        case 0: {   // cosmic :209-218
            const double ph = __dmul_rn(mid, PI);
            r = scale255(__dadd_rn(__dmul_rn(I, 0.8), __dmul_rn(0.2, lyap_sin(ph))));
            g = scale255(__dmul_rn(I, 0.3));
            b = scale255(__dadd_rn(__dmul_rn(I, 0.9), __dmul_rn(0.1, lyap_cos(ph))));
        } break;
        case 1:     // nebula :219-227
            r = scale255(__dadd_rn(__dmul_rn(I, 0.9), __dmul_rn(0.1, lyap_pow_tab(t, 1.5, tab, 1))));
            g = scale255(__dmul_rn(I, 0.5));
            b = scale255(__dmul_rn(I, 0.8));
            break;
        case 2: {   // aurora :228-237
            const double ph = __dmul_rn(mid, PI);
            r = scale255(__dmul_rn(I, 0.6));
            g = scale255(__dadd_rn(__dmul_rn(I, 0.9), __dmul_rn(0.1, lyap_sin(ph))));
            b = scale255(__dmul_rn(I, 0.7));
        } break;
        case 3:     // solarflare :238-246
            r = scale255(__dmul_rn(I, 0.95));
            g = scale255(__dmul_rn(I, 0.6));
            b = scale255(__dmul_rn(I, 0.2));
            break;
        case 4: {   // blackhole :247-256
            const double ph = __dmul_rn(mid, PI);
            r = scale255(__dmul_rn(I, 0.5));
            g = scale255(__dmul_rn(I, 0.7));
            b = scale255(__dadd_rn(__dmul_rn(I, 0.9), __dmul_rn(0.1, lyap_sin(ph))));
        } break;
        case 5: {   // psychedelic :257-266
            const double ph = __dmul_rn(__dmul_rn(t, PI), 6.0);
            const double o1 = __ddiv_rn(__dmul_rn(2.0, PI), 3.0), o2 = __ddiv_rn(__dmul_rn(4.0, PI), 3.0);
            r = scale255(__dmul_rn(I, __dadd_rn(0.5, __dmul_rn(0.5, lyap_sin(ph)))));
            g = scale255(__dmul_rn(I, __dadd_rn(0.5, __dmul_rn(0.5, lyap_sin(__dadd_rn(ph, o1))))));
            b = scale255(__dmul_rn(I, __dadd_rn(0.5, __dmul_rn(0.5, lyap_sin(__dadd_rn(ph, o2))))));
        } break;
        case 6: {   // rainbow :267-278 with hslToRgb(hue, 1, 0.5) :26-47
            const double h = __ddiv_rn(__dmul_rn(t, 360.0), 360.0);
            const double q = 1.0, p = 0.0;
            const double cr = hue2rgb(p, q, __dadd_rn(h, 1.0 / 3));
            const double cg = hue2rgb(p, q, h);
            const double cb = hue2rgb(p, q, __dsub_rn(h, 1.0 / 3));
            r = scale255(__dmul_rn(I, cr));
            g = scale255(__dmul_rn(I, cg));
            b = scale255(__dmul_rn(I, cb));
        } break;
    }
    return clamp_u8(r) | (clamp_u8(g) << 8) | (clamp_u8(b) << 16) | 0xFF000000u;
}

// The palette for the t of a picture, 0 <= t <= 1 (nebula: 2^-300 <= t): palette_rgba's operations without special cases.
// Sine and cosine of one angle share their reduction and their two polynomials, and a channel's floor is one addition that
// rounds down.
__device__ __forceinline__ void sincos_plain(double x, double* sn, double* cs) {   // 0 <= x <= 24: lyap_sin, lyap_cos
    const double magic = 0x1.8p52;
    const double z = __fma_rn(x, c_col.two_over_pi, magic);
    const double nf = __dsub_rn(z, magic);
    double r = __fma_rn(-nf, c_col.pio2[0], x);
    r = __fma_rn(-nf, c_col.pio2[1], r);
    r = __fma_rn(-nf, c_col.pio2[2], r);
    const int q = __double2loint(z);
    const double u = __dmul_rn(r, r);
    double p = c_col.sin_c[6], w = c_col.cos_c[6];   // lyap_sin_kernel, lyap_cos_kernel
#pragma unroll
    for (int k = 5; k >= 0; --k) {
        p = __fma_rn(p, u, c_col.sin_c[k]);
        w = __fma_rn(w, u, c_col.cos_c[k]);
    }
    const double s = __fma_rn(__dmul_rn(r, u), p, r);
    const double c = __fma_rn(__dmul_rn(u, u), w, __fma_rn(u, -0.5, 1.0));
    const double a = (q & 1) ? c : s, b = (q & 1) ? s : c;
    *sn = (q & 2) ? -a : a;
    *cs = ((q + 1) & 2) ? -b : b;
}

__device__ __forceinline__ double sin_plain(double x) {
    double s, c;
    sincos_plain(x, &s, &c);
    return s;
}

__device__ __forceinline__ unsigned channel(double v) {   // clamp_u8(scale255(v)) for |v| < 2^20
    const int n = __double2loint(__dadd_rd(__dmul_rn(255.0, v), 0x1.8p52));
    return (unsigned)max(0, min(255, n));
}

template <int PALETTE>
__device__ __forceinline__ unsigned palette_plain(double t, const lyap_logtab_entry* tab) {
    const double mid = __dmul_rn(fabs(__dsub_rn(t, 0.5)), 2.0);
    const double I = __dsub_rn(1.0, mid);
    double r, g, b;
    if (PALETTE == 0) {          // cosmic
        double sn, cs;
        sincos_plain(__dmul_rn(mid, c_col.pi), &sn, &cs);
        r = __dadd_rn(__dmul_rn(I, c_col.pal[0]), __dmul_rn(c_col.fifth, sn));
        g = __dmul_rn(I, c_col.pal[1]);
        b = __dadd_rn(__dmul_rn(I, c_col.pal[2]), __dmul_rn(c_col.tenth, cs));
    } else if (PALETTE == 1) {   // nebula
        r = __dadd_rn(__dmul_rn(I, c_col.pal[2]), __dmul_rn(c_col.tenth, pow_plain(t, 1.5, tab)));
        g = __dmul_rn(I, 0.5);
        b = __dmul_rn(I, c_col.pal[0]);
    } else if (PALETTE == 2) {   // aurora
        r = __dmul_rn(I, c_col.pal[4]);
        g = __dadd_rn(__dmul_rn(I, c_col.pal[2]), __dmul_rn(c_col.tenth, sin_plain(__dmul_rn(mid, c_col.pi))));
        b = __dmul_rn(I, c_col.pal[3]);
    } else if (PALETTE == 3) {   // solarflare
        r = __dmul_rn(I, c_col.p95);
        g = __dmul_rn(I, c_col.pal[4]);
        b = __dmul_rn(I, c_col.fifth);
    } else if (PALETTE == 4) {   // blackhole
        r = __dmul_rn(I, 0.5);
        g = __dmul_rn(I, c_col.pal[3]);
        b = __dadd_rn(__dmul_rn(I, c_col.pal[2]), __dmul_rn(c_col.tenth, sin_plain(__dmul_rn(mid, c_col.pi))));
    } else if (PALETTE == 5) {   // psychedelic
        const double ph = __dmul_rn(__dmul_rn(t, c_col.pi), 6.0);
        r = __dmul_rn(I, __dadd_rn(0.5, __dmul_rn(0.5, sin_plain(ph))));
        g = __dmul_rn(I, __dadd_rn(0.5, __dmul_rn(0.5, sin_plain(__dadd_rn(ph, c_col.third2pi)))));
        b = __dmul_rn(I, __dadd_rn(0.5, __dmul_rn(0.5, sin_plain(__dadd_rn(ph, c_col.third4pi)))));
    } else {                     // rainbow
        const double h = __ddiv_rn(__dmul_rn(t, 360.0), 360.0);
        r = __dmul_rn(I, hue2rgb(0.0, 1.0, __dadd_rn(h, 1.0 / 3)));
        g = __dmul_rn(I, hue2rgb(0.0, 1.0, h));
        b = __dmul_rn(I, hue2rgb(0.0, 1.0, __dsub_rn(h, 1.0 / 3)));
    }
    return channel(r) | (channel(g) << 8) | (channel(b) << 16) | 0xFF000000u;
}

constexpr int kColorThreads = 256;

// One pixel from its 3 x 3 values (row by row), `count` of them there: summed in the page's order, and divided through the
// reciprocal: with y = RN(1/n), q = RN(s*y) is within an ulp of s/n, and RN(q + y*(s - nq)) is s/n correctly rounded
// (Markstein 1990).  A mean above 1 goes the general way, one below 2^-300 where the palette takes its power: the others'
// channels are multiples of I or functions of `mid`, 0 and 1 for any t below 2^-54.
template <int PALETTE>
__device__ __forceinline__ unsigned colorize_inner(const double (&above)[3], const double (&row)[3], const double (&below)[3],
                                                   double count, double recip, const lyap_logtab_entry* tab) {
    double s = row[1];                                                                   // :292
#pragma unroll
    for (int k = 0; k < 3; ++k) s = __dadd_rn(s, above[k]);
    s = __dadd_rn(s, row[0]);
    s = __dadd_rn(s, row[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) s = __dadd_rn(s, below[k]);
    const double q = __dmul_rn(s, recip);
    const double t = __fma_rn(__fma_rn(-count, q, s), recip, q);                         // :307
    if (t >= (PALETTE == 1 ? 0x1p-300 : 0.0) && t <= 1.0) return palette_plain<PALETTE>(t, tab);
    return palette_rgba(__ddiv_rn(s, count), PALETTE, tab);
}

// A thread takes one column of kColorRows rows: its rows' values and their left and right neighbours are loaded once, side by
// side across the warp, and stay in registers for the pixels above and below.  A block is up to 256 columns wide and, in a
// narrow frame, as many strips high as fill it.  A warp with a pixel at the frame's edge goes row by row and
// takes -0 for a neighbour that is not there, which leaves any sum as it is.  The palette is a template parameter: its code is
// then straight-line.
// 3840 x 2160 with the launch, aurora / solarflare (the cheapest palette): 102 / 90 us with nine loads behind tests a pixel,
// 51 / 41 us as here.  Four pixels of a row to a thread (18 loads, but 32 bytes apart across the warp) cost 14 / 17 us more,
// tests for the rows that exist inside every strip's code 30, the edge's code unrolled like the strip's 4 / 5 (spills; as many
// with 3 blocks an SM).
// Solarflare, two million pixels in 32 / 8 columns: 31 / 32 us with nine loads a pixel, 117 / 432 in blocks of 256 columns of
// one strip, 20 / 21 so.
constexpr int kColorRows = 4;

template <int PALETTE>
__global__ void __launch_bounds__(kColorThreads, 4)
k_colorize(const double* __restrict__ norm, int width, long long rows, int rows_above, int rows_below,
           unsigned int* __restrict__ rgba) {
    __shared__ lyap_logtab_entry tab[LYAP_LOG_BINS];
    if (PALETTE == 1) {
        for (int e = threadIdx.y * blockDim.x + threadIdx.x; e < LYAP_LOG_BINS; e += blockDim.x * blockDim.y) tab[e] = g_lyap_logtab[e];
        __syncthreads();
    }
    const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= width) return;
    const long long step = (long long)gridDim.y * blockDim.y * kColorRows;
    for (long long y0 = ((long long)blockIdx.y * blockDim.y + threadIdx.y) * kColorRows; y0 < rows; y0 += step) {
        const double* at = norm + (y0 - 1) * width + x;   // in the row above: read only if that exists
        const bool whole = (y0 > 0 || rows_above) && (y0 + kColorRows < rows || (y0 + kColorRows == rows && rows_below));
        unsigned int* out = rgba + y0 * width + x;
        if (__all_sync(__activemask(), whole && x > 0 && x < width - 1)) {
            double v[kColorRows + 2][3];
#pragma unroll
            for (int r = 0; r < kColorRows + 2; ++r) {
#pragma unroll
                for (int k = 0; k < 3; ++k) v[r][k] = at[k - 1];
                at += width;
            }
#pragma unroll
            for (int r = 0; r < kColorRows; ++r) {
                *out = colorize_inner<PALETTE>(v[r], v[r + 1], v[r + 2], 9.0, c_col.recip[9], tab);
                out += width;
            }
        } else {
            const bool left = x > 0, right = x < width - 1;
            const int columns = 1 + left + right, there = (int)min(rows - y0, (long long)kColorRows);
            const int first = y0 > 0 || rows_above ? 0 : 1, last = y0 + there < rows || rows_below ? there + 1 : there;
            double w[3][3];   // the rows above, at and below the pixel
            const auto load = [&](int r, double (&q)[3]) {
                const bool row = r >= first && r <= last;
                q[0] = row && left ? at[-1] : -0.0;
                q[1] = row ? at[0] : -0.0;
                q[2] = row && right ? at[1] : -0.0;
                at += width;
            };
            load(0, w[0]);
            load(1, w[1]);
#pragma unroll 1
            for (int r = 0; r < there; ++r) {
                load(r + 2, w[2]);
                const int count = columns * (1 + (r >= first) + (r + 2 <= last));
                *out = colorize_inner<PALETTE>(w[0], w[1], w[2], (double)count, c_col.recip[count], tab);
                out += width;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    w[0][k] = w[1][k];
                    w[1][k] = w[2][k];
                }
            }
        }
    }
}

cudaError_t launch_colorize(const double* norm, int width, long long rows, int rows_above, int rows_below,
                            int palette, unsigned char* rgba, int sm_count, cudaStream_t st) {
    const long long n = rows * (long long)width;
    if (n <= 0) return cudaSuccess;
    const dim3 block = column_block(width, kColorThreads);
    const long long strips = (rows + kColorRows - 1) / kColorRows, high = (strips + block.y - 1) / block.y;
    const dim3 grid((unsigned)((width + block.x - 1LL) / block.x), (unsigned)(high < 65535 ? high : 65535));
    auto kern = k_colorize<0>;
    switch (palette) {
        case 1: kern = k_colorize<1>; break;
        case 2: kern = k_colorize<2>; break;
        case 3: kern = k_colorize<3>; break;
        case 4: kern = k_colorize<4>; break;
        case 5: kern = k_colorize<5>; break;
        case 6: kern = k_colorize<6>; break;
        default: break;
    }
    kern<<<grid, block, 0, st>>>(norm, width, rows, rows_above, rows_below, reinterpret_cast<unsigned int*>(rgba));
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Glow (web/fractal_renderer.js:313-334): the canvas drawn onto itself three times with 'screen' compositing,
// blur(6px) at alpha 0.3, blur(2px) at alpha 0.4, unfiltered at alpha 0.1.  The browser's compositor defines
// the exact arithmetic in the reference; these kernels implement this project's reading of the Canvas / CSS
// rules (stated in full beside oracle_glow in the CPU checker): Gaussian truncated at ceil(3 sigma),
// transparent black outside, opaque backdrop, out = Cb + alpha * Sp * (1 - Cb), 8-bit rounding per draw.
// ---------------------------------------------------------------------------------------------
constexpr int kGlowMaxRadius = 18;
struct GlowArgs {
    double w[2 * kGlowMaxRadius + 1];
    double alpha, last_alpha;   // last_alpha: of a draw without a blur on top of this one, 0 for none
};

// A blur is bound by its 2 (2R + 1) fp64 operations a channel and direction, which the arithmetic's definition fixes (a product
// and a sum per tap, in order).  So that nothing else is issued, a thread computes several neighbouring outputs of one
// channel along the blur's direction: an input is read once for all of them, and the weights, whose places are then known
// when the code is compiled, are constant-memory operands.  A tap outside the picture adds nothing; here it adds w * 0,
// which leaves a sum that is not negative as it is.  1920 x 1080, all three draws: 303 us with an output a thread, its
// taps behind tests and the canvas looked up per tap; 149 us so (fp64 alone: 69).  8 columns' outputs a thread with at
// most 128 registers; without that limit 175 us, 6 outputs 155, 12 outputs 171.
// Pictures of which a block's row or strip would be half empty have several to a block, once they have rows enough for all
// SMs (the instance for one has the block's shape as a constant: 1920 x 1080 in 147 us, with the other 152).  Two million pixels
// in 32 / 8 / 1 columns: 303 / 266 / 258 us with an output a thread, 546 / 1890 / 14160 in blocks of one row, 175 / 164 / 207 so.
constexpr int kGlowRowOut = 9;                      // odd: 9 outputs a thread put the lanes' inputs in different banks
constexpr int kGlowRowThreads = 96;                 // 32 threads a channel
constexpr int kGlowColOut = 8, kGlowColThreads = 128;
constexpr int kGlowTall = 2048;

// some_lanes: those of each channel's 32 that work on one row, if the block has several
template <int R, bool kOneRow>
__global__ void __launch_bounds__(kGlowRowThreads)
k_glow_blur_rows(const __grid_constant__ GlowArgs g, const unsigned char* __restrict__ canvas, int width, int height, int some_lanes,
                 double* __restrict__ tmp) {
    extern __shared__ double in_all[];   // of each channel, of each row: the outputs' inputs and R more on either side
    __shared__ double unit[256];
    for (int i = threadIdx.x; i < 256; i += kGlowRowThreads) unit[i] = __ddiv_rn((double)i, 255.0);
    constexpr int kOut = kGlowRowOut;
    const int lanes = kOneRow ? 32 : some_lanes, rows = 32 / lanes, columns = lanes * kOut, pitch = columns + 2 * R, inputs = rows * pitch;
    const long long x0 = (long long)blockIdx.x * columns;
    const int channel = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lane_row = lane / lanes, lane_column = (lane - lane_row * lanes) * kOut;
    const bool idle = lane_row >= rows;   // 32 is no multiple of every number of lanes
    double* in = in_all + channel * inputs;
    const long long plane = (long long)width * height;
    for (long long y0 = (long long)blockIdx.y * rows; y0 < height; y0 += (long long)gridDim.y * rows) {
        __syncthreads();
        for (int i = threadIdx.x; i < inputs; i += kGlowRowThreads) {
            const int r = rows > 1 ? i / pitch : 0;
            const long long x = x0 + (i - r * pitch) - R, y = y0 + r;
            const bool inside = x >= 0 && x < width && y < height;
            const uchar4 c = inside ? reinterpret_cast<const uchar4*>(canvas)[y * width + x] : make_uchar4(0, 0, 0, 0);   // unit[0] is 0
            in_all[i] = unit[c.x];
            in_all[i + inputs] = unit[c.y];
            in_all[i + 2 * inputs] = unit[c.z];
        }
        __syncthreads();
        double s[kOut];
#pragma unroll
        for (int o = 0; o < kOut; ++o) s[o] = 0.0;
        double* at = in + (idle ? 0 : lane_row * pitch + lane_column);
#pragma unroll
        for (int j = 0; j < kOut + 2 * R; ++j) {
            const double v = at[j];
#pragma unroll
            for (int o = 0; o < kOut; ++o)
                if (j >= o && j <= o + 2 * R) s[o] = __dadd_rn(s[o], __dmul_rn(g.w[j - o], v));
        }
        __syncthreads();   // all inputs are read: the outputs take their place, to be written in order
        if (!idle) {
#pragma unroll
            for (int o = 0; o < kOut; ++o) at[o] = s[o];
        }
        __syncwarp();      // a warp writes its own channel
        const int there = (int)min((long long)columns, width - x0), n = (int)min((long long)rows, height - y0) * there;
        double* out = tmp + channel * plane + y0 * width + x0;   // several rows are whole ones
        for (int i = lane; i < n; i += 32) {
            const int r = rows > 1 ? i / there : 0;
            out[i] = in[r * pitch + (i - r * there)];
        }
    }
}

// The rows' blur of a picture of at most kGlowNarrow columns: few taps are inside it, and a lane's outputs would be more than
// it has.
constexpr int kGlowNarrow = 8;
template <int R>
__global__ void __launch_bounds__(kGlowColThreads)
k_glow_blur_rows_narrow(const __grid_constant__ GlowArgs g, const unsigned char* __restrict__ canvas, int width, long long n,
                        double* __restrict__ tmp) {
    __shared__ double unit[256];
    for (int i = threadIdx.x; i < 256; i += kGlowColThreads) unit[i] = __ddiv_rn((double)i, 255.0);
    __syncthreads();
    for (long long i = (long long)blockIdx.x * kGlowColThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kGlowColThreads) {
        const int x = (int)(i % width);
        const uchar4* at = reinterpret_cast<const uchar4*>(canvas) + i;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        for (int k = max(-R, -x); k <= min(R, width - 1 - x); ++k) {
            const uchar4 c = at[k];
            s0 = __dadd_rn(s0, __dmul_rn(g.w[k + R], unit[c.x]));
            s1 = __dadd_rn(s1, __dmul_rn(g.w[k + R], unit[c.y]));
            s2 = __dadd_rn(s2, __dmul_rn(g.w[k + R], unit[c.z]));
        }
        tmp[i] = s0;
        tmp[i + n] = s1;
        tmp[i + 2 * n] = s2;
    }
}

__device__ __forceinline__ unsigned glow_mix(double cb, double sp, double alpha) {
    const double out = __dadd_rn(cb, __dmul_rn(__dmul_rn(alpha, sp), __dsub_rn(1.0, cb)));
    const int q = __double2loint(__dadd_rd(__dadd_rn(__dmul_rn(out, 255.0), 0.5), 0x1.8p52));   // floor: 0 <= out < 2
    return (unsigned)max(0, min(255, q));
}

// The columns' blur of the rows' blur, mixed into the canvas; and the last draw, which needs no neighbours, on top.  kOut is
// one output a thread in a picture of at most kGlowLow rows.
constexpr int kGlowLow = 3;
template <int R, int kOut, bool kOneStrip>
__global__ void __launch_bounds__(kGlowColThreads, 4)
k_glow_blur_cols_mix(const __grid_constant__ GlowArgs g, unsigned char* __restrict__ canvas, int width, int height,
                     const double* __restrict__ tmp) {
    __shared__ double unit[256];
    const int columns = kOneStrip ? kGlowColThreads : blockDim.x, strips = kOneStrip ? 1 : blockDim.y, strip = kOneStrip ? 0 : threadIdx.y;
    for (int i = strip * columns + threadIdx.x; i < 256; i += columns * strips) unit[i] = __ddiv_rn((double)i, 255.0);
    __syncthreads();
    const long long x = (long long)blockIdx.x * columns + threadIdx.x;
    if (x >= width) return;
    const long long plane = (long long)width * height;
    const long long step = (long long)gridDim.y * strips * kOut;
    for (long long y0 = ((long long)blockIdx.y * strips + strip) * kOut; y0 < height; y0 += step) {
        // input row j of this strip is the picture's row y0 + j - R
        const int first = y0 < R ? R - (int)y0 : 0, left = (int)min((long long)kOut + R, height - y0), last = left + R;
        unsigned* out = reinterpret_cast<unsigned*>(canvas) + y0 * width + x;
        unsigned px[kOut], mixed[kOut];
#pragma unroll
        for (int o = 0; o < kOut; ++o) {
            px[o] = o < left ? out[(long long)o * width] : 0u;
            mixed[o] = px[o] & 0xFF000000u;
        }
#pragma unroll 1
        for (int channel = 0; channel < 3; ++channel) {
            const double* at = tmp + channel * plane + (y0 - R) * width + x;   // read from row j == first on
            double s[kOut];
#pragma unroll
            for (int o = 0; o < kOut; ++o) s[o] = 0.0;
            if (kOut == 1) {   // a low picture: few taps are inside it
                at += (long long)first * width;
                for (int j = first; j < last; ++j, at += width) s[0] = __dadd_rn(s[0], __dmul_rn(g.w[j], *at));
            }
#pragma unroll
            for (int j = 0; kOut > 1 && j < kOut + 2 * R; ++j) {
                const double v = j >= first && j < last ? *at : 0.0;
                at += width;
#pragma unroll
                for (int o = 0; o < kOut; ++o)
                    if (j >= o && j <= o + 2 * R) s[o] = __dadd_rn(s[o], __dmul_rn(g.w[j - o], v));
            }
#pragma unroll
            for (int o = 0; o < kOut; ++o) {
                unsigned q = glow_mix(unit[(px[o] >> (8 * channel)) & 255u], s[o], g.alpha);
                if (g.last_alpha != 0.0) q = glow_mix(unit[q], unit[q], g.last_alpha);
                mixed[o] |= q << (8 * channel);
            }
        }
#pragma unroll
        for (int o = 0; o < kOut; ++o)
            if (o < left) out[(long long)o * width] = mixed[o];
    }
}

template <int R>
static cudaError_t launch_glow_blur(double sigma, double alpha, double last_alpha, unsigned char* canvas, int width, int height,
                                    double* scratch, cudaStream_t st) {
    GlowArgs g{};
    g.alpha = alpha;
    g.last_alpha = last_alpha;
    double sum = 0.0;
    for (int k = -R; k <= R; ++k) {
        g.w[k + R] = lyap_exp(-(double)(k * k) / (2.0 * sigma * sigma));
        sum += g.w[k + R];
    }
    for (int k = 0; k <= 2 * R; ++k) g.w[k] /= sum;
    if (width <= kGlowNarrow) {
        const long long n = (long long)width * height, blocks = (n + kGlowColThreads - 1) / kGlowColThreads;
        k_glow_blur_rows_narrow<R><<<(unsigned)min(blocks, 1LL << 20), kGlowColThreads, 0, st>>>(g, canvas, width, n, scratch);
    } else {
        const int needed = (width - 1) / kGlowRowOut + 1, lanes = needed <= 16 && height > kGlowTall ? needed : 32;
        const int across = (int)(((long long)width + lanes * kGlowRowOut - 1) / (lanes * kGlowRowOut)), high = 32 / lanes;
        const size_t smem = 3 * sizeof(double) * high * (lanes * kGlowRowOut + 2 * R);   // at most 34.6 KB
        const dim3 grid((unsigned)across, (unsigned)min((height - 1) / high + 1, 65535));
        auto kern = lanes == 32 ? k_glow_blur_rows<R, true> : k_glow_blur_rows<R, false>;
        kern<<<grid, kGlowRowThreads, smem, st>>>(g, canvas, width, height, lanes, scratch);
    }
    if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
    const int out = height <= kGlowLow ? 1 : kGlowColOut;
    const dim3 block = height > kGlowTall ? column_block(width, kGlowColThreads) : dim3(kGlowColThreads, 1);
    const long long strips = ((long long)height + out - 1) / out, high = (strips + block.y - 1) / block.y;
    const dim3 grid((unsigned)((width + block.x - 1LL) / block.x), (unsigned)(high < 65535 ? high : 65535));
    auto kern = out == 1 ? k_glow_blur_cols_mix<R, 1, true>
                         : (block.x == kGlowColThreads ? k_glow_blur_cols_mix<R, kGlowColOut, true> : k_glow_blur_cols_mix<R, kGlowColOut, false>);
    kern<<<grid, block, 0, st>>>(g, canvas, width, height, scratch);
    return cudaGetLastError();
}

cudaError_t launch_glow(unsigned char* canvas, int width, int height, double* scratch, cudaStream_t st) {
    // radius ceil(3 sigma); the third draw (alpha 0.1, no blur) rides on the second
    if (cudaError_t e = launch_glow_blur<18>(6.0, 0.3, 0.0, canvas, width, height, scratch, st); e != cudaSuccess) return e;
    return launch_glow_blur<6>(2.0, 0.4, 0.1, canvas, width, height, scratch, st);
}

// ---------------------------------------------------------------------------------------------
// Pipe issue-rate micro-benchmarks: 8 independent FMA chains per thread, nothing else in the loop.
// ---------------------------------------------------------------------------------------------
constexpr int kPeakThreads = 512;
constexpr int kPeakChains = 8;
constexpr int kPeakInner = 64;

__global__ void __launch_bounds__(kPeakThreads) k_fp64_peak(double* sink, int iters) {
    double acc[kPeakChains];
#pragma unroll
    for (int c = 0; c < kPeakChains; ++c) acc[c] = 1.0 + 1e-9 * (threadIdx.x + c);
    const double m = 0.999999, k = 1e-7;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int u = 0; u < kPeakInner; ++u) {
#pragma unroll
            for (int c = 0; c < kPeakChains; ++c) acc[c] = __fma_rn(acc[c], m, k);
        }
    }
    double s = 0;
#pragma unroll
    for (int c = 0; c < kPeakChains; ++c) s += acc[c];
    if (s == 12345.678) sink[0] = s;
}

__global__ void __launch_bounds__(kPeakThreads) k_fp32_peak(float* sink, int iters) {
    float acc[kPeakChains];
#pragma unroll
    for (int c = 0; c < kPeakChains; ++c) acc[c] = 1.0f + 1e-6f * (threadIdx.x + c);
    const float m = 0.9999f, k = 1e-5f;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int u = 0; u < kPeakInner; ++u) {
#pragma unroll
            for (int c = 0; c < kPeakChains; ++c) acc[c] = __fmaf_rn(acc[c], m, k);
        }
    }
    float s = 0;
#pragma unroll
    for (int c = 0; c < kPeakChains; ++c) s += acc[c];
    if (s == 12345.678f) sink[0] = s;
}

cudaError_t launch_fp64_peak(double* sink, int sm_count, int iters, unsigned long long* instr, cudaStream_t st) {
    const int grid = sm_count * 2;
    k_fp64_peak<<<grid, kPeakThreads, 0, st>>>(sink, iters);
    *instr = (unsigned long long)grid * kPeakThreads * kPeakChains * kPeakInner * (unsigned long long)iters;
    return cudaGetLastError();
}

cudaError_t launch_fp32_peak(float* sink, int sm_count, int iters, unsigned long long* instr, cudaStream_t st) {
    const int grid = sm_count * 4;
    k_fp32_peak<<<grid, kPeakThreads, 0, st>>>(sink, iters);
    *instr = (unsigned long long)grid * kPeakThreads * kPeakChains * kPeakInner * (unsigned long long)iters;
    return cudaGetLastError();
}

}  // namespace lyap

namespace lyap {

template <typename FL, int P>
static cudaError_t launch_lambda_fast_t(const LambdaArgs& a, double* out64, float* out32, unsigned long long* steps, cudaStream_t st, int kind, int spec_ppt, int spec_threads,
                                        const char* generic_name) {
    if (a.n_pixels <= 0) return cudaSuccess;
    // one tile of 32 * pixels a warp: blocks are many and small, so that the tiles, some of which take a tenth of others'
    // time, are dealt out as SMs have room
    const auto grid = [&](int pixels, int threads) {
        const long long rows = a.n_pixels / a.width;   // the larger of the two ways to cut a frame (see lambda_fast_body)
        const long long positions = std::max((rows + pixels - 1) / pixels * a.width, (a.n_pixels + pixels - 1) / pixels);
        return (unsigned)((positions + threads - 1) / threads);
    };
    {   // a periodic sequence can run an instance made for its patterns (same switches as the exact kernel)
        bool launched = false;
        const cudaError_t e = launch_lambda_spec(a, out64, out32, steps, grid(spec_ppt, spec_threads), st, kind, spec_ppt, spec_threads, 0,
                                                 spec_mode(), &launched);
        if (e != cudaSuccess || launched) return e;
    }
    k_lambda_fast<FL, P, kFastThreads><<<grid(P, kFastThreads), kFastThreads, 0, st>>>(a, out64, out32, steps);
    note_lambda_kernel(generic_name);
    return cudaGetLastError();
}

// Two pixels a thread, which come into cycles together more often than more do and leave registers for more warps: 2731 x 1537
// of "ABB" 150 + 1500 over [2,4]^2 in fp64 with 4 / 3 / 2 pixels 1.10 / 0.97 / 0.94 ms, 4096^2 of "AABAB" 200 + 2000 in fp32 with
// 4 / 2 pixels 3.95 / 3.40.
cudaError_t launch_lambda_fast64(const LambdaArgs& a, double* out64, float* out32, unsigned long long* steps, cudaStream_t st) {
    return launch_lambda_fast_t<FusedF64, 2>(a, out64, out32, steps, st, 1, 2, 128, "k_lambda_fast<FusedF64,2,128> (generic)");
}

cudaError_t launch_lambda_fast32(const LambdaArgs& a, double* out64, float* out32, unsigned long long* steps, cudaStream_t st) {
    return launch_lambda_fast_t<FusedF32, 2>(a, out64, out32, steps, st, 2, 2, 128, "k_lambda_fast<FusedF32,2,128> (generic)");
}

cudaError_t launch_lambda_orbit64(const LambdaArgs& a, double* out64, float* out32, unsigned long long* steps, cudaStream_t st) {
    return launch_lambda_fast_t<OrbitF64, 2>(a, out64, out32, steps, st, 3, 2, 128, "k_lambda_fast<OrbitF64,2,128> (generic)");
}

}  // namespace lyap
