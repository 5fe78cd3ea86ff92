// Common definitions for the batch ODE integrator device code.
//
// Compiled at run time by NVRTC for sm_100a together with a generated
// system struct and a generated configuration struct (see
// cubie_b200/kernelgen.py).  Everything here is header-only device code.
#pragma once

// Functions whose body is large and called from many places (the class-
// grouped right-hand side and J v of the warp layout) are kept as one copy:
// inlined at every call site of every unrolled stage they multiplied the
// kernel's code size until instruction fetch, not arithmetic, bounded it.
#ifdef CBX_HOST_EMULATION
#define CBX_NOINLINE __attribute__((noinline))
#else
#define CBX_NOINLINE __noinline__
#endif

namespace cbx {

// Per-run status bits; values match the reference's CUBIE_RESULT_CODES
// (src/cubie/result_codes.py:50-58).
enum Status : int {
    SUCCESS = 0,
    MAX_NEWTON_ITERATIONS_EXCEEDED = 2,
    MAX_LINEAR_ITERATIONS_EXCEEDED = 4,
    STEP_TOO_SMALL = 8,
    DT_EFF_EFFECTIVELY_ZERO = 16,
    MAX_LOOP_ITERS_EXCEEDED = 32,
    STAGNATION = 64,
    BICGSTAB_BREAKDOWN = 128,
    NEWTON_DIVERGENCE = 256,
};

// Algorithm families and linear solvers selected by the configuration.
enum Algo : int { ALGO_ERK = 0, ALGO_DIRK = 1, ALGO_FIRK = 2, ALGO_ROSENBROCK = 3 };
enum Lin : int { LIN_MR = 0, LIN_SD = 1, LIN_BICGSTAB = 2, LIN_GMRES = 3, LIN_DIRECT = 4 };
enum Ctrl : int { CTRL_FIXED = 0, CTRL_I = 1, CTRL_PI = 2, CTRL_PID = 3, CTRL_GUSTAFSSON = 4 };

// Python's max/min semantics for two arguments (the reference uses the
// Python builtins, which keep the first argument unless the second is
// strictly larger/smaller; this decides NaN propagation).
template <class T> __device__ __forceinline__ T pymax(T a, T b) { return (b > a) ? b : a; }
template <class T> __device__ __forceinline__ T pymin(T a, T b) { return (b < a) ? b : a; }

// |v| (a free operand modifier on the device).
__device__ __forceinline__ float absv(float v) { return fabsf(v); }
__device__ __forceinline__ double absv(double v) { return fabs(v); }

// max and min in one instruction, NaN when either operand is one.  They equal
// pymax / pymin wherever a NaN can only come first (or comes in both), which
// is a compare and a select otherwise.
template <class T> __device__ __forceinline__ T max_nan(T a, T b) { return (b > a) ? b : a; }
template <class T> __device__ __forceinline__ T min_nan(T a, T b) { return (b < a) ? b : a; }
#ifndef CBX_HOST_EMULATION
template <> __device__ __forceinline__ float max_nan<float>(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
template <> __device__ __forceinline__ float min_nan<float>(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
#endif

// v clamped to [lo, hi]; lo for a NaN.
template <class T> __device__ __forceinline__ T clampv(T v, T lo, T hi) { return pymax(lo, pymin(v, hi)); }
#ifndef CBX_HOST_EMULATION
template <> __device__ __forceinline__ float clampv<float>(float v, float lo, float hi) {
    return fmaxf(lo, min_nan(v, hi));   // fmaxf drops the NaN
}
#endif

// A round-to-nearest add the compiler never fuses with the multiply that
// produced an operand.  Used where a value crosses from the step function
// into the loop's state update: whether an FMA forms there otherwise depends
// on the surrounding control flow, and the adjoint's replay must reproduce
// the forward bit for bit from different surroundings.
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

// Type selection (A when B holds, else Bt) without the standard library,
// which NVRTC does not provide.
template <bool B, class A, class Bt> struct Pick { using type = A; };
template <class A, class Bt> struct Pick<false, A, Bt> { using type = Bt; };

__device__ __forceinline__ bool is_finite(float v) { return isfinite(v); }
__device__ __forceinline__ bool is_finite(double v) { return isfinite(v); }
__device__ __forceinline__ bool is_nan(float v) { return isnan(v); }
__device__ __forceinline__ bool is_nan(double v) { return isnan(v); }

__device__ __forceinline__ float sqrt_t(float v) { return sqrtf(v); }
__device__ __forceinline__ double sqrt_t(double v) { return sqrt(v); }
__device__ __forceinline__ float pow_t(float a, float b) { return powf(a, b); }
__device__ __forceinline__ float log2_t(float a) { return log2f(a); }
__device__ __forceinline__ double log2_t(double a) { return log2(a); }
__device__ __forceinline__ float exp2_t(float a) { return exp2f(a); }
__device__ __forceinline__ double exp2_t(double a) { return exp2(a); }

// e / tol of the norms.  In FP64 on the device: the hardware's approximate
// reciprocal refined by two Newton iterations, then the quotient corrected by
// its residual (Markstein, Computation of elementary functions on the IBM RISC
// System/6000, IBM J. Res. Dev. 34, 1990), without the general division's
// scaling; where that leaves the finite numbers (a zero or infinite tolerance,
// an infinite or NaN term, an overflow) the product with the unrefined
// reciprocal is the division's value.  For every term and tolerance of the
// norms it has the division's bits (tests/test_ratio_gpu.py); tolerances below
// 2^-1022 count as zero and those above 2^1021 as infinite.  Divisions were
// what the FP64 norms cost: Tsit5, 50,021 Lorenz runs 949 -> 908 us; ROS3P,
// 20,001 Van der Pol runs 1.85 -> 1.62 ms; Radau IIA5 with GMRES, 10,001 runs
// 7.04 -> 6.13 ms.
__device__ __forceinline__ float ratio_t(float e, float tol) { return e / tol; }
__device__ __forceinline__ double ratio_t(double e, double tol) {
#ifdef CBX_HOST_EMULATION
    return e / tol;
#else
    double r0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(tol));
    double r = fma(r0, fma(-tol, r0, 1.0), r0);
    r = fma(r, fma(-tol, r, 1.0), r);
    const double q = e * r;
    const double corrected = fma(r, fma(-tol, q, e), q);
    return is_finite(corrected) ? corrected : e * r0;
#endif
}

#ifdef CBX_HOST_EMULATION
__device__ __forceinline__ double pow_t(double a, double b) { return pow(a, b); }
#else
// The FP64 controllers' powers of error norms and step ratios.  pow carries
// its logarithm to twice the precision, because log2 a has its exponent's
// size and b log2 a loses that many bits to it.  Here a = 2^k m with m in
// [1, 2): b k is formed exactly for b rounded to a multiple of 2^-40, its
// integer part becomes the result's exponent, and log2 m, the remainder of b
// and the fraction are a few units at most, so the result is about as close as
// pow's (tests/test_gain_powers_gpu.py) at half its instructions: with pow and
// the division in the norms Tsit5 on 50,021 Lorenz runs took 1,233 us, ROS3P on
// 20,001 Van der Pol runs 2,280, now 917 and 1,641.  Finite
// a >= 0 (the controllers map other norms to 1e16); zero and subnormal a count
// as 2^-1023 and infinity as 2^1024, whose powers lie beyond a gain's clamp.
struct Log2Parts {
    double k, m;      // a = 2^k 2^m, 0 <= m <= 1
    __device__ __forceinline__ explicit Log2Parts(double a) {
        const int hi = __double2hiint(a);
        k = double((hi >> 20) - 1023);
        m = log2(__hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(a)));
    }
};
// b to a multiple of 2^-40 (its product with an exponent is exact)
__device__ __forceinline__ double coarse(double b) { return (b + 0x1.8p12) - 0x1.8p12; }
// c 2^(whole + rest): ``whole`` a multiple of 2^-40, ``rest`` a few units.  What
// their sum's rounding loses multiplies the result.
__device__ __forceinline__ double scaled_exp2(double c, double whole, double rest) {
    const double shifted = whole + 0x1.8p52;               // rounds to an integer
    const double fraction = whole - (shifted - 0x1.8p52);
    const double f = fraction + rest;
    const double lost = (fraction - f) + rest;
    int n = __double2loint(shifted);
    n = n < -1022 ? -1022 : (n > 1023 ? 1023 : n);         // far outside any gain's clamp
    const double e = exp2(f);
    return c * fma(e, lost * 0.69314718055994531, e) * __hiloint2double((n + 1023) << 20, 0);
}
__device__ __forceinline__ double pow_t(double a, double b) {
    const Log2Parts l(a);
    const double bh = coarse(b);
    return scaled_exp2(1.0, bh * l.k, fma(b, l.m, (b - bh) * l.k));
}
#endif

// c a^x b^y for a, b > 0.  In FP64 on the device one exponential serves both
// powers; in FP32 the two approximate powers side by side have the shorter
// chain.
__device__ __forceinline__ float scaled_powers(float c, float a, float x, float b, float y) {
    return c * pow_t(a, x) * pow_t(b, y);
}
__device__ __forceinline__ double scaled_powers(double c, double a, double x, double b, double y) {
#ifndef CBX_HOST_EMULATION
    const Log2Parts la(a), lb(b);
    const double xh = coarse(x), yh = coarse(y);
    return scaled_exp2(c, xh * la.k + yh * lb.k,
                       fma(x, la.m, fma(y, lb.m, fma(x - xh, la.k, (y - yh) * lb.k))));
#else
    return c * pow_t(a, x) * pow_t(b, y);
#endif
}

template <class T> struct Limits;
template <> struct Limits<float> {
    static __device__ __forceinline__ float huge() { return 3.4028234663852886e38f; }
    static __device__ __forceinline__ float eps() { return 1.1920928955078125e-07f; }
};
template <> struct Limits<double> {
    static __device__ __forceinline__ double huge() { return 1.7976931348623157e308; }
    static __device__ __forceinline__ double eps() { return 2.220446049250313e-16; }
};

// Compensated (Kahan) accumulation of a sum of terms in type T.
template <class T> struct Kahan {
    T sum, comp;
    __device__ __forceinline__ Kahan() : sum(T(0)), comp(T(0)) {}
    __device__ __forceinline__ void add(T term) {
        T y = term - comp;
        T s = sum + y;
        comp = (s - sum) - y;
        sum = s;
    }
};

}  // namespace cbx
