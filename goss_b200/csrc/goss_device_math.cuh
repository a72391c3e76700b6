// Scalar math used by the generated model code and the solver kernels.
//
// Every function has a float and a double overload.  The double overloads
// call CUDA's double-precision functions, those of models::F64 below are
// branch-free (the FP64 paths are checked state for state against the FP64 CPU
// oracle).  The float overloads
// map to the SFU approximations (ex2/lg2/rcp/rsqrt based intrinsics) that make
// the FP32 path fast; its accuracy is checked against FP64 in the tests.
#ifndef GOSS_DEVICE_MATH_CUH
#define GOSS_DEVICE_MATH_CUH

#include <cuda_runtime.h>
#include <math.h>

namespace goss_b200 { namespace models {

__device__ __forceinline__ double gexp(double x) { return exp(x); }
__device__ __forceinline__ float gexp(float x) { return __expf(x); }
// 2^x: the hardware exponential (ex2.approx, flush-to-zero, as __expf uses) in
// FP32; exp2 in FP64.  The generator prints exp(c*x) as gexp2((c*log2 e)*x).
__device__ __forceinline__ double gexp2(double x) { return exp2(x); }
__device__ __forceinline__ float gexp2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ double glog(double x) { return log(x); }
__device__ __forceinline__ float glog(float x) { return __logf(x); }
__device__ __forceinline__ double gsqrt(double x) { return ::sqrt(x); }
__device__ __forceinline__ float gsqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double gfabs(double x) { return fabs(x); }
__device__ __forceinline__ float gfabs(float x) { return fabsf(x); }
__device__ __forceinline__ double gfloor(double x) { return floor(x); }
__device__ __forceinline__ float gfloor(float x) { return floorf(x); }
__device__ __forceinline__ double gceil(double x) { return ceil(x); }
__device__ __forceinline__ float gceil(float x) { return ceilf(x); }
__device__ __forceinline__ double gpow(double x, double y) { return pow(x, y); }
__device__ __forceinline__ float gpow(float x, float y) { return __powf(x, y); }
__device__ __forceinline__ double gfmax(double x, double y) { return fmax(x, y); }
__device__ __forceinline__ float gfmax(float x, float y) { return fmaxf(x, y); }
__device__ __forceinline__ double gfmin(double x, double y) { return fmin(x, y); }
__device__ __forceinline__ float gfmin(float x, float y) { return fminf(x, y); }
__device__ __forceinline__ double gsin(double x) { return sin(x); }
__device__ __forceinline__ float gsin(float x) { return __sinf(x); }
__device__ __forceinline__ double gcos(double x) { return cos(x); }
__device__ __forceinline__ float gcos(float x) { return __cosf(x); }
__device__ __forceinline__ double gtan(double x) { return tan(x); }
__device__ __forceinline__ float gtan(float x) { return __tanf(x); }
__device__ __forceinline__ double gtanh(double x) { return tanh(x); }
__device__ __forceinline__ float gtanh(float x) { return tanhf(x); }

// ---------------------------------------------------------------------------
// FP64 scalar functions of the split model programs
// ---------------------------------------------------------------------------
// CUDA's double-precision division, sqrt, exp and log each end in a rarely
// taken branch, so a model evaluation with ~65 reciprocals and ~50
// exponentials becomes a chain of short basic blocks whose dependent FP64
// instructions are not interleaved: ncu measured the FP64 pipe at 24-44 % of
// its rate, every warp waiting on its own previous instruction.  The functions
// below have no branch, so the scheduler overlaps as many of them as the
// registers allow, and the reciprocals of one denominator are shared.
// Measured (TP06 with four fields, 262,144 nodes): RK4 x 50 steps 9.81 -> 6.36
// ms, ExplicitEuler x 100 steps 4.07 -> 2.71 ms.
//
// Zeros, infinities and NaN give what IEEE arithmetic gives, by integer
// operations on the exponent bits.  At the ends of the range results saturate
// early: reciprocals of subnormal numbers are infinite (as nearly all of them
// are), those of numbers from 2^1022 on are 0, and 2^t is infinite from
// t = 1023.5 and 0 below t = -1022.5.

__device__ __forceinline__ double f64_make(int hi, int lo) { return __hiloint2double(hi, lo); }

// true when v is neither zero, subnormal, infinite nor NaN
__device__ __forceinline__ bool f64_normal(double v)
{
    return ((unsigned)__double2hiint(v) << 1) - 0x00200000u < 0xffc00000u;
}

// 1/x: the hardware's 20-bit estimate r0 and one third-order step
// r0 (1 + e + e^2), e = 1 - x r0 (Householder's method; e is one rounded FMA):
// truncation e^3 < 2^-60, so the error is the last rounding's half ulp.
// |e| < 2^-19 has the top exponent bit clear; where r0 is 0 or infinite e is
// NaN or -infinity, and clearing that bit (and setting the last one, so that
// -infinity becomes -1 - 2^-52) makes e + e^2 a positive number, which leaves
// r0 as it is.
__device__ __forceinline__ double f64_rcp(double x)
{
    double r0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(x));
    const double d = fma(-x, r0, 1.0);
    const double e = f64_make(__double2hiint(d) & 0xbfffffff, __double2loint(d) | 1);
    return fma(r0, fma(e, e, e), r0);
}

// a/b from b's reciprocal with one residual correction (Markstein 1990)
__device__ __forceinline__ double f64_div(double a, double b)
{
    const double r = f64_rcp(b);
    const double q = a * r;
    const double c = fma(fma(-b, q, a), r, q);
    return f64_normal(q) ? c : q;
}

// sqrt(x): the hardware's reciprocal square root, one coupled step on
// g ~ sqrt(x) and h ~ 1/(2 sqrt(x)) (Goldschmidt) and a residual correction;
// subnormal operands scaled by 2^54
__device__ __forceinline__ double f64_sqrt(double x)
{
    const bool tiny = __double2hiint(x) < 0x00100000 && x > 0.0;
    const double xs = tiny ? x * 0x1p54 : x;
    double r0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(xs));
    double g = xs * r0, h = 0.5 * r0;
    const double e = fma(-g, h, 0.5);
    g = fma(g, e, g);
    h = fma(h, e, h);
    g = fma(fma(-g, g, xs), h, g);
    const double special = x >= 0.0 ? x : f64_make(0x7ff80000, 0);  // +-0, +inf; negative, NaN
    return f64_normal(r0) ? (tiny ? g * 0x1p-27 : g) : special;
}

// log(x): x = 2^k m with m in [sqrt(1/2), sqrt(2)), log m = 2 atanh(s) with
// s = (m - 1)/(m + 1), whose rounding error is carried along; the series in
// s^2 as a minimax polynomial of degree 6 (Remez exchange, 1.2e-18), k ln 2 in
// two parts
__device__ __forceinline__ double f64_log(double x)
{
    const bool tiny = __double2hiint(x) < 0x00100000 && x > 0.0;  // subnormal
    const double xs = tiny ? x * 0x1p54 : x;
    const int hx = __double2hiint(xs);
    const int k = (hx - 0x3fe6a09e) >> 20;
    const double m = f64_make(hx - (k << 20), __double2loint(xs));
    const double kd = f64_make(0x43300000, (k - (tiny ? 54 : 0)) ^ 0x80000000) - (0x1p52 + 0x1p31);
    const double f = m - 1.0, d = m + 1.0;
    const double r = f64_rcp(d);
    const double s = f * r;
    const double s_lo = fma(-s, m - (d - 1.0), fma(-s, d, f)) * r;
    const double z = s * s, w = z * z;
    double a = 0x1.2f0113766d435p-3, b = 0x1.39a22b5279601p-3;
    a = fma(a, w, 0x1.74663a6ada14fp-3);
    b = fma(b, w, 0x1.c71c521fe9f3dp-3);
    a = fma(a, w, 0x1.24924941d4850p-2);
    b = fma(b, w, 0x1.999999997ffcep-2);
    a = fma(a, w, 0x1.5555555555592p-1);
    const double t = fma(s * z, fma(b, z, a), fma(kd, 0x1.a39ef35793c76p-33, 2.0 * s_lo));
    const double y = fma(kd, 0x1.62e42fee00000p-1, fma(2.0, s, t));
    const double special = x > 0.0 ? x : (x == 0.0 ? f64_make(0xfff00000, 0) : f64_make(0x7ff80000, 0));
    return (unsigned)hx - 0x00100000u < 0x7fe00000u ? y : special;
}

// t, or +-2^20 where |t| is at least that (infinities too; NaN stays)
__device__ __forceinline__ double f64_clamp(double t)
{
    const unsigned h = (unsigned)__double2hiint(t);
    const bool far = (h << 1) - 0x82600000u <= 0x7d800000u;  // 0x41300000 <= |h| <= 0x7ff00000
    return f64_make(far ? (h & 0x80000000u) | 0x41300000u : h, __double2loint(t));
}

// 1.5 * 2^52 + 1023: v + kRoundBias has round(v) + 1023, the exponent field of
// 2^round(v), in its low word
constexpr double kRoundBias = 6755399441055744.0 + 1023.0;

// p * 2^n from the low word n + 1023 (one saturating min/max: infinity, 0)
__device__ __forceinline__ double f64_scale(double p, int biased)
{
    return p * f64_make(__vimin_s32_relu(biased, 0x7ff) << 20, 0);
}

// 2^t = 2^n * 2^f, n the nearest integer, f in [-1/2, 1/2];
// 2^f = 1 + f q(f) with q the minimax polynomial of degree 10 of (2^f - 1)/f
// (Remez exchange, relative error 1.8e-17), the terms above the constant split
// into even and odd ones (half the chain of a Horner form for one more multiply)
__device__ __forceinline__ double f64_exp2(double x)
{
    const double t = f64_clamp(x);
    const double m = t + kRoundBias;
    const double f = t - (m - kRoundBias);
    const double g = f * f;
    double a = 0x1.e605d246f3c56p-28, b = 0x1.e8cabfafcc3e1p-32;
    a = fma(a, g, 0x1.62bfd4b4d28e0p-20);
    b = fma(b, g, 0x1.b525a08e76058p-24);
    a = fma(a, g, 0x1.4309130958dadp-13);
    b = fma(b, g, 0x1.ffcbfc1ea57a5p-17);
    a = fma(a, g, 0x1.3b2ab6fba1e40p-7);
    b = fma(b, g, 0x1.5d87fe78b2115p-10);
    a = fma(a, g, 0x1.ebfbdff82c598p-3);
    b = fma(b, g, 0x1.c6b08d704a08ep-5);
    const double q = fma(fma(b, f, a), f, 0x1.62e42fefa39efp-1);
    return f64_scale(fma(f, q, 1.0), __double2loint(m));
}

// e^x = 2^n e^r, r = x - n ln 2 in two parts (Cody and Waite 1980);
// e^r = 1 + r q(r), q the minimax polynomial of degree 10 of (e^r - 1)/r
__device__ __forceinline__ double f64_exp(double y)
{
    const double x = f64_clamp(y);
    const double m = fma(x, 1.4426950408889634, kRoundBias);
    const double n = m - kRoundBias;
    const double r = fma(n, -0x1.abc9e3b39803fp-56, fma(n, -0x1.62e42fefa39efp-1, x));
    const double g = r * r;
    double a = 0x1.28a27e19fd3b5p-22, b = 0x1.ae644fe01339ep-26;
    a = fma(a, g, 0x1.a019a6b25f4ccp-16);
    b = fma(b, g, 0x1.71de8e61019f2p-19);
    a = fma(a, g, 0x1.6c16c17f29c03p-10);
    b = fma(b, g, 0x1.a01a017107b31p-13);
    a = fma(a, g, 0x1.555555555211ep-5);
    b = fma(b, g, 0x1.111111111a24bp-7);
    a = fma(a, g, 0x1.0000000000005p-1);
    b = fma(b, g, 0x1.5555555555530p-3);
    const double q = fma(fma(b, r, a), r, 1.0);
    return f64_scale(fma(r, q, 1.0), __double2loint(m));
}

// (e^x - 1)/x for |x| < 1/8: minimax polynomial of degree 8 (relative error 8e-18)
__device__ __forceinline__ double f64_phi1_small(double x)
{
    const double g = x * x;
    double a = 0x1.71de3b62d0df6p-19, b = 0x1.a0439d7707c08p-16;
    a = fma(a, g, 0x1.a01a03fd2e02cp-13);
    b = fma(b, g, 0x1.6c16bf78e5977p-10);
    a = fma(a, g, 0x1.11111110f18dep-7);
    b = fma(b, g, 0x1.5555555566a8fp-5);
    a = fma(a, g, 0x1.5555555555572p-3);
    b = fma(b, g, 0x1.ffffffffffff6p-2);
    a = fma(a, g, 1.0);
    return fma(b, x, a);
}

// The arithmetic type the split FP64 programs are instantiated with: a double
// whose division and functions are the ones above.
struct F64 {
    double v;
    F64() = default;
    __device__ __forceinline__ explicit F64(double x) : v(x) {}
    __device__ __forceinline__ F64& operator=(double x)
    {
        v = x;
        return *this;
    }
    __device__ __forceinline__ operator double() const { return v; }
    __device__ __forceinline__ F64 operator-() const { return F64(-v); }
    __device__ __forceinline__ F64& operator-=(double x)
    {
        v -= x;
        return *this;
    }
};
#define GOSS_F64_OP(op, expr)                                                                     \
    __device__ __forceinline__ F64 operator op(F64 x, F64 y) { const double a = x.v, b = y.v; return F64(expr); } \
    __device__ __forceinline__ F64 operator op(F64 x, double b) { const double a = x.v; return F64(expr); }       \
    __device__ __forceinline__ F64 operator op(double a, F64 y) { const double b = y.v; return F64(expr); }
GOSS_F64_OP(+, a + b)
GOSS_F64_OP(-, a - b)
GOSS_F64_OP(*, a * b)
GOSS_F64_OP(/, f64_div(a, b))
#undef GOSS_F64_OP

__device__ __forceinline__ F64 gexp(F64 x) { return F64(f64_exp(x.v)); }
__device__ __forceinline__ F64 gexp2(F64 x) { return F64(f64_exp2(x.v)); }
__device__ __forceinline__ F64 gsqrt(F64 x) { return F64(f64_sqrt(x.v)); }
__device__ __forceinline__ F64 glog(F64 x) { return F64(f64_log(x.v)); }
__device__ __forceinline__ F64 gfabs(F64 x) { return F64(::fabs(x.v)); }
__device__ __forceinline__ F64 gfloor(F64 x) { return F64(::floor(x.v)); }
__device__ __forceinline__ F64 gceil(F64 x) { return F64(::ceil(x.v)); }
__device__ __forceinline__ F64 gpow(F64 x, F64 y) { return F64(::pow(x.v, y.v)); }
__device__ __forceinline__ F64 gfmax(F64 x, F64 y) { return F64(::fmax(x.v, y.v)); }
__device__ __forceinline__ F64 gfmin(F64 x, F64 y) { return F64(::fmin(x.v, y.v)); }
__device__ __forceinline__ F64 gsin(F64 x) { return F64(::sin(x.v)); }
__device__ __forceinline__ F64 gcos(F64 x) { return F64(::cos(x.v)); }
__device__ __forceinline__ F64 gtan(F64 x) { return F64(::tan(x.v)); }
__device__ __forceinline__ F64 gtanh(F64 x) { return F64(::tanh(x.v)); }
// the step of the generated forward differences, delta = sqrt(1e-15 max(1e-5, |y|))
// (the host's derived constants keep the library's)
__host__ __device__ __forceinline__ double sqrt(double x)
{
#ifdef __CUDA_ARCH__
    return f64_sqrt(x);
#else
    return ::sqrt(x);
#endif
}

}}  // namespace goss_b200::models

namespace goss_b200 {

// Two FP32 numbers in one 64-bit register pair.  sm_100a adds, multiplies and
// fuses both halves with one instruction, which halves the issue slots of
// arithmetic that comes in pairs (the kernels that use it are bound by
// instruction issue); each half rounds and flushes as the scalar instruction.
struct F32x2 {
    unsigned long long v;
    F32x2() = default;
    __device__ __forceinline__ F32x2(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
    __device__ __forceinline__ explicit F32x2(float a) : F32x2(a, a) {}
    __device__ __forceinline__ void unpack(float& a, float& b) const
    {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    }
};
__device__ __forceinline__ F32x2 operator+(F32x2 a, F32x2 b)
{
    F32x2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// rounded toward zero
__device__ __forceinline__ F32x2 vadd_rz(F32x2 a, F32x2 b)
{
    F32x2 r;
    asm("add.rz.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F32x2 operator-(F32x2 a, F32x2 b)
{
    F32x2 r;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F32x2 operator*(F32x2 a, F32x2 b)
{
    F32x2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F32x2 vfma(F32x2 a, F32x2 b, F32x2 c)
{
    F32x2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }

// phi1(x) = (e^x - 1)/x with phi1(0) = 1, in single precision.
//
// The generalised Rush-Larsen update y + b/a (e^{a h} - 1) equals
// y + b h phi1(a h).  Evaluating e^{a h} - 1 in single precision cancels
// catastrophically when |a h| is small (gating variables with time constants
// of hundreds of ms at h = 0.01 ms give |a h| ~ 1e-5, leaving ~2 correct
// digits), so the FP32 kernels use phi1 instead: for |x| < 1/4 the Taylor
// series sum_k x^k/(k+1)! truncated after x^6 (relative truncation error
// < (1/4)^7/8! < 2e-9), otherwise (e^x - 1)/x with the SFU exponential.
template <typename V>
__device__ __forceinline__ V phi1f_small(V x)
{
    // Horner form of 1 + x/2 + x^2/6 + x^3/24 + x^4/120 + x^5/720 + x^6/5040
    V p = V(1.0f / 5040.0f);
    p = vfma(p, x, V(1.0f / 720.0f));
    p = vfma(p, x, V(1.0f / 120.0f));
    p = vfma(p, x, V(1.0f / 24.0f));
    p = vfma(p, x, V(1.0f / 6.0f));
    p = vfma(p, x, V(0.5f));
    return vfma(p, x, V(1.0f));
}
__device__ __forceinline__ float phi1f_large(float x) { return __fdividef(__expf(x) - 1.0f, x); }
__device__ __forceinline__ float phi1f(float x) { return fabsf(x) < 0.25f ? phi1f_small(x) : phi1f_large(x); }

}  // namespace goss_b200

#endif
