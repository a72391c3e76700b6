// sm_100a solver kernels of the multi-node solve path.
//
// One CUDA thread owns one mesh node for the whole call: its states are
// loaded once from the component-major FP64 arrays (states[i*ld + node],
// coalesced across the warp), kept in registers across every internal step
// of the interval, and stored once at the end.  Uniform model parameters
// travel in the kernel's parameter block (constant bank, read as free
// operands); per-node field parameters are loaded once into registers.
//
// Each kernel restates the arithmetic of one reference solver.  The FP64
// instantiations evaluate the model with common factors pulled out and every
// distinct exponential and reciprocal once, so they agree with the FP64 CPU
// oracle to rounding; GOSS_FP64_PRINTED keeps the reference's own order.
//
//   explicit_kernel<M, T, ExplicitEuler>  cpp/goss/ExplicitEuler.cpp:64-87
//   explicit_kernel<M, T, RK4>            cpp/goss/RK4.cpp:68-102
//   explicit_kernel<M, T, GRL1>           cpp/goss/GRL1.cpp:61-82, GRL1.h:72-84
//   explicit_kernel<M, T, GRL2>           cpp/goss/GRL2.cpp:63-86
//   theta_kernel<M>                       cpp/goss/ThetaSolver.cpp:49-155,
//                                         ImplicitODESolver.cpp:92-262, ODE.cpp:47-132
//   esdirk_kernel<M>                      cpp/goss/ESDIRK23a.cpp:101-316
#ifndef GOSS_KERNELS_CUH
#define GOSS_KERNELS_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "goss_b200.h"
#include "goss_device_math.cuh"

namespace goss_b200 {

constexpr double kGossEps = 3.0e-16;  // GOSS_EPS, cpp/goss/constants.h:25

template <class M>
struct Dims {
    static constexpr int n = M::num_states;
    // parameter block: the model parameters followed by the derived constants
    static constexpr int npd = M::num_params + M::num_derived;
    static constexpr int np = npd > 0 ? npd : 1;
    static constexpr int nfp = M::num_field_params > 0 ? M::num_field_params : 1;
};

// Fill the FP64 parameter block: parameters, then the model's derived
// constants computed from them (once per launch, on the host).
template <class M>
inline void parameter_block(const double* params, double (&out)[Dims<M>::np])
{
    for (int i = 0; i < Dims<M>::np; ++i)
        out[i] = i < M::num_params ? params[i] : 0.0;
    if (M::num_derived > 0)
        M::derived(out, out + M::num_params);
}

// std::max / std::min semantics (first argument wins ties and NaNs)
__device__ __forceinline__ double std_max(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double std_min(double a, double b) { return (b < a) ? b : a; }

// ---------------------------------------------------------------------------
// kernel argument blocks (passed by value; __grid_constant__ keeps them in the
// parameter bank so indexing them costs no local-memory copy)
// ---------------------------------------------------------------------------
template <class M, typename T>
struct ExplicitArgs {
    double* states;
    const double* fparams;
    uint32_t* flags;
    uint8_t* node_status;
    uint64_t ld;
    uint64_t nsteps;
    double t;
    double ldt;
    double delta;
    uint32_t N;
    T P[Dims<M>::np];
    double PD[Dims<M>::np];
    // goss_launch's schedule, outputs and exchange vector (see there); behind the
    // parameters, since in front of them they cost the plain GRL1 kernels spills
    // (262,144 TP06 nodes x 100 steps FP64 6.72 -> 6.87 ms, 2^20 FP32 2.96 -> 3.02)
    uint32_t forwards;
    const goss_forward* schedule;
    double* out;
    double* vector;
    const int64_t* dofs;
    uint64_t num_dofs;
    uint32_t num_fields;
    int32_t tangled;
    int8_t field_of[M::num_states];  // field of a state row, -1: none
};

template <class M>
struct ImplicitArgs {
    double* states;
    const double* fparams;
    double* sstate;  // per-node solver state, [rows][ld]
    uint32_t* flags;
    uint8_t* node_status;
    uint64_t ld;
    uint64_t max_loop;
    double t;
    double interval;
    goss_solver_params sp;
    uint32_t N;
    double P[Dims<M>::np];
    float P32[Dims<M>::np];  // the same block in FP32 (the FP32 Jacobian of GOSS_FP32)
};

template <class M, typename T>
struct EvalArgs {
    const double* states;
    const double* fparams;
    const double* times;
    double* out;
    uint64_t ld;
    uint32_t N;
    int32_t what;
    T P[Dims<M>::np];
    double PD[Dims<M>::np];
};

// ---------------------------------------------------------------------------
// explicit solvers
// ---------------------------------------------------------------------------
// GRL1Printed: GRL1 with the model evaluated in its printed operation order
// (the arithmetic of the reference's generated model code), FP64 only.
enum class Explicit { Euler, RK4, GRL1, GRL2, RL1, RL2, RK2, GRL1Printed };

template <class M, typename T>
__device__ __forceinline__ void load_field(const double* __restrict__ fp, uint64_t ld, uint32_t node,
                                           T (&F)[Dims<M>::nfp])
{
#pragma unroll
    for (int k = 0; k < Dims<M>::nfp; ++k)
        F[k] = (k < M::num_field_params) ? T(fp[k * ld + node]) : T(0);
}

// GRL increment of one state, FP64, in the reference's own expression
// b/a*(exp(a*h) - 1.0) or b*h (GRL1.h:80-83)
__device__ __forceinline__ double grl_increment(double a, double b, double h, double delta)
{
    return (fabs(a) > delta) ? b / a * (exp(a * h) - 1.0) : b * h;
}

// GRL increment of one state, FP32: b*h*phi1(a*h), algebraically identical
// and free of the cancellation in exp(a*h) - 1 (see phi1f).  (h phi1 with
// the polynomial's coefficients scaled by h, one multiply fewer per state,
// measured 1.4 % slower on B200: TP06, 1,048,576 nodes, 162 registers
// instead of 150.)
__device__ __forceinline__ float grl_increment(float a, float b, float h, float /*delta*/)
{
    return b * h * phi1f(a * h);
}

// 2 N states at once in packed FP32: the operations of grl_increment in the
// same order.  One branch for all of them, so that their polynomials overlap.
template <int N>
__device__ __forceinline__ void grl_increments(const float* a, const float* b, F32x2 h, F32x2* inc)
{
    F32x2 x[N], p[N];
    float far[N], all = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        x[i] = F32x2(a[2 * i], a[2 * i + 1]) * h;
        p[i] = phi1f_small(x[i]);
        float x0, x1;
        x[i].unpack(x0, x1);
        far[i] = fmaxf(fabsf(x0), fabsf(x1));
        all = fmaxf(all, far[i]);
    }
    if (all >= 0.25f) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (far[i] >= 0.25f) {
                float x0, x1, p0, p1;
                x[i].unpack(x0, x1);
                p[i].unpack(p0, p1);
                p[i] = F32x2(fabsf(x0) < 0.25f ? p0 : phi1f_large(x0), fabsf(x1) < 0.25f ? p1 : phi1f_large(x1));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
        inc[i] = F32x2(b[2 * i], b[2 * i + 1]) * h * p[i];
}

// RL increment of one state (RL1.h:68-77): the exponential form for the model's
// linear-term states whatever the coefficient (the reference divides by it),
// the Euler increment otherwise
__device__ __forceinline__ double rl_increment(bool linear, double a, double b, double h)
{
    return linear ? models::f64_div(b, a) * (models::f64_exp(a * h) - 1.0) : b * h;
}
__device__ __forceinline__ float rl_increment(bool linear, float a, float b, float h)
{
    return linear ? b * h * phi1f(a * h) : b * h;
}

// State accumulators.  FP64 kernels hold each state as a double and update it
// exactly as the reference does (y = y + increment).  FP32 kernels hold each
// state as an unevaluated sum hi + lo of two floats with compensated (Kahan)
// updates: the model reads hi, lo carries what hi could not absorb, so
// increments far below one float ulp of the state (K_i ~ 138 mM changes by
// less than one ulp per step) still accumulate.  Four FP32 adds per update,
// no FP32<->FP64 conversions (those would compete with the model's
// exponentials and reciprocals for the XU pipe on every step).
template <typename T>
struct Acc;

template <>
struct Acc<double> {
    double y;
    __device__ __forceinline__ void load(double v) { y = v; }
    __device__ __forceinline__ double store() const { return y; }
    __device__ __forceinline__ double value() const { return y; }
    __device__ __forceinline__ double plus(double d) const { return y + d; }
    __device__ __forceinline__ void add(double d) { y = y + d; }
    __device__ __forceinline__ void renormalize() {}
};

template <>
struct Acc<float> {
    float hi, lo;
    __device__ __forceinline__ void load(double v)
    {
        hi = float(v);
        lo = float(v - double(hi));
    }
    __device__ __forceinline__ double store() const { return double(hi) + double(lo); }
    __device__ __forceinline__ float value() const { return hi; }
    __device__ __forceinline__ float plus(float d) const { return hi + (lo + d); }
    __device__ __forceinline__ void add(float d)
    {
        // hi + lo + d: the sum goes to hi, its rounding error (exact when
        // |hi| >= |y|, Fast2Sum) back to lo
        const float y = __fadd_rn(d, lo);
        const float t = __fadd_rn(hi, y);
        lo = __fsub_rn(y, __fsub_rn(t, hi));
        hi = t;
    }
    // the same for two states at once.  d is a product, and ptxas fuses a
    // packed product and sum into one rounding; d * 1 + lo with a 1 it cannot
    // see keeps the scalar form's two.
    static __device__ __forceinline__ F32x2 opaque_one()
    {
        return F32x2(__uint_as_float(0x3f800000u + threadIdx.z));  // blocks are one-dimensional
    }
    static __device__ __forceinline__ F32x2 plus(const Acc& a, const Acc& b, F32x2 d)
    {
        return F32x2(a.hi, b.hi) + (F32x2(a.lo, b.lo) + d);
    }
    static __device__ __forceinline__ void add(Acc& a, Acc& b, F32x2 d)
    {
        const F32x2 hi(a.hi, b.hi);
        const F32x2 y = vfma(d, opaque_one(), F32x2(a.lo, b.lo));
        const F32x2 t = hi + y;
        (y - (t - hi)).unpack(a.lo, b.lo);
        t.unpack(a.hi, b.hi);
    }
    // between two forwards of one launch: bit for bit what store() to the
    // FP64 state array and load() by the next launch do, in FP32 arithmetic
    // (five FP64 conversions per state would double the XU pipe's work on a
    // one-step forward).  hi' = hi + lo rounded to FP32 and e its exact error
    // (two-sum); the FP64 round trip keeps e only to the FP64 grid of hi + lo,
    // g = 2^(floor(log2|hi + lo|) - 52), so e is rounded to a multiple of g
    // (ties to even) by adding and subtracting P = 2^23 g with e's sign, which
    // is exact for |e| < P; larger e are multiples of g already.  The binade
    // of hi + lo is that of hi' + e rounded toward zero (one below hi' when
    // hi' is a power of two and e has the opposite sign).  Sums below 2^-72
    // (where flushed FP32 subnormals would differ from the FP64 grid) and
    // non-finite sums take the FP64 round trip itself.
    __device__ __forceinline__ void renormalize()
    {
        const float t = __fadd_rn(hi, lo);
        const float at = fabsf(t);
        if (!(at >= 0x1p-72f && at <= 3.402823466e38f)) {
            load(store());
            return;
        }
        const float bp = __fsub_rn(t, hi);
        const float ap = __fsub_rn(t, bp);
        const float e = __fadd_rn(__fsub_rn(hi, ap), __fsub_rn(lo, bp));
        const float pow2 = __uint_as_float(__float_as_uint(__fadd_rz(t, e)) & 0x7f800000u);
        const float P = __fmul_rn(pow2, 0x1p-29f);
        const float C = copysignf(P, e);
        const float r = __fsub_rn(__fadd_rn(e, C), C);
        lo = fabsf(e) < P ? r : e;
        hi = t;
    }
};

// renormalize() of all states.  FP32: the same operations on pairs of states in
// packed arithmetic, with one range check for all of them instead of one branch
// per state; where a sum is outside the range (zero, tiny, infinite) every
// state takes the scalar form.  The check does not see a NaN, which passes
// through the packed form as a NaN and leaves its pair's other state alone.  A one-step forward of a cardiac model spends
// about as many instructions here as in its update, and the batch kernel is
// bound by issuing them: 492,003 nodes of three models x 100 forwards 2.28 -> 1.94 ms.
template <int n>
__device__ __forceinline__ void renormalize_states(Acc<double>*)
{
}
template <int n>
__device__ __forceinline__ void renormalize_states(Acc<float>* y)
{
    constexpr int pairs = n / 2, P = pairs > 0 ? pairs : 1;
    F32x2 t[P];
    float least = 3.402823466e38f, most = 0x1p-72f;
#pragma unroll
    for (int i = 0; i < pairs; ++i) {
        t[i] = F32x2(y[2 * i].hi, y[2 * i + 1].hi) + F32x2(y[2 * i].lo, y[2 * i + 1].lo);
        float t0, t1;
        t[i].unpack(t0, t1);
        least = fminf(least, fminf(fabsf(t0), fabsf(t1)));
        most = fmaxf(most, fmaxf(fabsf(t0), fabsf(t1)));
    }
    if (least >= 0x1p-72f && most <= 3.402823466e38f) {
#pragma unroll
        for (int i = 0; i < pairs; ++i) {
            Acc<float>&a = y[2 * i], &b = y[2 * i + 1];
            const F32x2 hi(a.hi, b.hi), lo(a.lo, b.lo);
            const F32x2 bp = t[i] - hi;
            const F32x2 ap = t[i] - bp;
            const F32x2 e = (hi - ap) + (lo - bp);
            float z0, z1, p0, p1, e0, e1, r0, r1;
            vadd_rz(t[i], e).unpack(z0, z1);
            const F32x2 pow2(__uint_as_float(__float_as_uint(z0) & 0x7f800000u),
                             __uint_as_float(__float_as_uint(z1) & 0x7f800000u));
            (pow2 * F32x2(0x1p-29f)).unpack(p0, p1);
            e.unpack(e0, e1);
            const F32x2 c(copysignf(p0, e0), copysignf(p1, e1));
            ((e + c) - c).unpack(r0, r1);
            a.lo = fabsf(e0) < p0 ? r0 : e0;
            b.lo = fabsf(e1) < p1 ? r1 : e1;
            t[i].unpack(a.hi, b.hi);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 2 * pairs; ++i)
            y[i].renormalize();
    }
    if constexpr (n % 2 != 0)
        y[n - 1].renormalize();
}

// Where one node's explicit solve reads and writes (shared by the
// single-population kernel and the batched kernel of goss_batch.cuh).
struct NodeIO {
    double* states;         // [n][ld]
    const double* fparams;  // [nfp][ld]
    uint8_t* node_status;   // [ld]
    uint32_t* flags;
    uint64_t ld;
    uint64_t nsteps;        // internal steps of one forward
    double t;
    double ldt;
    double delta;
    // consecutive forwards of one launch: forward f starts at
    // t + (first + f) * interval (the host loop's t0 + k * interval)
    uint32_t forwards = 1;
    uint64_t first = 0;
    double interval = 0.0;
};

// The model evaluations the explicit steps use: the split forms (every
// distinct transcendental and reciprocal of a state-dependent operand
// evaluated once), in FP32 and in FP64.  The split FP64 programs change the
// reference's results by re-association only; they stay within 1e-10 of the
// reference over 10^5 TP06 GRL1 steps.  GRL1Printed takes the programs in
// the printed operation order of the model (one exp per occurrence, divisions
// as written), the arithmetic of the reference's own generated code.
// Split FP64 programs run on models::F64, a double whose division,
// exponentials and square root have no branches (goss_device_math.cuh), but
// those of GRL1 and GRL2, see grl_linearized.
template <typename T>
struct SplitScalar {
    using type = T;
};
template <>
struct SplitScalar<double> {
    using type = models::F64;
};
template <typename T>
using split_t = typename SplitScalar<T>::type;
// a double array as the split programs' scalars, and the reverse
template <typename T>
__device__ __forceinline__ const split_t<T>* as_split(const T* p)
{
    return reinterpret_cast<const split_t<T>*>(p);
}
template <typename T>
__device__ __forceinline__ split_t<T>* as_split(T* p)
{
    return reinterpret_cast<split_t<T>*>(p);
}

template <class M, typename T>
__device__ __forceinline__ void model_linearized(const T* y, double t, const T* P, const double* PD, const T* F,
                                                 T* lin, T* rhs)
{
    M::template linearized_split<split_t<T>>(as_split(y), t, as_split(P), PD, as_split(F), as_split(lin),
                                             as_split(rhs));
}
template <class M, typename T>
__device__ __forceinline__ void model_rhs(const T* y, double t, const T* P, const double* PD, const T* F, T* f)
{
    M::template rhs_split<split_t<T>>(as_split(y), t, as_split(P), PD, as_split(F), as_split(f));
}

// The linearised model of the GRL steps.  FP64: plain doubles with CUDA's own
// division, exponentials and logarithms, whose rounding every result of the
// solver carries.  Where a state's coefficient a crosses zero (V's does in
// every upstroke) e^{ah} - 1 is a few multiples of 2^-53, so the last bit of a
// decides 1e-8 of that node's increment: on models::F64 the evaluation takes
// half the time (262,144 TP06 nodes x 100 steps 3.76 instead of 7.13 ms) but
// moved single nodes by 5e-8 of the states' scale, no nearer to nor further
// from the exact increment.
template <class M, typename T, bool Printed = false>
__device__ __forceinline__ void grl_linearized(const T* y, double t, const T* P, const double* PD, const T* F, T* lin,
                                               T* rhs)
{
    if constexpr (Printed)
        M::template linearized<T>(y, t, P, PD, F, lin, rhs);
    else
        M::template linearized_split<T>(y, t, P, PD, F, lin, rhs);
}

// The GRL update of every state: y[i].add(increment), or with Half the states
// of the half step, yt[i] = y[i].plus(increment).
template <int n, bool Half>
__device__ __forceinline__ void grl_update(Acc<double>* y, double* yt, const double* lin, const double* rhs, double h,
                                           double delta)
{
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const double d = grl_increment(lin[i], rhs[i], h, delta);
        if constexpr (Half)
            yt[i] = y[i].plus(d);
        else
            y[i].add(d);
    }
}

// FP32: two states at a time in packed arithmetic, the increments and the
// compensated accumulation alike, and up to ten pairs under one branch.
// Measured (TP06 GRL1, four fields, 262,144 nodes x 100 steps): one state at a
// time 0.929 ms; packed, 1 / 2 / 3 / 5 / 9 pairs under one branch 0.815 / 0.797
// / 0.777 / 0.764 / 0.748, which is 0.99 of the XU pipe's rate for the 131
// exponentials, logarithms and reciprocals of a step; one warp alone 0.087 ->
// 0.079 ms.
constexpr int kGrlPairs = 10;

template <int n, bool Half>
__device__ __forceinline__ void grl_update(Acc<float>* y, float* yt, const float* lin, const float* rhs, float h,
                                           float delta)
{
    constexpr int pairs = n / 2, N = kGrlPairs;
    const F32x2 hh(h);
    F32x2 d[pairs > 0 ? pairs : 1];
#pragma unroll
    for (int i = 0; i + N <= pairs; i += N)
        grl_increments<N>(lin + 2 * i, rhs + 2 * i, hh, d + i);
    if constexpr (pairs % N != 0)
        grl_increments<pairs % N>(lin + 2 * (pairs - pairs % N), rhs + 2 * (pairs - pairs % N), hh,
                                  d + pairs - pairs % N);
#pragma unroll
    for (int i = 0; i < pairs; ++i) {
        if constexpr (Half)
            Acc<float>::plus(y[2 * i], y[2 * i + 1], d[i]).unpack(yt[2 * i], yt[2 * i + 1]);
        else
            Acc<float>::add(y[2 * i], y[2 * i + 1], d[i]);
    }
    if constexpr (n % 2 != 0) {
        const float d = grl_increment(lin[n - 1], rhs[n - 1], h, delta);
        if constexpr (Half)
            yt[n - 1] = y[n - 1].plus(d);
        else
            y[n - 1].add(d);
    }
}

struct KeepNothing {
    template <typename T>
    __device__ __forceinline__ void operator()(int, const T*) const
    {
    }
};

// One internal step of an explicit solver at time lt with step ldt, in place
// on the accumulated states (shared by the thread-per-node solver kernels, the
// batch kernel and the adjoint kernels' record and recompute passes, so all take
// identical arithmetic; FP64 GRL1 on few nodes goes by group_step, which differs
// by rounding).
// keep(stage, k) sees RK4's stage derivatives.
template <class M, typename T, Explicit S, class Keep = KeepNothing>
__device__ __forceinline__ void explicit_step(Acc<T>* y, const double lt, const double ldt, const T* __restrict__ P,
                                              const double* __restrict__ PD, const T* __restrict__ F, const T delta,
                                              Keep keep = Keep())
{
    constexpr int n = M::num_states;
    const T h = T(ldt);
    const T hh = T(0.5 * ldt);
    T yt[n];
#pragma unroll
    for (int i = 0; i < n; ++i)
        yt[i] = y[i].value();
    if constexpr (S == Explicit::Euler) {
        // ExplicitEuler.cpp:80-81
        T f[n];
        model_rhs<M, T>(yt, lt, P, PD, F, f);
#pragma unroll
        for (int i = 0; i < n; ++i)
            y[i].add(h * f[i]);
    } else if constexpr (S == Explicit::RK4) {
        // RK4.cpp:79-98 with RK4::axpy (RK4.h:70-74); the weighted sum is
        // accumulated in the order k1 + 2 k2 + 2 k3 + k4 of the reference.
        // FP64: one copy of the right-hand side for the four stages (four
        // copies do not stay in the instruction cache: TP06, 262,144 nodes x
        // 100 steps 16.7 -> 12.2 ms; FP32, with a third of the instructions
        // per evaluation, 2.49 -> 2.66 ms, stays unrolled).
        T sum[n];
#pragma unroll(sizeof(T) == 4 ? 4 : 1)
        for (int st = 0; st < 4; ++st) {
            T k[n];
            model_rhs<M, T>(yt, st == 0 ? lt : st == 3 ? lt + ldt : lt + 0.5 * ldt, P, PD, F, k);
            keep(st, k);
            const T w = st == 1 || st == 2 ? T(2.0) : T(1.0), c = st == 2 ? h : hh;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                sum[i] = st == 0 ? k[i] : sum[i] + w * k[i];
                yt[i] = y[i].plus(c * k[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < n; ++i)
            y[i].add(T(split_t<T>(h * sum[i]) / split_t<T>(6.0)));
    } else if constexpr (S == Explicit::GRL1) {
        // GRL1.h:72-84
        T lin[n], rhs[n];
        grl_linearized<M, T>(yt, lt, P, PD, F, lin, rhs);
        grl_update<n, false>(y, yt, lin, rhs, h, delta);
    } else if constexpr (S == Explicit::GRL1Printed) {
        // GRL1.h:72-84 over the printed model program
        T lin[n], rhs[n];
        grl_linearized<M, T, true>(yt, lt, P, PD, F, lin, rhs);
        grl_update<n, false>(y, yt, lin, rhs, h, delta);
    } else if constexpr (S == Explicit::GRL2) {
        // GRL2: GRL2.cpp:78-82.  The reference's branch threshold is a
        // self-initialised local (GRL2.cpp:67) whose -O3 build behaves as 0:
        // the exponential form is used whenever the linear term is non-zero.
        // FP64: one copy of the linearised model for both evaluations, as in
        // RK4 (9.4 -> 8.2 ms; FP32 1.82 -> 1.92 ms, stays unrolled).
#pragma unroll(sizeof(T) == 4 ? 2 : 1)
        for (int st = 0; st < 2; ++st) {
            T lin[n], rhs[n];
            grl_linearized<M, T>(yt, lt, P, PD, F, lin, rhs);
            if (st == 0)
                grl_update<n, true>(y, yt, lin, rhs, hh, T(0));
            else
                grl_update<n, false>(y, yt, lin, rhs, h, T(0));
        }
    } else if constexpr (S == Explicit::RL1) {
        // RL1.h:68-77
        T lin[n], rhs[n];
        model_linearized<M, T>(yt, lt, P, PD, F, lin, rhs);
#pragma unroll
        for (int i = 0; i < n; ++i)
            y[i].add(rl_increment(M::linear_term(i), lin[i], rhs[i], h));
    } else if constexpr (S == Explicit::RL2) {
        // RL2.cpp:78-83: a half step to y2 linearised at y, then the full step
        // from y linearised at y2, both at time lt
#pragma unroll(sizeof(T) == 4 ? 2 : 1)
        for (int st = 0; st < 2; ++st) {
            T lin[n], rhs[n];
            model_linearized<M, T>(yt, lt, P, PD, F, lin, rhs);
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const T d = rl_increment(M::linear_term(i), lin[i], rhs[i], st == 0 ? hh : h);
                if (st == 0)
                    yt[i] = y[i].plus(d);
                else
                    y[i].add(d);
            }
        }
    } else {
        // RK2: RK2.cpp:78-89 with RK2::axpy (RK2.h:70-74), the midpoint rule
        static_assert(S == Explicit::RK2, "unhandled explicit solver");
#pragma unroll(sizeof(T) == 4 ? 2 : 1)
        for (int st = 0; st < 2; ++st) {
            T k[n];
            model_rhs<M, T>(yt, st == 0 ? lt : lt + 0.5 * ldt, P, PD, F, k);
#pragma unroll
            for (int i = 0; i < n; ++i) {
                if (st == 0)
                    yt[i] = y[i].plus(hh * k[i]);
                else
                    y[i].add(h * k[i]);
            }
        }
    }
}

// A step of 32 nodes by the four warps of a block, one lane of each warp to a
// node: warp W evaluates and updates the states of its row group
// (M::linear_group, M::rhs_group: the rows dealt out by the cost of what each
// needs), and what only the other rows need falls out of its copy of the
// model's program.  All warps hold all states; share(values) exchanges the new
// ones.  For grids that leave SMs idle, see explicit_in_groups.
template <class M, Explicit S>
__host__ __device__ constexpr int row_group(int i)
{
    return S == Explicit::GRL1 ? M::linear_group(i) : M::rhs_group(i);
}
constexpr int kGrlStates = 4;  // states under one branch

template <class M, Explicit S, int W>
__host__ __device__ constexpr int group_size()
{
    int c = 0;
    for (int i = 0; i < M::num_states; ++i)
        c += row_group<M, S>(i) == W;
    return c;
}

// GRL increments of N states at once, without branches but one for the N.
// e^x - 1 keeps the rounding of e^x to a double, as the reference's expression
// does (the exact (e^x - 1)/x, cheaper, differed from it by up to 1.4e-10 of V
// through an upstroke).  For |x| < 1/8 -- gates slower than 8 h, nearly all
// states of a cardiac model at its usual step -- e^x is 1 + x phi1(x) in one
// FMA over a polynomial, beyond that f64_exp.
template <int N>
__device__ __forceinline__ void grl_increments(const double* a, const double* b, double h, double delta, double* inc)
{
    double x[N], e[N];
    int far = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        x[i] = a[i] * h;
        e[i] = fma(x[i], models::f64_phi1_small(x[i]), 1.0);
        inc[i] = models::f64_div(b[i], a[i]);
        far = max(far, __double2hiint(x[i]) & 0x7fffffff);
    }
    if (far >= 0x3fc00000) {  // |x| >= 1/8, infinite or NaN
#pragma unroll
        for (int i = 0; i < N; ++i)
            if ((__double2hiint(x[i]) & 0x7fffffff) >= 0x3fc00000)
                e[i] = models::f64_exp(x[i]);
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
        inc[i] = fabs(a[i]) > delta ? inc[i] * (e[i] - 1.0) : b[i] * h;
}

// the update of this warp's states
template <class M, Explicit S, int W>
__device__ __forceinline__ void grl_update_group(Acc<double>* y, const double* lin, const double* rhs, double h,
                                                 double delta)
{
    constexpr int n = M::num_states, N = group_size<M, S, W>();
    if constexpr (N > 0) {
        double a[N], b[N], d[N];
        int c = 0;
#pragma unroll
        for (int i = 0; i < n; ++i)
            if (row_group<M, S>(i) == W) {
                a[c] = lin[i];
                b[c] = rhs[i];
                ++c;
            }
        constexpr int rest = N % kGrlStates;
#pragma unroll
        for (int i = 0; i + kGrlStates <= N; i += kGrlStates)
            grl_increments<kGrlStates>(a + i, b + i, h, delta, d + i);
        if constexpr (rest != 0)
            grl_increments<rest>(a + N - rest, b + N - rest, h, delta, d + N - rest);
        c = 0;
#pragma unroll
        for (int i = 0; i < n; ++i)
            if (row_group<M, S>(i) == W)
                y[i].add(d[c++]);
    }
}

template <class M, Explicit S, int W, class Share>
__device__ __forceinline__ void group_step(Acc<double>* y, const double lt, const double h, const double* __restrict__ P,
                                           const double* __restrict__ PD, const double* __restrict__ F,
                                           const double delta, Share share)
{
    constexpr int n = M::num_states;
    const double hh = 0.5 * h;
    double yt[n];
#pragma unroll
    for (int i = 0; i < n; ++i)
        yt[i] = y[i].value();
    if constexpr (S == Explicit::RK4) {
        double sum[n];
#pragma unroll 1
        for (int st = 0; st < 4; ++st) {
            double k[n];
            model_rhs<M, double>(yt, st == 0 ? lt : st == 3 ? lt + h : lt + 0.5 * h, P, PD, F, k);
            const double w = st == 1 || st == 2 ? 2.0 : 1.0, c = st == 2 ? h : hh;
#pragma unroll
            for (int i = 0; i < n; ++i)
                if (row_group<M, S>(i) == W) {
                    sum[i] = st == 0 ? k[i] : sum[i] + w * k[i];
                    if (st == 3) {
                        y[i].add(double(models::F64(h * sum[i]) / models::F64(6.0)));
                        yt[i] = y[i].value();
                    } else {
                        yt[i] = y[i].plus(c * k[i]);
                    }
                }
            share(yt);
        }
    } else {
        static_assert(S == Explicit::GRL1, "unhandled explicit solver");
        double lin[n], rhs[n];
        model_linearized<M, double>(yt, lt, P, PD, F, lin, rhs);
        grl_update_group<M, S, W>(y, lin, rhs, h, delta);
#pragma unroll
        for (int i = 0; i < n; ++i)
            yt[i] = y[i].value();
        share(yt);
    }
#pragma unroll
    for (int i = 0; i < n; ++i)
        y[i].load(yt[i]);
}

// Advance one node over nsteps internal steps of one explicit solver, from
// its accumulated states and field parameters, and store the result.
template <class M, typename T, Explicit S>
__device__ __forceinline__ void explicit_node_core(const NodeIO& a, uint32_t node, const T* __restrict__ P,
                                                   const double* __restrict__ PD, Acc<T>* y, const T* F)
{
    constexpr int n = M::num_states;
    const double ldt = a.ldt;
    const T delta = T(a.delta);
    for (uint32_t f = 0; f < a.forwards; ++f) {
        if (f)
            renormalize_states<n>(y);
        // rounded like the host's t0 + k * interval (no fused multiply-add)
        double lt = __dadd_rn(a.t, __dmul_rn(double(a.first + f), a.interval));
        for (uint64_t step = 0; step < a.nsteps; ++step) {
            explicit_step<M, T, S>(y, lt, ldt, P, PD, F, delta);
            lt += ldt;
        }
    }
    bool finite = true;
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const double v = y[i].store();
        a.states[i * a.ld + node] = v;
        finite = finite && isfinite(v);
    }
    if (!finite) {
        a.node_status[node] |= GOSS_FLAG_NONFINITE;
        atomicOr(a.flags, GOSS_FLAG_NONFINITE);
    }
}

// ... reading the node's states and field parameters from global memory
template <class M, typename T, Explicit S>
__device__ __forceinline__ void explicit_node(const NodeIO& a, uint32_t node, const T* __restrict__ P,
                                              const double* __restrict__ PD)
{
    constexpr int n = M::num_states;
    Acc<T> y[n];
#pragma unroll
    for (int i = 0; i < n; ++i)
        y[i].load(a.states[i * a.ld + node]);
    T F[Dims<M>::nfp];
    load_field<M, T>(a.fparams, a.ld, node, F);
    explicit_node_core<M, T, S>(a, node, P, PD, y, F);
}

// ... reading them from rows[r * stride]: the n state rows, then the field
// parameter rows (a tile staged in shared memory by the batch kernel)
template <class M, typename T, Explicit S>
__device__ __forceinline__ void explicit_node_from(const NodeIO& a, uint32_t node, const T* __restrict__ P,
                                                   const double* __restrict__ PD, const double* rows,
                                                   uint32_t stride)
{
    constexpr int n = M::num_states;
    Acc<T> y[n];
#pragma unroll
    for (int i = 0; i < n; ++i)
        y[i].load(rows[i * stride]);
    T F[Dims<M>::nfp];
#pragma unroll
    for (int k = 0; k < Dims<M>::nfp; ++k)
        F[k] = (k < M::num_field_params) ? T(rows[(n + k) * stride]) : T(0);
    explicit_node_core<M, T, S>(a, node, P, PD, y, F);
}

// Resident blocks of 128 threads per SM the explicit kernels are compiled for
// (register cap 65536 / (128 * blocks)).  FP32: uncapped (150 registers for
// TP06 GRL1, 3 blocks per SM; capped at 128 it measured 1-13 % slower at every
// size).  FP64: 3 (168 registers), whose extra warps hide the FP64 latencies
// better than the spills cost; GRL1, GRL2 and RK4 also 2 (255 registers), which
// is faster while the grid leaves an SM no third block, see explicit_blocks.
#ifndef GOSS_EXPLICIT_MIN_BLOCKS_FP32
#define GOSS_EXPLICIT_MIN_BLOCKS_FP32 1
#endif
template <typename T>
struct ExplicitMinBlocks {
    static constexpr int value = sizeof(T) == 4 ? GOSS_EXPLICIT_MIN_BLOCKS_FP32 : 3;
};
template <typename T, Explicit S>
constexpr bool explicit_two_shapes =
    sizeof(T) == 8 && (S == Explicit::GRL1 || S == Explicit::GRL2 || S == Explicit::RK4);

// Resident blocks per SM to run `grid` FP64 blocks of 128 with: the time of the
// full waves and of the last one under either register cap.  Time of a wave
// with one, two (three) blocks on every SM, measured for TP06 and 100 steps
// (GRL2's are GRL1's to 2 % in proportion): e.g. GRL1 one node 2, 50,021 nodes 3
// (1.49 against 2.16 ms), 65,536 nodes 2 (2.16 against 2.56 ms), 262,144 nodes 3
// (6.74 against 7.41 ms).
template <Explicit S>
inline int explicit_blocks(unsigned grid)
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        return 3;
    auto time = [&](unsigned k, const double* wave) {
        const unsigned slots = k * (unsigned)sms, full = grid / slots, rest = grid % slots;
        return full * wave[k] + wave[(rest + sms - 1) / sms];
    };
    constexpr bool rk4 = S == Explicit::RK4;
    constexpr double wide[] = {0.0, rk4 ? 1.81 : 1.007, rk4 ? 1.85 : 1.082};
    constexpr double narrow[] = {0.0, rk4 ? 1.99 : 1.063, rk4 ? 2.14 : 1.149, rk4 ? 2.80 : 1.494};
    return time(2, wide) < time(3, narrow) ? 2 : 3;
}

template <class M, typename T, Explicit S, int Blocks>
__global__ void __launch_bounds__(128, Blocks) explicit_kernel(const __grid_constant__ ExplicitArgs<M, T> a)
{
    const uint32_t node = blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= a.N)
        return;
    const NodeIO io{a.states, a.fparams, a.node_status, a.flags, a.ld, a.nsteps, a.t, a.ldt, a.delta};
    explicit_node<M, T, S>(io, node, a.P, a.PD);
}

// The solvers that also take goss_launch's schedule, outputs and exchange
// vector.  A kernel of their own: with the step length and count in registers
// instead of the argument block, plain forwards measured 0.5 % (FP32) to 2.5 %
// (FP64, spills) slower.
template <Explicit S>
constexpr bool explicit_extended =
    S == Explicit::Euler || S == Explicit::RK4 || S == Explicit::GRL1 || S == Explicit::GRL2;

// A node's entry of the exchange vector; none without a vector, and none, with
// the status flag set, for a dof outside it.
template <class M, typename T>
__device__ __forceinline__ double* exchange_entry(const ExplicitArgs<M, T>& a, uint32_t node)
{
    if (!a.vector)
        return nullptr;
    const uint64_t dof = (uint64_t)a.dofs[node];
    if (dof < a.num_dofs)
        return a.vector + dof * a.num_fields;
    a.node_status[node] |= GOSS_FLAG_BAD_DOF;
    atomicOr(a.flags, GOSS_FLAG_BAD_DOF);
    return nullptr;
}

// One forward, or the forwards of a schedule with the states in registers from
// one to the next (rounded between them as a store and load would); field
// states from and to a vector and into outputs after every forward.  Saves a
// small system the launches between: ten output times of a two-state cell
// 184 -> 129 us, a coupled step of 72,002 + 28,001 nodes 89 -> 76 us.
template <class M, typename T, Explicit S, int Blocks>
__global__ void __launch_bounds__(128, Blocks) schedule_kernel(const __grid_constant__ ExplicitArgs<M, T> a)
{
    constexpr int n = M::num_states;
    const uint32_t node = blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= a.N)
        return;
    Acc<T> y[n];
    {
        const double* const v = exchange_entry(a, node);
#pragma unroll
        for (int i = 0; i < n; ++i)
            y[i].load(v && a.field_of[i] >= 0 ? v[a.field_of[i]] : a.states[i * a.ld + node]);
    }
    T F[Dims<M>::nfp];
    load_field<M, T>(a.fparams, a.ld, node, F);
    const T delta = T(a.delta);
    double lt = a.t, ldt = a.ldt;
    uint64_t nsteps = a.nsteps;
    bool finite = true;
    for (uint32_t f = 0; f < a.forwards; ++f) {
        if (f)
            renormalize_states<n>(y);
        if (a.schedule) {
            lt = a.schedule[f].t;
            ldt = a.schedule[f].ldt;
            nsteps = a.schedule[f].nsteps;
        }
        for (uint64_t step = 0; step < nsteps; ++step) {
            explicit_step<M, T, S>(y, lt, ldt, a.P, a.PD, F, delta);
            lt += ldt;
        }
        if (a.out) {
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const double w = y[i].store();
                finite = finite && isfinite(w);
                if (a.field_of[i] >= 0) {
                    const uint64_t k = (uint64_t)a.field_of[i], row = (uint64_t)f * a.num_fields;
                    a.out[a.tangled ? row * a.N + (uint64_t)node * a.num_fields + k : (row + k) * a.N + node] = w;
                }
            }
        }
    }
    double* const v = exchange_entry(a, node);
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const double w = y[i].store();
        a.states[i * a.ld + node] = w;
        if (v && a.field_of[i] >= 0)
            v[a.field_of[i]] = w;
        finite = finite && isfinite(w);
    }
    if (!finite) {
        a.node_status[node] |= GOSS_FLAG_NONFINITE;
        atomicOr(a.flags, GOSS_FLAG_NONFINITE);
    }
}

// a barrier of the block's 128 threads that its warps reach at different places
__device__ __forceinline__ void block_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// schedule_kernel with the rows of a node split over the block's four warps (W:
// this warp's), the model on models::F64 for GRL1 too: a population of the size
// that comes here has no node near enough to a coefficient's zero for that to
// show (2,000 to 2,368 nodes through the stimulus: at most 7e-10 of the states'
// scale between the two kernels; RK4's are equal bit for bit).  A thread alone on its scheduler is bound by the length of its
// instruction stream; here that is a third of the step's (TP06's four groups
// cost 1.3 times the whole between them).  One exchange through shared memory
// and one barrier per model evaluation.
template <class M, Explicit S, int W>
__device__ __forceinline__ void group_node(const ExplicitArgs<M, double>& a, double (*shared)[M::num_states][32])
{
    constexpr int n = M::num_states;
    const uint32_t lane = threadIdx.x & 31, at = blockIdx.x * 32 + lane;
    const bool active = at < a.N;
    const uint32_t node = active ? at : a.N - 1;
    Acc<double> y[n];
    double* const v = exchange_entry(a, node);
#pragma unroll
    for (int i = 0; i < n; ++i)
        y[i].load(v && a.field_of[i] >= 0 ? v[a.field_of[i]] : a.states[i * a.ld + node]);
    double F[Dims<M>::nfp];
    load_field<M, double>(a.fparams, a.ld, node, F);
    block_barrier();  // every warp has read the states the others will write
    unsigned turn = 0;
    // two buffers in turn: a warp is at most one barrier ahead of the others
    const auto share = [&](double* values) {
        double(*const s)[32] = shared[turn];
        turn ^= 1;
#pragma unroll
        for (int i = 0; i < n; ++i)
            if (row_group<M, S>(i) == W)
                s[i][lane] = values[i];
        block_barrier();
#pragma unroll
        for (int i = 0; i < n; ++i)
            if (row_group<M, S>(i) != W)
                values[i] = s[i][lane];
    };
    double lt = a.t, ldt = a.ldt;
    uint64_t nsteps = a.nsteps;
    bool finite = true;
    for (uint32_t f = 0; f < a.forwards; ++f) {
        if (a.schedule) {
            lt = a.schedule[f].t;
            ldt = a.schedule[f].ldt;
            nsteps = a.schedule[f].nsteps;
        }
        for (uint64_t step = 0; step < nsteps; ++step) {
            group_step<M, S, W>(y, lt, ldt, a.P, a.PD, F, a.delta, share);
            lt += ldt;
        }
        if (a.out && active) {
#pragma unroll
            for (int i = 0; i < n; ++i) {
                if (row_group<M, S>(i) != W)
                    continue;
                const double w = y[i].store();
                finite = finite && isfinite(w);
                if (a.field_of[i] >= 0) {
                    const uint64_t k = (uint64_t)a.field_of[i], row = (uint64_t)f * a.num_fields;
                    a.out[a.tangled ? row * a.N + (uint64_t)node * a.num_fields + k : (row + k) * a.N + node] = w;
                }
            }
        }
    }
    if (!active)
        return;
#pragma unroll
    for (int i = 0; i < n; ++i) {
        if (row_group<M, S>(i) != W)
            continue;
        const double w = y[i].store();
        a.states[i * a.ld + node] = w;
        if (v && a.field_of[i] >= 0)
            v[a.field_of[i]] = w;
        finite = finite && isfinite(w);
    }
    if (!finite) {
        a.node_status[node] |= GOSS_FLAG_NONFINITE;  // every warp writes the same value
        atomicOr(a.flags, GOSS_FLAG_NONFINITE);
    }
}

template <class M, Explicit S>
__global__ void __launch_bounds__(128, 2) group_kernel(const __grid_constant__ ExplicitArgs<M, double> a)
{
    __shared__ double shared[2][M::num_states][32];
    switch (threadIdx.x >> 5) {
    case 0: group_node<M, S, 0>(a, shared); break;
    case 1: group_node<M, S, 1>(a, shared); break;
    case 2: group_node<M, S, 2>(a, shared); break;
    default: group_node<M, S, 3>(a, shared); break;
    }
}

// Models generated without row groups (too few states to share out, or too many
// for the exchange buffers) keep a thread per node.  So does GRL2: a copy
// of the program that leaves out rows contracts other products, and over 100 ms
// of 2,048 nodes GRL2 carried that to 1.6e-9 of the reference (bar 1e-9).
template <class M, class = void>
struct HasRowGroups {
    static constexpr bool value = false;
};
template <class M>
struct HasRowGroups<M, decltype(void(M::linear_group(0) + M::rhs_group(0)))> {
    static constexpr bool value = true;
};
template <class M, typename T, Explicit S>
constexpr bool explicit_groups =
    sizeof(T) == 8 && (S == Explicit::GRL1 || S == Explicit::RK4) && HasRowGroups<M>::value;

// Whether to split the rows: blocks of 32 nodes on at most half the SMs.  The
// time is flat to a quarter of them, then grows by the block as the SMs of a
// GPC fetch four instruction streams each through one cache.  100 steps, thread
// per node / split, ms (4 fields, FP64; at 3,840 nodes TP06's RK4 takes 1.56 / 2.08):
//   nodes          1            256          1,184         1,792         2,368
//   TP06 GRL1  0.97 / 0.19   0.97 / 0.21   0.97 / 0.22   0.97 / 0.34   0.98 / 0.40
//   TP06 RK4   1.42 / 0.62   1.34 / 0.70   1.50 / 0.76   1.50 / 1.17   1.56 / 1.39
//   TT04 GRL1  0.88 / 0.17   0.88 / 0.19   0.88 / 0.21   0.88 / 0.32   0.88 / 0.38
//   TT04 RK4   1.19 / 0.55   1.06 / 0.65   1.30 / 0.71   1.30 / 1.11   1.36 / 1.32
// Coefficients within [-delta, delta] take the Euler increment; a delta below
// kGrlTiny stays with the thread per node, whose division takes every operand.
constexpr double kGrlTiny = 0x1p-1000;

inline bool explicit_in_groups(uint32_t num_nodes, double delta)
{
    if (!(delta >= kGrlTiny))
        return false;
    int dev = 0, sms = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
           cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
           num_nodes <= 16u * (uint32_t)sms;
}

// ---------------------------------------------------------------------------
// dense linear algebra on one node's n x n matrix
// ---------------------------------------------------------------------------
// Newton matrices of the implicit solvers are stored packed (the model's
// lu_nnz entries of the LU structure of I - h*alpha*J, generated with the
// structure-aware factorisation and solve that reproduce ODE::lu_factorize and
// ODE::forward_backward_subst, ODE.cpp:69-132), their entries models::F64 (a
// double whose divisions have no branches): in a thread-local array, or in a
// tiled region: the 32 nodes of a tile keep their entries together
// ([tile][k][32]), so a warp's lu_nnz entries are one contiguous block of
// 256-byte rows instead of lu_nnz rows ld apart (each 2 MiB apart at 262,144
// nodes, whose cost depended on how the allocation happened to be mapped)
struct PackedTile {
    double* base;
    __device__ __forceinline__ models::F64& operator[](int k) const { return *as_split(base + (uint64_t)k * 32); }
};

__device__ __forceinline__ PackedTile packed_tile(double* region, uint32_t node, int nnz)
{
    return PackedTile{region + (((uint64_t)(node >> 5) * (uint64_t)nnz) << 5) + (node & 31u)};
}

template <int n>
__device__ __forceinline__ double l2norm(const double* v)
{
    double s = 0;
#pragma unroll
    for (int i = 0; i < n; ++i)
        s += v[i] * v[i];
    return models::f64_sqrt(s);
}

// pow(x, 0.8) of a positive convergence rate (the Newton stopping rules' eta):
// the exponential of 0.8 log x, whose argument carries its rounding into up to
// 10 ulp of the result, one Newton step on y^5 = x^4, and the x^(0.8 - 4/5) by
// which the double 0.8 exceeds 4/5.  At most 1.31 ulp over 4 million x from
// 2^-52 to 1e16, pow 1.34 (pow itself takes 6-8 % of a ThetaSolver interval, this
// 1 %); pow where x^4 leaves the normal range.
__device__ __forceinline__ double pow_0_8(double x)
{
    const double l = models::f64_log(x), y = models::f64_exp(0.8 * l);
    const double x2 = x * x, y2 = y * y, x4 = x2 * x2;
    if (!models::f64_normal(x4))
        return pow(x, 0.8);
    return fma(y, fma(0.2 * fma(-(y2 * y2), y, x4), models::f64_rcp(x4), 4.440892098500626e-17 * l), y);
}

// x^(1/4) (ESDIRK23a's step-size controller)
__device__ __forceinline__ double root4(double x) { return models::f64_sqrt(models::f64_sqrt(x)); }

// x^n of a finite x by squaring, with what each product's rounding left out
// carried along in p_lo and b_lo (each of up to nine products rounds, and a
// squaring doubles the error before it)
__device__ __forceinline__ double pow_int(double x, int n)
{
    double p = 1.0, p_lo = 0.0, b = x, b_lo = 0.0;
    for (int k = n < 0 ? -n : n; k; k >>= 1) {
        if (k & 1) {
            const double q = p * b;
            p_lo = fma(p, b, -q) + fma(p, b_lo, p_lo * b);
            p = q;
        }
        const double s = b * b;
        b_lo = fma(b, b, -s) + 2.0 * (b * b_lo);
        b = s;
    }
    p += p_lo;
    return n < 0 ? models::f64_div(1.0, p) : p;
}

// FP64 model right-hand side of the implicit solvers: the split form (every
// distinct exp and reciprocal once, common factors pulled out), whose values
// differ from the reference's operation order by rounding only; Newton
// iterates to the same states (the implicit parity tests hold at 1e-10).  The
// right-hand side, the Jacobians, the packed LU and the step control run on
// models::F64: without the slow-path branches of CUDA's division, exp, log,
// sqrt and pow, and with one reciprocal per pivot and per forward-difference
// step, a 0.1 ms interval of 262,144 TT04 nodes takes (blocks of 256, 255
// registers; at 128 or 168 registers 1.2-1.8x longer):
//   ThetaSolver 0.89 -> 0.62 ms, + Jacobian 0.43 -> 0.27, ImplicitEuler
//   1.47 -> 0.87, + Jacobian 0.95 -> 0.68, ESDIRK23a 3.8 -> 2.5, + Jacobian
//   3.4 -> 2.25 (intervals of a relaxing population, min_dt 1e-4).
// Inlined at every call site: on TT04 with the analytic Jacobian, called
// (__noinline__) versions of these two measured 1.3x slower, and capping the
// kernels at 128 or 170 registers (3 or 4 blocks of 128 per SM) 1.3-1.4x
// slower, than the 255-register inlined kernel.
template <class M>
__device__ __forceinline__ void rhs64(const double* y, double t, const double* P, const double* F, double* out)
{
    model_rhs<M, double>(y, t, P, P, F, out);
}

// The analytic Jacobian evaluated in FP32 at the FP64 point (y, t) and stored
// into the FP64 packed Newton matrix: the implicit solvers' GOSS_FP32 mode.
// The matrix only steers the simplified Newton iteration (the residual, the
// right-hand sides, the LU and the updates stay FP64), so the iteration
// converges to the same tolerance with an FP32-accurate matrix.
template <class M, class A>
__device__ __forceinline__ void jacobian32(const double* y, double t, const float* P32, const double* PD,
                                           const double* F, A J)
{
    float yf[M::num_states];
#pragma unroll
    for (int i = 0; i < M::num_states; ++i)
        yf[i] = float(y[i]);
    float Ff[Dims<M>::nfp];
#pragma unroll
    for (int k = 0; k < Dims<M>::nfp; ++k)
        Ff[k] = float(F[k]);
    M::template jacobian<float>(yf, t, P32, PD, Ff, J);
}

// ---------------------------------------------------------------------------
// ThetaSolver
// ---------------------------------------------------------------------------
// per-node solver state rows
enum ThetaRows { TH_ETA = 0, TH_RECOMPUTE, TH_ALWAYS, TH_JUSTREFINED, TH_JACCOMP, TH_REJECTS, TH_ACCEPTED, TH_ROWS };

// ThetaSolver::forward (ThetaSolver.cpp:49-155); with IE, ImplicitEuler::forward
// (ImplicitEuler.cpp:57-152): theta = 1 (no explicit part, stage time t + ldt),
// the Jacobian always recomputed once MORE than num_refinements_without_
// always_recomputing_jacobian refinements happened (Theta: up to that many),
// and a failed step requests a new Jacobian.
// Lockstep form: every pass of the block-uniform loop runs one Newton
// iteration of every node that is not done (starting its next step first
// when the previous one ended), then the block synchronises, so the block's
// warps walk the large inlined right-hand side, Jacobian and LU together and
// share instruction-cache lines.  The per-node arithmetic and its order are
// those of the nested loops of ThetaSolver::forward (the states equal the
// nested-loop kernel's bit for bit).  Measured on B200 (TT04, 262,144 nodes,
// 0.1 ms intervals, blocks of 256 against the nested loops in blocks of 64):
// ImplicitEuler with the analytic Jacobian 2.49 -> 1.53 ms, ThetaSolver with
// it 1.24 -> 1.16 ms, with forward differences unchanged (4.41 ms).  Again
// with one model evaluation site per iteration (below), against each warp
// looping on its own (__any_sync): ImplicitEuler 1.03 against 1.33 ms (1.56
// against 2.36 with forward differences), ThetaSolver within 2 %.  Blocks of
// up to 256 threads; __launch_bounds__(256, 1) keeps the 255-register budget
// (without the minimum of one block ptxas capped it at 128 and spilled more).
//
// Launch shape: at most GOSS_THETA_THREADS threads per block, compiled for
// GOSS_THETA_MIN_BLOCKS resident blocks per SM (register cap 65536 / product).
// Measured on B200 (TT04 with the analytic Jacobian, 262,144 nodes, 0.1 ms
// intervals): 256 x 1 with the Newton matrix, z1 and prev in registers and
// local memory 0.61 ms per interval; the same with them in dynamic shared
// memory 0.77 ms (the DRAM spill traffic disappears, but the shared memory
// takes the L1 capacity the remaining spills hit in); the matrix alone in
// shared memory 0.79 ms, and in blocks of 128 x 3 (168 registers) 0.92 ms.
#ifndef GOSS_THETA_THREADS
#define GOSS_THETA_THREADS 256
#endif
#ifndef GOSS_THETA_MIN_BLOCKS
#define GOSS_THETA_MIN_BLOCKS 1
#endif
template <class M, bool IE, bool J32 = false>
__global__ void __launch_bounds__(GOSS_THETA_THREADS, GOSS_THETA_MIN_BLOCKS)
    theta_kernel(const __grid_constant__ ImplicitArgs<M> a)
{
    constexpr int n = M::num_states;
    // One inlined copy of the model evaluation (an instruction-cache effect:
    // the per-node code is far larger than the cache, and instruction fetch is
    // the top stall).  ImplicitEuler, which keeps its Jacobian and mostly
    // evaluates f alone: every iteration through rhs_jacobian_sel or
    // rhs_fd_jacobian_sel (the Jacobian's own statements under a run-time
    // condition).  ThetaSolver, which refactorises in (nearly) every
    // iteration: every refactorising iteration through rhs2_jacobian or
    // rhs2_fd_jacobian, f(y, t) used at a step's first iteration only (the
    // time-dependent statements are evaluated at t each time).  Measured when
    // introduced (TT04, 262,144 nodes, 0.1 ms intervals, A/B in one process):
    // ImplicitEuler 1.30 -> 1.04 ms per interval with the analytic Jacobian,
    // 1.88 -> 1.54 ms with forward differences; ThetaSolver with the analytic
    // Jacobian 0.61 -> 0.55 ms (through rhs_jacobian_sel instead: 0.69 ms, the
    // Jacobian's statements no longer interleave with f's), with forward
    // differences 0.578 -> 0.559 ms.
    constexpr bool one_eval = !J32 && IE;
    // ImplicitEuler with the FP32 Jacobian: one FP64 right-hand-side call
    // site for every iteration, the FP32 Jacobian when refactorising (1.22 ->
    // 0.77 ms per interval; for ThetaSolver, with f(y, t) of a step's first
    // iteration from the same call site, 0.57 -> 0.73 ms, not used)
    constexpr bool one_eval32 = J32 && IE;
    const uint32_t node = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = node < a.N;
    const uint32_t src = active ? node : a.N - 1;  // threads past the end only take part in the barriers
    const goss_solver_params& sp = a.sp;
    const models::F64* const PS = as_split(a.P);
    double y[n], z1[n], prev[n], yz[n], f1[n], b[n];
    models::F64 J[M::lu_nnz];
    for (int i = 0; i < n; ++i)
        y[i] = a.states[i * a.ld + src];
    double F[Dims<M>::nfp];
    load_field<M, double>(a.fparams, a.ld, src, F);
    double* ss = a.sstate + src;
    const uint64_t ld = a.ld;
    double eta = ss[TH_ETA * ld];
    int recompute = ss[TH_RECOMPUTE * ld] != 0.0;
    int always = ss[TH_ALWAYS * ld] != 0.0;
    int justrefined = ss[TH_JUSTREFINED * ld] != 0.0;
    double jac_comp = ss[TH_JACCOMP * ld], rejects = ss[TH_REJECTS * ld], accepted = ss[TH_ACCEPTED * ld];
    double* const jrows = ss + (uint64_t)TH_ROWS * ld;
    if constexpr (IE) {
#pragma unroll
        for (int k = 0; k < M::lu_nnz; ++k)
            J[k] = jrows[(uint64_t)k * ld];
    }

    double t = a.t;
    const double dt = a.interval;
    const double t_end = t + dt;
    const double ldt_0 = sp.ldt;
    double ldt = ldt_0 > 0 ? ldt_0 : dt;
    int num_refinements = 0;
    const double eps = kGossEps * 1000;
    uint8_t status = 0;
    for (int i = 0; i < n; ++i)
        prev[i] = 0.0;
    uint64_t guard = 0;
    // the step in progress and its Newton iteration state
    bool done = !active, in_step = false, step_ok = true, prev_pending = false;
    double tn = 0.0, alpha = 1.0;
    int newton_iterations = 0;
    double relative_previous_residual = 1.0, relative_residual = 1.0, previous_residual = 1.0;
    double initial_residual = 1.0, residual;
    while (__syncthreads_or(!done)) {
        if (done)
            continue;
        if (!in_step) {
            if (++guard > a.max_loop) {
                status |= GOSS_FLAG_ITERATION_CAP;
                done = true;
                continue;
            }
            for (int i = 0; i < n; ++i)
                z1[i] = 0.0;
            if (IE ? num_refinements > sp.num_refinements_without_always_recomputing_jacobian
                   : num_refinements <= sp.num_refinements_without_always_recomputing_jacobian)
                always = 1;
            tn = IE ? t + ldt : t + sp.theta * ldt;
            alpha = IE ? 1.0 : sp.theta;
            step_ok = true;
            newton_iterations = 0;
            relative_previous_residual = relative_residual = previous_residual = initial_residual = 1.0;
            // (1 - theta) f(y, t): when the step's first Newton iteration will
            // refactorise, its f(y, tn) evaluation writes f(y, t) as well
            prev_pending = false;
            if (!IE && fabs(sp.theta - 1.0) > kGossEps) {
                if (!(relative_residual < sp.relative_tolerance) && (recompute || always)) {
                    prev_pending = true;
                } else {
                    rhs64<M>(y, t, a.P, F, f1);
                    for (int i = 0; i < n; ++i)
                        prev[i] = (1 - sp.theta) * f1[i];
                }
            }
            in_step = true;
        }
        // one iteration of ImplicitODESolver::newton_solve (ImplicitODESolver.cpp:114-245)
        bool newton_done = false;
        for (int i = 0; i < n; ++i)
            yz[i] = y[i] + z1[i];
        // when this iteration will refactorise (both conditions are known
        // before f(yz) is evaluated), f(yz) and the Jacobian come from one
        // evaluation: the unperturbed statements of the forward differences,
        // or the statements the analytic Jacobian shares with f
        if constexpr (one_eval32) {
            const bool want_jac = !(relative_residual < sp.relative_tolerance) && (recompute || always);
            rhs64<M>(yz, tn, a.P, F, f1);
            if (want_jac)
                jacobian32<M>(yz, tn, a.P32, a.P, F, J);
        } else if constexpr (one_eval) {
            // f(yz, tn), and the Jacobian when this iteration refactorises
            const bool want_jac = !(relative_residual < sp.relative_tolerance) && (recompute || always);
            if constexpr (M::has_jacobian)
                M::template rhs_jacobian_sel<models::F64>(as_split(yz), tn, PS, a.P, as_split(F), t, false, want_jac,
                                                          as_split(b), as_split(f1), J);
            else
                M::template rhs_fd_jacobian_sel<models::F64>(as_split(yz), tn, PS, a.P, as_split(F), want_jac,
                                                             as_split(f1), J);
        } else if (!(relative_residual < sp.relative_tolerance) && (recompute || always)) {
            if constexpr (J32) {
                // FP64 right-hand sides, the FP32 Jacobian
                if (prev_pending) {
                    rhs64<M>(yz, t, a.P, F, b);
                    for (int i = 0; i < n; ++i)
                        prev[i] = (1 - sp.theta) * b[i];
                    prev_pending = false;
                }
                rhs64<M>(yz, tn, a.P, F, f1);
                jacobian32<M>(yz, tn, a.P32, a.P, F, J);
            } else {
                // ThetaSolver: f(yz, t) into b, at the first iteration of the
                // step (yz = y) the explicit part
                if constexpr (M::has_jacobian) {
                    M::template rhs2_jacobian<models::F64>(as_split(yz), tn, PS, a.P, as_split(F), t, as_split(b),
                                                           as_split(f1), J);
                } else {
                    M::fd_clear(J);
                    M::template rhs2_fd_jacobian<models::F64>(as_split(yz), tn, PS, a.P, as_split(F), t, as_split(b),
                                                              as_split(f1), J);
                }
                if (prev_pending) {
                    for (int i = 0; i < n; ++i)
                        prev[i] = (1 - sp.theta) * b[i];
                    prev_pending = false;
                }
            }
        } else {
            rhs64<M>(yz, tn, a.P, F, f1);
        }
        for (int i = 0; i < n; ++i)
            b[i] = -z1[i] * 1.0 + ldt * (prev[i] + alpha * f1[i]);
        residual = l2norm<n>(b);
        if (relative_residual < sp.relative_tolerance) {
            newton_done = true;
        } else {
            if (recompute || always) {
                M::lu_shift(J, -ldt * alpha);
                M::lu_factorize(J);
                jac_comp += 1;
                recompute = 0;
            }
            M::lu_solve(J, b, b);
            if (newton_iterations == 0) {
                initial_residual = residual;
                eta = eta > kGossEps ? eta : kGossEps;
                eta = pow_0_8(eta);
            } else {
                relative_previous_residual = models::f64_div(residual, previous_residual);
                recompute = relative_previous_residual >= sp.max_relative_previous_residual;
                if (relative_previous_residual >= 1) {
                    step_ok = false;
                    rejects += 1;
                    recompute = 1;
                    newton_done = true;
                } else {
                    const double scaled = std_max(
                        pow_int(relative_previous_residual, sp.max_iterations - newton_iterations), kGossEps);
                    const double limit = sp.kappa * sp.relative_tolerance * (1 - relative_previous_residual);
                    if (residual > models::f64_div(limit, scaled))
                        recompute = 1;
                    eta = models::f64_div(relative_previous_residual, 1.0 - relative_previous_residual);
                }
            }
            if (!newton_done && newton_iterations > sp.max_iterations) {
                recompute = 1;
                rejects += 1;
                step_ok = false;
                newton_done = true;
            }
            if (!newton_done) {
                for (int i = 0; i < n; ++i)
                    z1[i] += b[i];
                relative_residual = models::f64_div(residual, initial_residual);
                previous_residual = residual;
                newton_iterations++;
                newton_done = !(eta * relative_residual >= sp.kappa * sp.relative_tolerance);
            }
        }
        if (!newton_done)
            continue;
        in_step = false;
        if (step_ok) {
            for (int i = 0; i < n; ++i)
                y[i] += z1[i];
            t += ldt;
            accepted += 1;
            if (fabs(t - t_end) < eps) {
                done = true;
                continue;
            }
            if (!justrefined) {
                const double tmp = 2.0 * ldt;
                if (ldt_0 > 0. && tmp >= ldt_0)
                    ldt = ldt_0;
                else
                    ldt = tmp;
            } else {
                justrefined = 0;
            }
            if ((t + ldt + kGossEps) > t_end)
                ldt = t_end - t;
        } else {
            ldt /= 2.0;
            if (ldt < sp.min_dt) {
                status |= GOSS_FLAG_NEWTON_FAILED;
                done = true;
                continue;
            }
            if (IE)
                recompute = 1;
            justrefined = 1;
            num_refinements += 1;
        }
    }
    if (!active)
        return;
    bool finite = true;
    for (int i = 0; i < n; ++i) {
        a.states[i * a.ld + node] = y[i];
        finite = finite && isfinite(y[i]);
    }
    if (!finite)
        status |= GOSS_FLAG_NONFINITE;
    if constexpr (IE) {
#pragma unroll
        for (int k = 0; k < M::lu_nnz; ++k)
            jrows[(uint64_t)k * ld] = J[k];
    }
    ss[TH_ETA * ld] = eta;
    ss[TH_RECOMPUTE * ld] = recompute;
    ss[TH_ALWAYS * ld] = always;
    ss[TH_JUSTREFINED * ld] = justrefined;
    ss[TH_JACCOMP * ld] = jac_comp;
    ss[TH_REJECTS * ld] = rejects;
    ss[TH_ACCEPTED * ld] = accepted;
    if (status) {
        a.node_status[node] |= status;
        atomicOr(a.flags, (uint32_t)status);
    }
}

// ---------------------------------------------------------------------------
// ESDIRK23a
// ---------------------------------------------------------------------------
enum EsdirkRows {
    ES_PREV_DT = 0, ES_LOC_ERROR, ES_ETA, ES_NEWTON_IT, ES_FIRST, ES_NEWJAC, ES_JACCOMP, ES_REJECTS, ES_ACCEPTED,
    ES_SCALARS  // then the packed jac and jfac, each lu_nnz x ld values tiled [ld/32][lu_nnz][32]
};

struct EsdirkCoef {
    double gamma, a21, a22, a31, a32, a33, a41, a42, a43, a44, b1, b2, b3, b4, bh1, bh2, bh3, c2, c3, c4;
    double s_fac, tol, etamin, kappa;
};

// ESDIRK23a constructor (ESDIRK23a.cpp:27-39)
__device__ __forceinline__ EsdirkCoef esdirk_coefficients()
{
    EsdirkCoef c;
    const double gamma = 0.43586652150845899942;
    c.gamma = gamma;
    c.a21 = gamma;
    c.a22 = gamma;
    c.a31 = (-4 * gamma * gamma + 6 * gamma - 1) / (4 * gamma);
    c.a32 = (-2 * gamma + 1) / (4 * gamma);
    c.a33 = gamma;
    c.a41 = (6 * gamma - 1) / (12 * gamma);
    c.a42 = -1 / ((24 * gamma - 12) * gamma);
    c.a43 = (-6 * gamma * gamma + 6 * gamma - 1) / (6 * gamma - 3);
    c.a44 = gamma;
    c.b1 = c.a41;
    c.b2 = c.a42;
    c.b3 = c.a43;
    c.b4 = c.a44;
    c.bh1 = c.a31;
    c.bh2 = c.a32;
    c.bh3 = c.a33;
    c.c2 = 2.0 * gamma;
    c.c3 = 1.0;
    c.c4 = 1.0;
    c.s_fac = 0.9;
    c.tol = 1.0e-5;
    c.etamin = 1.0e-10;
    c.kappa = 1.0e-1;
    return c;
}

// ESDIRK23a as one loop per node in which every pass evaluates the right-hand
// side at most once and runs at most one substitution with the factorised
// matrix, whatever phase of the method the node is in: the start of a step
// attempt (f(y, t), the first stage), a Newton iteration of stage 2, 3 or 4,
// or the error estimate.  The lanes of a warp drift apart in their Newton
// iteration and step counts; in the nested form each lane then runs a
// different inlined copy of the stage loop and the warp executes the copies
// one after the other, here they share one copy of the model code.  The
// Jacobian (at most once per pass) and the factorisation follow the same rule.
// Per node the operations and their order are the nested form's
// (ESDIRK23a::forward, advance_one_step, do_step, compute_stage_val,
// reduce_time_step; ESDIRK23a.cpp:101-316).
// The passes run in block lockstep (a block barrier after each pass, until
// every node of the block has finished the interval), so the block's warps
// walk the large straight-line pass code together and share its
// instruction-cache lines, at the cost of waiting for the block's slowest
// node.  Measured on B200 (TT04, 262,144 nodes, 0.1 ms intervals, the same
// states): with the analytic Jacobian 17.5 ms per interval without barriers,
// 14.4 / 11.8 / 10.2 ms in lockstep blocks of 64 / 128 / 256 where steps are
// accepted (min_dt 1e-4), 284 ms against 231 / 173 / 136 ms where every
// attempt is rejected (default min_dt); with forward differences 18.4 against
// 15.0 / 12.4 / 10.7 ms and 354 against 302 / 211 / 156 ms.
#ifndef GOSS_ESDIRK_THREADS
#define GOSS_ESDIRK_THREADS 256
#endif
#ifndef GOSS_ESDIRK_MIN_BLOCKS
#define GOSS_ESDIRK_MIN_BLOCKS 1
#endif
#ifndef GOSS_ESDIRK_REUSE_F
#define GOSS_ESDIRK_REUSE_F 1
#endif
template <class M, bool J32 = false>
__global__ void __launch_bounds__(GOSS_ESDIRK_THREADS, GOSS_ESDIRK_MIN_BLOCKS)
    esdirk_kernel(const __grid_constant__ ImplicitArgs<M> a)
{
    constexpr int n = M::num_states;
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = gid < a.N;
    // threads past the last node shadow it (reads only) and take part in the barriers
    const uint32_t node = active ? gid : a.N - 1;
    const uint64_t ld = a.ld;
    double y[n];
    for (int i = 0; i < n; ++i)
        y[i] = a.states[i * ld + node];
    double F[Dims<M>::nfp];
    load_field<M, double>(a.fparams, ld, node, F);
    double* ss = a.sstate + node;
    const EsdirkCoef c = esdirk_coefficients();
    const goss_solver_params& sp = a.sp;
    const models::F64* const PS = as_split(a.P);
    const PackedTile jac = packed_tile(a.sstate + (uint64_t)ES_SCALARS * ld, node, M::lu_nnz);
    const PackedTile jfac = packed_tile(a.sstate + (uint64_t)(ES_SCALARS + M::lu_nnz) * ld, node, M::lu_nnz);
    double prev_dt = ss[ES_PREV_DT * ld];
    double loc_error = ss[ES_LOC_ERROR * ld];
    double eta = ss[ES_ETA * ld];
    int newton_iterations = (int)ss[ES_NEWTON_IT * ld];
    int first_step = ss[ES_FIRST * ld] != 0.0;
    int new_jacobian = ss[ES_NEWJAC * ld] != 0.0;
    double jac_comp = ss[ES_JACCOMP * ld], rejects = ss[ES_REJECTS * ld], accepted = ss[ES_ACCEPTED * ld];

    // stage derivatives z1, z2, z3 and the current stage's z (z2, z3 or z4)
    double z1[n], z2[n], z3[n], z[n], prev[n];
    enum { PH_BEGIN = 0, PH_NEWTON = 1, PH_ERROR = 2 };
    int phase = PH_BEGIN, stage = 2;
    double t_step = 0.0, t_s = 0.0, dz_norm = 0.0;
    int newton_guard = 0, advance_guard = 0;
    int jac_pending = 0;  // Jacobians due at the top of the next pass (same y and t)
    double t_jac = 0.0;
    bool fact_pending = false;

    const double t0 = a.t, interval = a.interval;
    const double min_dt = sp.min_dt;
    double local_t = 0;
    uint8_t status = 0;
    uint64_t guard = 0;
    // ESDIRK23a::forward (ESDIRK23a.cpp:280-316)
    double h = std_max(c.s_fac * prev_dt * root4(models::f64_div(c.tol, loc_error)), min_dt);
    h = std_min(h, interval);
    if (first_step) {
        prev_dt = h;
        jac_pending = 1;
        t_jac = t0;
    }
    // top of the while loop of forward: returns false when the interval is done
    auto outer_begin = [&]() -> bool {
        if (!(local_t < interval))
            return false;
        if (++guard > a.max_loop) {
            status |= GOSS_FLAG_ITERATION_CAP;
            return false;
        }
        if (h * 1.1 >= interval - local_t)
            h = interval - local_t;
        if (newton_iterations >= 2) {
            jac_pending += 1;
            t_jac = t0 + local_t;
        }
        if (fabs(models::f64_div(h - prev_dt, prev_dt)) > 0.2 || new_jacobian || jac_pending)
            fact_pending = true;
        t_step = t0 + local_t;
        advance_guard = 0;
        phase = PH_BEGIN;
        return true;
    };
    // compute_stage_val's entry
    auto start_stage = [&](int st, double t_stage) {
        stage = st;
        t_s = t_stage;
        newton_iterations = 0;
        dz_norm = 0.0;
        newton_guard = 0;
        eta = pow_0_8(std_max(eta, c.etamin));
        phase = PH_NEWTON;
    };
    // the end of advance_one_step and of the while loop's body
    auto end_advance = [&]() -> bool {
        new_jacobian = 0;
        prev_dt = h;
        local_t += h;
        h = std_max(c.s_fac * prev_dt * root4(models::f64_div(c.tol, loc_error)), min_dt);
        return outer_begin();
    };
    // do_step returned false: advance_one_step's retry loop
    auto step_failed = [&]() -> bool {
        if (h > min_dt && ++advance_guard < 4096) {
            if (!new_jacobian) {
                jac_pending = 1;
                t_jac = t_step;
            }
            // reduce_time_step (ESDIRK23a.cpp:260-278)
            double reduction_factor = 1.0, e = loc_error;
            int g = 0;
            do {
                reduction_factor *= 0.6;
                e *= 0.1;
            } while (e > c.tol && ++g < 4096);
            h = std_max(reduction_factor * h, min_dt);
            fact_pending = true;
            phase = PH_BEGIN;
            return true;
        }
        return end_advance();
    };

    // block-uniform loop: every pass, a block barrier (see above)
    bool running = active && outer_begin();
    while (__syncthreads_or(running)) {
        if (!running)
            continue;
        // f(y, t_step) of an attempt's first stage, when this pass's Jacobian
        // evaluation produced it (then held in z1)
        bool f_known = false;
        if (jac_pending || fact_pending) {
            // both are due only before an attempt's first stage, which
            // rewrites z1, z and prev before reading them, and z2, z3 before
            // reading them: their old values are dead here, and saying so
            // keeps them out of the registers the Jacobian code needs
#pragma unroll
            for (int i = 0; i < n; i++)
                z1[i] = z2[i] = z3[i] = z[i] = prev[i] = 0.0;
        }
        // ESDIRK23a::compute_ode_jacobian (ESDIRK23a.h:58-63)
        if (jac_pending) {
            double g1[n];  // f(y), a by-product of the fused evaluations
            if constexpr (J32) {
                (void)g1;
                jacobian32<M>(y, t_jac, a.P32, a.P, F, jac);
            } else if constexpr (M::has_jacobian) {
                M::template rhs_jacobian<models::F64>(as_split(y), t_jac, PS, a.P, as_split(F), as_split(g1), jac);
            } else {
                M::fd_clear(jac);
                M::template rhs_fd_jacobian<models::F64>(as_split(y), t_jac, PS, a.P, as_split(F), as_split(g1), jac);
            }
            jac_comp += jac_pending;
            jac_pending = 0;
            new_jacobian = 1;
            // The Jacobian is due only before an attempt's first stage and is
            // taken at that stage's (y, t_step); the evaluation that fused it
            // with f(y) leaves f(y, t_step), which do_step (ESDIRK23a.cpp:
            // 134-140) evaluates once more for z1.  Only the FP32 Jacobian
            // does not produce it.
            if constexpr (!J32 && GOSS_ESDIRK_REUSE_F) {
                if (phase == PH_BEGIN && t_jac == t_step) {
#pragma unroll
                    for (int i = 0; i < n; i++)
                        z1[i] = g1[i];
                    f_known = true;
                }
            }
        }
        // ESDIRK23a::compute_factorized_jacobian(dt) (ESDIRK23a.cpp:101-115)
        if (fact_pending) {
            M::lu_copy_shift(jac, jfac, -h * c.a22);
            M::lu_factorize(jfac);
            fact_pending = false;
        }
        // the pass's right-hand side: f(y, t) at an attempt's start, else
        // f(y + h prev + gamma h z, t_s) of a Newton iteration
        double f[n];
        if (phase != PH_ERROR && !f_known) {
            double x[n];
#pragma unroll
            for (int i = 0; i < n; i++)
                x[i] = phase == PH_BEGIN ? y[i] : y[i] + h * prev[i] + c.gamma * h * z[i];
            rhs64<M>(x, phase == PH_BEGIN ? t_step : t_s, a.P, F, f);
        }
        // the pass's substitution: the Newton update, or the error estimate
        double dz[n];
        if (phase != PH_BEGIN) {
            double v[n];
#pragma unroll
            for (int i = 0; i < n; i++)
                v[i] = phase == PH_NEWTON
                           ? -z[i] + f[i]
                           : h * ((c.b1 - c.bh1) * z1[i] + (c.b2 - c.bh2) * z2[i] + (c.b3 - c.gamma) * z3[i] +
                                  c.gamma * z[i]);
            M::lu_solve(jfac, v, dz);
        }
        if (phase == PH_BEGIN) {
            // do_step: z1 = f(y, t0), z2 = z1, prev = a21 z1
#pragma unroll
            for (int i = 0; i < n; i++) {
                const double fi = f_known ? z1[i] : f[i];
                z1[i] = fi;
                z[i] = fi;
                prev[i] = fi * c.a21;
            }
            start_stage(2, t_step + c.c2 * h);
        } else if (phase == PH_NEWTON) {
            // one iteration of compute_stage_val (ESDIRK23a.cpp:201-258)
            const double prev_dz_norm = dz_norm;
            dz_norm = l2norm<n>(dz);
            bool fail = false;
            if (newton_iterations >= 1) {
                const double theta = models::f64_div(dz_norm, prev_dz_norm);
                if (!(theta <= 1)) {
                    rejects += 1;
                    fail = true;
                } else {
                    eta = models::f64_div(theta, 1.0 - theta);
                }
            }
            if (!fail && (newton_iterations > sp.max_iterations || ++newton_guard > 100000)) {
                rejects += 1;
                fail = true;
            }
            if (fail) {
                running = step_failed();
                continue;
            }
#pragma unroll
            for (int i = 0; i < n; i++)
                z[i] += dz[i];
            newton_iterations++;
            if (!(eta * dz_norm > c.kappa * c.tol)) {
                if (stage == 2) {
#pragma unroll
                    for (int i = 0; i < n; i++) {
                        z2[i] = z[i];
                        prev[i] = z1[i] * c.bh1 + z2[i] * c.bh2;
                    }
                    start_stage(3, t_step + c.c3 * h);
                } else if (stage == 3) {
#pragma unroll
                    for (int i = 0; i < n; i++) {
                        z3[i] = z[i];
                        prev[i] = z1[i] * c.b1 + z2[i] * c.b2 + z3[i] * c.b3;
                    }
                    start_stage(4, t_step + c.c4 * h);
                } else {
                    phase = PH_ERROR;  // z holds z4
                }
            }
        } else {
            // do_step's error test (ESDIRK23a.cpp:180-196)
            loc_error = l2norm<n>(dz);
            if (loc_error > c.tol) {
                rejects += 1;
                running = step_failed();
            } else {
#pragma unroll
                for (int i = 0; i < n; i++)
                    y[i] = y[i] + h * (c.b1 * z1[i] + c.b2 * z2[i] + c.b3 * z3[i] + c.gamma * z[i]);
                accepted += 1;
                running = end_advance();
            }
        }
    }
    if (!active)
        return;
    first_step = 0;
    bool finite = true;
    for (int i = 0; i < n; ++i) {
        a.states[i * ld + node] = y[i];
        finite = finite && isfinite(y[i]);
    }
    if (!finite)
        status |= GOSS_FLAG_NONFINITE;
    ss[ES_PREV_DT * ld] = prev_dt;
    ss[ES_LOC_ERROR * ld] = loc_error;
    ss[ES_ETA * ld] = eta;
    ss[ES_NEWTON_IT * ld] = newton_iterations;
    ss[ES_FIRST * ld] = first_step;
    ss[ES_NEWJAC * ld] = new_jacobian;
    ss[ES_JACCOMP * ld] = jac_comp;
    ss[ES_REJECTS * ld] = rejects;
    ss[ES_ACCEPTED * ld] = accepted;
    if (status) {
        a.node_status[node] |= status;
        atomicOr(a.flags, (uint32_t)status);
    }
}

// ---------------------------------------------------------------------------
// batched model evaluation (ODE::eval / ODE::linearized_eval on many states)
// ---------------------------------------------------------------------------
template <class M, typename T>
__global__ void __launch_bounds__(128) eval_kernel(const __grid_constant__ EvalArgs<M, T> a)
{
    constexpr int n = M::num_states;
    const uint32_t node = blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= a.N)
        return;
    T y[n], o1[n], o2[n];
    for (int i = 0; i < n; ++i)
        y[i] = T(a.states[i * a.ld + node]);
    T F[Dims<M>::nfp];
    load_field<M, T>(a.fparams, a.ld, node, F);
    const double t = a.times[node];
    if (a.what == 0) {
        M::template rhs<T>(y, t, a.P, a.PD, F, o1);
        for (int i = 0; i < n; ++i)
            a.out[i * a.ld + node] = double(o1[i]);
    } else if (a.what == 1) {
        M::template linearized<T>(y, t, a.P, a.PD, F, o1, o2);
        for (int i = 0; i < n; ++i) {
            a.out[i * a.ld + node] = double(o1[i]);
            a.out[(n + i) * a.ld + node] = double(o2[i]);
        }
    } else if (a.what == 2) {
        if constexpr (M::num_monitored > 0) {
            T mon[M::num_monitored];
            M::template monitored_values<T>(y, t, a.P, a.PD, F, mon);
            for (int i = 0; i < M::num_monitored; ++i)
                a.out[i * a.ld + node] = double(mon[i]);
        }
    } else if constexpr (M::has_jacobian) {
        T J[M::lu_nnz];
        M::template jacobian<T>(y, t, a.P, a.PD, F, J);
        M::lu_unpack(J, [&](int k, T v) { a.out[(uint64_t)k * a.ld + node] = double(v); });
    }
}

// ---------------------------------------------------------------------------
// host-side launchers (called through goss_model_desc::launch / ::eval)
// ---------------------------------------------------------------------------
inline unsigned long explicit_num_steps(double ldt_0, double dt)
{
    // e.g. GRL1.cpp:66
    return ldt_0 > 0 ? (unsigned long)ceil(dt / ldt_0 - 1.0E-12) : 1UL;
}

template <class M>
inline uint32_t solver_state_rows(int32_t solver)
{
    if (solver == GOSS_THETA)
        return TH_ROWS;
    if (solver == GOSS_IMPLICIT_EULER)
        return TH_ROWS + M::lu_nnz;
    if (solver == GOSS_ESDIRK23A)
        return ES_SCALARS + 2 * M::lu_nnz;
    return 0;
}

template <class M, typename T, Explicit S>
inline int launch_explicit(const goss_launch* L)
{
    ExplicitArgs<M, T> a;
    a.states = L->states;
    a.fparams = L->field_params;
    a.flags = L->flags;
    a.node_status = L->node_status;
    a.ld = L->ld;
    a.N = L->num_nodes;
    const double ldt_0 = L->solver_params->ldt;
    const unsigned long nsteps = explicit_num_steps(ldt_0, L->interval);
    a.nsteps = nsteps;
    a.ldt = L->interval / nsteps;
    a.t = L->t;
    a.delta = L->solver_params->delta;
    a.schedule = L->schedule;
    a.forwards = L->schedule ? L->forwards : 1u;
    a.out = L->out;
    a.vector = L->vector;
    a.dofs = L->dofs;
    a.num_dofs = L->num_dofs;
    a.num_fields = L->num_fields;
    a.tangled = L->tangled;
    for (int i = 0; i < M::num_states; ++i)
        a.field_of[i] = -1;
    for (uint32_t k = 0; k < L->num_fields; ++k) {
        if (L->field_rows[k] >= (uint32_t)M::num_states || k > 127)
            return GOSS_ERR_ARGUMENT;
        a.field_of[L->field_rows[k]] = (int8_t)k;
    }
    parameter_block<M>(L->params, a.PD);
    for (int i = 0; i < Dims<M>::np; ++i)
        a.P[i] = T(a.PD[i]);
    const unsigned block = L->block ? L->block : 128;
    const unsigned grid = (L->num_nodes + block - 1) / block;
    if (grid == 0)
        return 0;
    const cudaStream_t st = (cudaStream_t)L->stream;
    const bool wide = explicit_two_shapes<T, S> && block == 128 && explicit_blocks<S>(grid) == 2;
    constexpr int wide_blocks = explicit_two_shapes<T, S> ? 2 : ExplicitMinBlocks<T>::value;
    if constexpr (explicit_groups<M, T, S>) {
        // a block size of the user's keeps a thread per node whatever the system's size
        if (!L->block && explicit_in_groups(L->num_nodes, S == Explicit::GRL1 ? a.delta : 1.0)) {
            group_kernel<M, S><<<(L->num_nodes + 31) / 32, 128, 0, st>>>(a);
            return cudaPeekAtLastError() == cudaSuccess ? 0 : GOSS_ERR_CUDA;
        }
    }
    if (L->schedule || L->vector) {
        if constexpr (explicit_extended<S>) {
            if (wide)
                schedule_kernel<M, T, S, wide_blocks><<<grid, block, 0, st>>>(a);
            else
                schedule_kernel<M, T, S, ExplicitMinBlocks<T>::value><<<grid, block, 0, st>>>(a);
        } else {
            return GOSS_ERR_UNSUPPORTED;
        }
    } else if (wide) {
        explicit_kernel<M, T, S, wide_blocks><<<grid, block, 0, st>>>(a);
    } else {
        explicit_kernel<M, T, S, ExplicitMinBlocks<T>::value><<<grid, block, 0, st>>>(a);
    }
    return cudaPeekAtLastError() == cudaSuccess ? 0 : GOSS_ERR_CUDA;
}

// Threads per block of the lockstep kernels, whose blocks of up to 256 threads
// fill an SM one at a time: as many waves as blocks of 256 take, the nodes
// spread evenly over their SMs (a multiple of 32).  Fewer warps on an SM pass
// faster, and a smaller block waits for fewer nodes.  Against blocks of 256
// (TT04 with the analytic Jacobian, ImplicitEuler / ESDIRK23a, us per 0.1 ms
// interval): 1,000 nodes, blocks of 32: 100 -> 64 / 696 -> 335; 8,000, 64: 104
// -> 73 / 788 -> 427; 20,011, 160: 105 -> 87 / 807 -> 676; 50,000, 192: 202 ->
// 179 / 1527 -> 1413; ThetaSolver 3-9 % throughout.
inline unsigned lockstep_block(uint32_t num_nodes, unsigned most)
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        return most;
    const uint64_t wave = (uint64_t)most * sms, waves = ((uint64_t)num_nodes + wave - 1) / wave;
    const uint64_t per = waves ? (num_nodes + waves * sms - 1) / (waves * sms) : 1;
    return (unsigned)((per + 31) / 32 * 32);
}

template <class M>
inline int launch_implicit(const goss_launch* L)
{
    ImplicitArgs<M> a;
    a.states = L->states;
    a.fparams = L->field_params;
    a.sstate = L->solver_state;
    a.flags = L->flags;
    a.node_status = L->node_status;
    a.ld = L->ld;
    a.N = L->num_nodes;
    a.t = L->t;
    a.interval = L->interval;
    a.sp = *L->solver_params;
    a.max_loop = L->max_loop ? L->max_loop : (1ull << 24);
    parameter_block<M>(L->params, a.P);
    for (int i = 0; i < Dims<M>::np; ++i)
        a.P32[i] = float(a.P[i]);
    // GOSS_FP32: the analytic Jacobian in FP32 (models generated with it)
    const bool j32 = L->precision == GOSS_FP32;
    if (j32 && !M::has_jacobian)
        return GOSS_ERR_UNSUPPORTED;
    // lockstep blocks of at most 256 (the kernels' limit)
    const bool theta = L->solver == GOSS_THETA || L->solver == GOSS_IMPLICIT_EULER;
    const unsigned most = theta ? GOSS_THETA_THREADS : GOSS_ESDIRK_THREADS;
    const unsigned block = L->block ? L->block : lockstep_block(L->num_nodes, most);
    if (block > most)
        return GOSS_ERR_ARGUMENT;
    const unsigned grid = (L->num_nodes + block - 1) / block;
    if (grid == 0)
        return 0;
    const cudaStream_t st = (cudaStream_t)L->stream;
    if (j32) {
        if constexpr (M::has_jacobian) {
            if (L->solver == GOSS_THETA)
                theta_kernel<M, false, true><<<grid, block, 0, st>>>(a);
            else if (L->solver == GOSS_IMPLICIT_EULER)
                theta_kernel<M, true, true><<<grid, block, 0, st>>>(a);
            else
                esdirk_kernel<M, true><<<grid, block, 0, st>>>(a);
        }
    } else if (L->solver == GOSS_THETA) {
        theta_kernel<M, false><<<grid, block, 0, st>>>(a);
    } else if (L->solver == GOSS_IMPLICIT_EULER) {
        theta_kernel<M, true><<<grid, block, 0, st>>>(a);
    } else {
        esdirk_kernel<M><<<grid, block, 0, st>>>(a);
    }
    return cudaPeekAtLastError() == cudaSuccess ? 0 : GOSS_ERR_CUDA;
}

template <class M>
inline int launch_solver(const goss_launch* L)
{
    const bool f32 = L->precision == GOSS_FP32;
    if (L->precision == GOSS_FP64_PRINTED)
        return L->solver == GOSS_GRL1 ? launch_explicit<M, double, Explicit::GRL1Printed>(L) : GOSS_ERR_UNSUPPORTED;
    switch (L->solver) {
    case GOSS_EXPLICIT_EULER:
        return f32 ? launch_explicit<M, float, Explicit::Euler>(L) : launch_explicit<M, double, Explicit::Euler>(L);
    case GOSS_RK4:
        return f32 ? launch_explicit<M, float, Explicit::RK4>(L) : launch_explicit<M, double, Explicit::RK4>(L);
    case GOSS_GRL1:
        return f32 ? launch_explicit<M, float, Explicit::GRL1>(L) : launch_explicit<M, double, Explicit::GRL1>(L);
    case GOSS_GRL2:
        return f32 ? launch_explicit<M, float, Explicit::GRL2>(L) : launch_explicit<M, double, Explicit::GRL2>(L);
    case GOSS_RL1:
        return f32 ? launch_explicit<M, float, Explicit::RL1>(L) : launch_explicit<M, double, Explicit::RL1>(L);
    case GOSS_RL2:
        return f32 ? launch_explicit<M, float, Explicit::RL2>(L) : launch_explicit<M, double, Explicit::RL2>(L);
    case GOSS_RK2:
        return f32 ? launch_explicit<M, float, Explicit::RK2>(L) : launch_explicit<M, double, Explicit::RK2>(L);
    case GOSS_THETA:
    case GOSS_ESDIRK23A:
    case GOSS_IMPLICIT_EULER:
        return launch_implicit<M>(L);
    default:
        return GOSS_ERR_ARGUMENT;
    }
}

template <class M, typename T>
inline int launch_eval_t(const goss_eval_launch* L)
{
    EvalArgs<M, T> a;
    a.states = L->states;
    a.fparams = L->field_params;
    a.times = L->times;
    a.out = L->out;
    a.ld = L->ld;
    a.N = L->num_nodes;
    a.what = L->what;
    parameter_block<M>(L->params, a.PD);
    for (int i = 0; i < Dims<M>::np; ++i)
        a.P[i] = T(a.PD[i]);
    const unsigned block = 128;
    const unsigned grid = (L->num_nodes + block - 1) / block;
    if (grid == 0)
        return 0;
    eval_kernel<M, T><<<grid, block, 0, (cudaStream_t)L->stream>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 0 : GOSS_ERR_CUDA;
}

template <class M>
inline int launch_eval(const goss_eval_launch* L)
{
    return L->precision == GOSS_FP32 ? launch_eval_t<M, float>(L) : launch_eval_t<M, double>(L);
}

}  // namespace goss_b200
#endif
