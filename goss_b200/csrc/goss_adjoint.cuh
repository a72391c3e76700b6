// Adjoint of GRL1 and RK4 trajectories with checkpointing (one thread per node).
//
// Forward (record_kernel): the reference's user loop
//     for j in 0..J-1:  forward(t0 + j*interval, interval)   (S internal
//                       steps, GRL1.cpp:61-82 / RK4.cpp:68-102)
// storing the traced state after every interval (the trace) and the full
// state every K internal steps (checkpoints; K a multiple of S).  Each step
// is explicit_step of goss_kernels.cuh, the arithmetic of the solver kernels with
// a thread per node.
//
// Backward (adjoint_kernel): given the cotangent of the trace, walk the
// checkpoint segments from last to first; recompute each segment's K states
// into per-node scratch, then apply the transposed Jacobian of every step in
// reverse, adding the trace cotangent to the traced state's lambda at every
// sample and accumulating the field-parameter gradient.
//
// GRL1:  Phi_i(y) = y_i + b_i h phi1(a_i h),   (a, b) = linearized(y, t)
//     lambda <- lambda + [abar^T d a/dy + bbar^T d b/dy]
//     abar_i = lambda_i b_i h^2 phi1'(a_i h),  bbar_i = lambda_i h phi1(a_i h)
// with the generated linearized_vjp for the bracket.  phi1(x) = (e^x - 1)/x
// is the same function as the reference's b/a (e^{a h} - 1); the derivative
// uses the smooth phi1 form.
//
// RK4:   y' = y + h/6 (k1 + 2 k2 + 2 k3 + k4),  k_s = f(u_s, t_s),
//        u_1 = y, u_2 = y + h/2 k1, u_3 = y + h/2 k2, u_4 = y + h k3
// reversed stage by stage with the generated rhs_vjp:
//     kbar_4 = h/6 lambda;  ubar_s = (df/du)(u_s)^T kbar_s;
//     kbar_{s-1} = w_{s-1} lambda + c_s ubar_s  (w = h/6, h/3, h/3; c = h/2, h/2, h)
//     lambda <- lambda + sum_s ubar_s
// after recomputing k1..k3 from the step's input state.
#ifndef GOSS_ADJOINT_CUH
#define GOSS_ADJOINT_CUH

#include "goss_kernels.cuh"

// Launch shape of the adjoint kernel per arithmetic type: the largest threads
// per block (a multiple of 32, at most 256) and the minimum resident blocks
// per SM it is compiled for (its register cap is 65536 / (threads * blocks)).
// In FP64 the warps of a block synchronise after every step of the recompute and
// reverse loops, so they walk the large straight-line step code together and
// share instruction-cache lines (65,536 nodes x 200 GRL1 steps 7.37 -> 7.22 ms,
// 30,000 nodes x 100 RK4 steps 9.09 -> 7.78); FP32, whose step code is a third
// as long, is faster without (65,536 x 1,000 GRL1 steps 9.64 -> 9.37 ms).
// Measured on B200
// (ten Tusscher-Panfilov, 65,536 nodes x 2,000 steps, backward pass):
//   FP32: blocks of up to 128 threads, 2 per SM (255 registers)
//         28.0 ms; 256 x 1: 29.3 ms; register caps of 168 or 128 (3 or 4
//         blocks of 128) spill more than the extra warps gain: 37.5 ms (with
//         the record's tape 2.0-2.3x the time);
//   FP64: 256 x 1: 207 ms; 128 x 2: 215 ms.
// Since then (65,536 nodes x 1,000 steps, taped): FP32 10.87 -> 9.64 ms with
// the step's seeds (phi1 and its derivative of every state) in packed FP32
// under one branch; FP64, 200 steps, 17.1 -> 10.1 ms with the sweeps on
// models::F64, whose division, exp and log have no branches.
// (the shape of the backward follows the arithmetic of its VJPs)
template <typename T>
struct AdjointShape {
    static constexpr unsigned block = sizeof(T) == 4 ? 128 : 256;
    static constexpr unsigned min_blocks = sizeof(T) == 4 ? 2 : 1;
    static constexpr bool lockstep = sizeof(T) == 8;
};

namespace goss_b200 {

// phi1(x) = (e^x - 1)/x and phi1'(x) = (e^x (x - 1) + 1)/x^2.  FP64, |x| < 1/8:
// f64_phi1_small and the Taylor series sum_k (k+1) x^k/(k+2)! to x^9
// (truncation 4e-17 relative), even and odd terms apart; closed forms beyond.
__device__ __forceinline__ double dphi1d_small(double x)
{
    const double g = x * x;
    double a = 9.0 / 3628800.0, b = 10.0 / 39916800.0;
    a = fma(a, g, 7.0 / 40320.0);
    b = fma(b, g, 8.0 / 362880.0);
    a = fma(a, g, 5.0 / 720.0);
    b = fma(b, g, 6.0 / 5040.0);
    a = fma(a, g, 3.0 / 24.0);
    b = fma(b, g, 4.0 / 120.0);
    a = fma(a, g, 0.5);
    b = fma(b, g, 2.0 / 6.0);
    return fma(b, x, a);
}

// FP32: Taylor series to x^7 for |x| < 1/4 (truncation < 2e-9), closed forms otherwise
template <typename V>
__device__ __forceinline__ V dphi1f_small(V x)
{
    // sum_{k=0}^{7} (k+1) x^k / (k+2)!
    V p = V(8.0f / 362880.0f);
    p = vfma(p, x, V(7.0f / 40320.0f));
    p = vfma(p, x, V(6.0f / 5040.0f));
    p = vfma(p, x, V(5.0f / 720.0f));
    p = vfma(p, x, V(4.0f / 120.0f));
    p = vfma(p, x, V(3.0f / 24.0f));
    p = vfma(p, x, V(2.0f / 6.0f));
    return vfma(p, x, V(0.5f));
}
__device__ __forceinline__ float dphi1f_large(float x)
{
    return __fdividef(__expf(x) * (x - 1.0f) + 1.0f, x * x);
}

// Cotangents of the linear coefficients and right-hand sides of one GRL1 step:
// bbar_i = lambda_i h phi1(a_i h), abar_i = lambda_i b_i h^2 phi1'(a_i h).
// FP64 in groups of four states under one branch (as grl_increments).
template <int N>
__device__ __forceinline__ void grl1_seed_group(const double* lv, const double* lin, const double* rhs, double h,
                                                double* abar, double* bbar)
{
    double x[N], p[N], d[N];
    int far = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        x[i] = lin[i] * h;
        p[i] = models::f64_phi1_small(x[i]);
        d[i] = dphi1d_small(x[i]);
        far = max(far, __double2hiint(x[i]) & 0x7fffffff);
    }
    if (far >= 0x3fc00000) {  // |x| >= 1/8, infinite or NaN
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if ((__double2hiint(x[i]) & 0x7fffffff) >= 0x3fc00000) {
                const double e = models::f64_exp(x[i]), r = models::f64_rcp(x[i]);
                p[i] = (e - 1.0) * r;
                d[i] = (e * (x[i] - 1.0) + 1.0) * (r * r);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        bbar[i] = lv[i] * h * p[i];
        abar[i] = lv[i] * rhs[i] * h * h * d[i];
    }
}

template <int n>
__device__ __forceinline__ void grl1_seed(const double* lv, const double* lin, const double* rhs, double h,
                                          double* abar, double* bbar)
{
    constexpr int rest = n % 4;
#pragma unroll
    for (int i = 0; i + 4 <= n; i += 4)
        grl1_seed_group<4>(lv + i, lin + i, rhs + i, h, abar + i, bbar + i);
    if constexpr (rest != 0)
        grl1_seed_group<rest>(lv + n - rest, lin + n - rest, rhs + n - rest, h, abar + n - rest, bbar + n - rest);
}

// FP32: two states at a time in packed arithmetic, all under one branch; the
// operations of the scalar form in its order.
template <int n>
__device__ __forceinline__ void grl1_seed(const float* lv, const float* lin, const float* rhs, float h, float* abar,
                                          float* bbar)
{
    constexpr int pairs = n / 2, P = pairs > 0 ? pairs : 1;
    const F32x2 hh(h);
    F32x2 p[P], d[P];
    float far[P], all = 0.0f;
#pragma unroll
    for (int i = 0; i < pairs; ++i) {
        const F32x2 x = F32x2(lin[2 * i], lin[2 * i + 1]) * hh;
        float x0, x1;
        x.unpack(x0, x1);
        p[i] = phi1f_small(x);
        d[i] = dphi1f_small(x);
        far[i] = fmaxf(fabsf(x0), fabsf(x1));
        all = fmaxf(all, far[i]);
    }
    if (all >= 0.25f) {
#pragma unroll
        for (int i = 0; i < pairs; ++i) {
            if (far[i] >= 0.25f) {
                const float x0 = lin[2 * i] * h, x1 = lin[2 * i + 1] * h;
                float p0, p1, d0, d1;
                p[i].unpack(p0, p1);
                d[i].unpack(d0, d1);
                const bool n0 = fabsf(x0) < 0.25f, n1 = fabsf(x1) < 0.25f;
                p[i] = F32x2(n0 ? p0 : phi1f_large(x0), n1 ? p1 : phi1f_large(x1));
                d[i] = F32x2(n0 ? d0 : dphi1f_large(x0), n1 ? d1 : dphi1f_large(x1));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < pairs; ++i) {
        const F32x2 l(lv[2 * i], lv[2 * i + 1]);
        (l * hh * p[i]).unpack(bbar[2 * i], bbar[2 * i + 1]);
        (l * F32x2(rhs[2 * i], rhs[2 * i + 1]) * hh * hh * d[i]).unpack(abar[2 * i], abar[2 * i + 1]);
    }
    if constexpr (n % 2 != 0) {
        const float x = lin[n - 1] * h;
        const bool near = fabsf(x) < 0.25f;
        bbar[n - 1] = lv[n - 1] * h * (near ? phi1f_small(x) : phi1f_large(x));
        abar[n - 1] = lv[n - 1] * rhs[n - 1] * h * h * (near ? dphi1f_small(x) : dphi1f_large(x));
    }
}

template <class M, typename T>
struct AdjointArgs {
    double* states;            // [n][ld] in: initial, out: final (record)
    const double* fparams;     // [nfp][ld]
    void* checkpoints;         // [C][2n][ld] float (FP32: hi, lo) or [C][n][ld] double
    double* trace;             // [J][ld]
    const double* trace_bar;   // [J][ld]
    T* scratch;                // [K][n][sld] ([K][4 n][sld] with keep_stages), sld = num_nodes rounded up to 256, plus 256
    T* tape;                   // [taped_segments][K][n][sld]: step inputs of the last segments
    double* fparams_bar;       // [nfp][ld]
    double* states_bar;        // [n][ld]
    uint32_t* flags;
    uint64_t ld;
    uint64_t sld;              // scratch row stride (>= grid * block)
    uint32_t N;
    uint32_t num_intervals;    // J
    uint32_t steps_per_interval;  // S
    uint32_t checkpoint_every;    // K (multiple of S)
    uint32_t trace_state;
    uint32_t taped_segments;
    double t0;
    double interval;
    T P[Dims<M>::np];
    double PD[Dims<M>::np];
};

// checkpoint I/O for the accumulators
__device__ __forceinline__ void cp_store(void* cp, uint64_t idx_hi, uint64_t idx_lo, const Acc<double>& a)
{
    static_cast<double*>(cp)[idx_hi] = a.y;
    (void)idx_lo;
}
__device__ __forceinline__ void cp_store(void* cp, uint64_t idx_hi, uint64_t idx_lo, const Acc<float>& a)
{
    static_cast<float*>(cp)[idx_hi] = a.hi;
    static_cast<float*>(cp)[idx_lo] = a.lo;
}
__device__ __forceinline__ void cp_load(const void* cp, uint64_t idx_hi, uint64_t idx_lo, Acc<double>& a)
{
    a.y = static_cast<const double*>(cp)[idx_hi];
    (void)idx_lo;
}
__device__ __forceinline__ void cp_load(const void* cp, uint64_t idx_hi, uint64_t idx_lo, Acc<float>& a)
{
    a.hi = static_cast<const float*>(cp)[idx_hi];
    a.lo = static_cast<const float*>(cp)[idx_lo];
}

// GRL1 threshold of the reference (GRL1.h:39) used by the traces
constexpr double kGrlDelta = 1e-8;

template <typename T>
__host__ __device__ constexpr int cp_rows(int n)
{
    return sizeof(T) == 4 ? 2 * n : n;
}

template <class M, typename T, Explicit S>
__global__ void __launch_bounds__(128) record_kernel(const __grid_constant__ AdjointArgs<M, T> a)
{
    constexpr int n = M::num_states;
    const uint32_t node = blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= a.N)
        return;
    Acc<T> y[n];
    for (int i = 0; i < n; ++i)
        y[i].load(a.states[i * a.ld + node]);
    T F[Dims<M>::nfp];
    load_field<M, T>(a.fparams, a.ld, node, F);
    const uint32_t S_ = a.steps_per_interval, K = a.checkpoint_every;
    const double ldt = a.interval / S_;
    constexpr int rows = cp_rows<T>(n);
    // the last taped_segments segments keep every step's input state: the
    // values the backward's recompute would write to its scratch
    const uint64_t total = (uint64_t)a.num_intervals * S_;
    const uint64_t num_cp = (total + K - 1) / K;
    const uint64_t tape_from = (num_cp - a.taped_segments) * K;
    T* const tape = a.tape + node;
    for (uint32_t j = 0; j < a.num_intervals; ++j) {
        const uint64_t g = (uint64_t)j * S_;
        if (g % K == 0) {
            const uint64_t c = g / K;
            for (int i = 0; i < n; ++i)
                cp_store(a.checkpoints, ((c * rows) + i) * a.ld + node, ((c * rows) + n + i) * a.ld + node, y[i]);
        }
        double lt = a.t0 + j * a.interval;
        for (uint32_t s = 0; s < S_; ++s) {
            if (g + s >= tape_from) {
                const uint64_t row = (g + s - tape_from) * n;
                for (int i = 0; i < n; ++i)
                    tape[(row + i) * a.sld] = y[i].value();
            }
            explicit_step<M, T, S>(y, lt, ldt, a.P, a.PD, F, T(kGrlDelta));
            lt += ldt;
        }
        a.trace[(uint64_t)j * a.ld + node] = y[a.trace_state].store();
    }
    bool finite = true;
    for (int i = 0; i < n; ++i) {
        const double v = y[i].store();
        a.states[i * a.ld + node] = v;
        finite = finite && isfinite(v);
    }
    if (!finite)
        atomicOr(a.flags, GOSS_FLAG_NONFINITE);
}

// lambda <- lambda + (dPhi/dy)(y)^T lambda - lambda for one GRL1 step, and the
// field-parameter part into gF
template <class M, typename T>
__device__ __forceinline__ void reverse_step_grl1(const T* yt, double lt, double ldt, const T* P, const double* PD,
                                                  const T* F, Acc<T>* lam, double* gF)
{
    constexpr int n = M::num_states;
    constexpr int nfp = Dims<M>::nfp;
    using V = split_t<T>;
    const T h = T(ldt);
    T lv[n], ybar[n], Fbar[nfp];
    for (int i = 0; i < n; ++i)
        lv[i] = lam[i].value();
    auto seed = [&](const V* lin, const V* rhs, V* abar, V* bbar) {
        grl1_seed<n>(lv, reinterpret_cast<const T*>(lin), reinterpret_cast<const T*>(rhs), h,
                     reinterpret_cast<T*>(abar), reinterpret_cast<T*>(bbar));
    };
    M::template linearized_vjp<V>(as_split(yt), lt, as_split(P), PD, as_split(F), seed, as_split(ybar),
                                  as_split(Fbar));
    for (int i = 0; i < n; ++i)
        lam[i].add(ybar[i]);
    for (int q = 0; q < M::num_field_params; ++q)
        gF[q] += double(Fbar[q]);
}

// the same for one RK4 step; the stage loops are not unrolled, so rhs and
// rhs_vjp are instantiated once.  The stage inputs are formed from the step's
// input value (in FP32 its high word; the forward adds the low word as well,
// a difference of at most half an FP32 ulp of the state).
// kept: the step's first three stage derivatives (rows ld apart) where the
// recompute kept them, which saves evaluating them again here -- the same
// values; FP64, 2,001 nodes x 200 steps 12.6 -> 10.1 ms, 30,000 x 100 9.2 -> 6.7.
template <class M, typename T>
__device__ __forceinline__ void reverse_step_rk4(const T* yt, double lt, double ldt, const T* P, const double* PD,
                                                 const T* F, Acc<T>* lam, double* gF, const T* kept, uint64_t ld)
{
    constexpr int n = M::num_states;
    constexpr int nfp = Dims<M>::nfp;
    const T h = T(ldt), hh = T(0.5 * ldt);
    T k1[n], k2[n], k3[n], u[n];
    if (kept) {
        for (int i = 0; i < n; ++i) {
            k1[i] = kept[i * ld];
            k2[i] = kept[(n + i) * ld];
            k3[i] = kept[(2 * n + i) * ld];
        }
    }
#pragma unroll 1
    for (int st = kept ? 3 : 0; st < 3; ++st) {
        const double ts = st == 0 ? lt : lt + 0.5 * ldt;
        for (int i = 0; i < n; ++i)
            u[i] = st == 0 ? yt[i] : yt[i] + hh * (st == 1 ? k1[i] : k2[i]);
        T k[n];
        model_rhs<M, T>(u, ts, P, PD, F, k);
        for (int i = 0; i < n; ++i) {
            k1[i] = st == 0 ? k[i] : k1[i];
            k2[i] = st == 1 ? k[i] : k2[i];
            k3[i] = st == 2 ? k[i] : k3[i];
        }
    }
    T lv[n], kb[n], ysum[n];
    const T w6 = T(split_t<T>(h) / split_t<T>(6.0)), w3 = T(split_t<T>(h) / split_t<T>(3.0));
    for (int i = 0; i < n; ++i) {
        lv[i] = lam[i].value();
        kb[i] = w6 * lv[i];
        ysum[i] = T(0.0);
    }
#pragma unroll 1
    for (int st = 3; st >= 0; --st) {
        const T c = st == 3 ? h : hh;
        const double ts = st == 3 ? lt + ldt : (st == 0 ? lt : lt + 0.5 * ldt);
        for (int i = 0; i < n; ++i)
            u[i] = st == 0 ? yt[i] : yt[i] + c * (st == 3 ? k3[i] : st == 2 ? k2[i] : k1[i]);
        T ub[n], Fb[nfp];
        auto seed = [&](const split_t<T>*, split_t<T>* bbar) {
#pragma unroll
            for (int i = 0; i < n; ++i)
                bbar[i] = split_t<T>(kb[i]);
        };
        M::template rhs_vjp<split_t<T>>(as_split(u), ts, as_split(P), PD, as_split(F), seed, as_split(ub),
                                        as_split(Fb));
        const T w = st == 1 ? w6 : w3;
        for (int i = 0; i < n; ++i) {
            ysum[i] = ysum[i] + ub[i];
            kb[i] = w * lv[i] + c * ub[i];
        }
        for (int q = 0; q < M::num_field_params; ++q)
            gF[q] += double(Fb[q]);
    }
    for (int i = 0; i < n; ++i)
        lam[i].add(ysum[i]);
}

// R is the arithmetic of the step VJPs and of lambda: T, or double over an
// FP32 trajectory (the recompute keeps T, so the same trajectory is
// differentiated; only the VJP arithmetic changes).
// Keep: the recompute keeps RK4's stage derivatives in scratch (a kernel of its
// own: where it has none to read, the choice at run time cost 5 %).
template <class M, typename T, Explicit S, typename R = T, bool Keep = false>
__global__ void __launch_bounds__(AdjointShape<R>::block, AdjointShape<R>::min_blocks)
adjoint_kernel(const __grid_constant__ AdjointArgs<M, T> a)
{
    constexpr int n = M::num_states;
    constexpr int nfp = Dims<M>::nfp;
    static_assert(sizeof(R) >= sizeof(T), "the VJP arithmetic is at least the trajectory's");
    // Every thread runs every loop (block-wide barriers below); threads past
    // the last node shadow it (reads only) and keep their own scratch column.
    const uint32_t node = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = node < a.N;
    const uint32_t src = active ? node : a.N - 1;
    extern __shared__ double s_time[];  // time of every step of a segment (same for all nodes)
    const uint32_t S_ = a.steps_per_interval, K = a.checkpoint_every;
    const double ldt = a.interval / S_;
    T F[nfp];
    load_field<M, T>(a.fparams, a.ld, src, F);
    R FR[nfp];
    load_field<M, R>(a.fparams, a.ld, src, FR);
    const R* PR;
    if constexpr (sizeof(R) == sizeof(T))
        PR = reinterpret_cast<const R*>(a.P);
    else
        PR = a.PD;
    Acc<R> lam[n];
    for (int i = 0; i < n; ++i)
        lam[i].load(0.0);
    double gF[nfp];
    for (int k = 0; k < nfp; ++k)
        gF[k] = 0.0;
    const uint64_t total = (uint64_t)a.num_intervals * S_;
    const uint32_t num_cp = (uint32_t)((total + K - 1) / K);
    constexpr int rows = cp_rows<T>(n);
    T* const scratch = a.scratch + node;
    for (int c = (int)num_cp - 1; c >= 0; --c) {
        const uint64_t g0 = (uint64_t)c * K;
        const uint32_t len = (uint32_t)((g0 + K <= total) ? K : total - g0);
        // times of the segment's steps, exactly as the forward accumulated them
        __syncthreads();
        if (threadIdx.x == 0) {
            double lt = 0.0;
            for (uint32_t k = 0; k < len; ++k) {
                const uint64_t g = g0 + k;
                if (g % S_ == 0)
                    lt = a.t0 + (g / S_) * a.interval;
                s_time[k] = lt;
                lt += ldt;
            }
        }
        __syncthreads();
        // the input state of every step of the segment: from the record's
        // tape, or recomputed from the checkpoint into scratch
        const T* seg = scratch;
        [[maybe_unused]] bool kept = Keep;
        if ((uint32_t)c >= num_cp - a.taped_segments) {
            kept = false;
            seg = a.tape + (uint64_t)(c - (num_cp - a.taped_segments)) * K * n * a.sld + src;
        } else {
            Acc<T> y[n];
            for (int i = 0; i < n; ++i)
                cp_load(a.checkpoints, ((uint64_t)c * rows + i) * a.ld + src,
                        ((uint64_t)c * rows + n + i) * a.ld + src, y[i]);
            for (uint32_t k = 0; k < len; ++k) {
                for (int i = 0; i < n; ++i)
                    scratch[((uint64_t)k * (Keep ? 4 * n : n) + i) * a.sld] = y[i].value();
                if constexpr (Keep) {
                    // the last step's stages are needed too
                    explicit_step<M, T, S>(y, s_time[k], ldt, a.P, a.PD, F, T(kGrlDelta), [&](int st, const T* kst) {
                        if (st < 3)
                            for (int i = 0; i < n; ++i)
                                scratch[((uint64_t)k * 4 * n + (st + 1) * n + i) * a.sld] = kst[i];
                    });
                } else if (k + 1 < len) {
                    explicit_step<M, T, S>(y, s_time[k], ldt, a.P, a.PD, F, T(kGrlDelta));
                }
                if constexpr (AdjointShape<R>::lockstep)
                    __syncthreads();
            }
        }
        // reverse through the segment
        for (int k = (int)len - 1; k >= 0; --k) {
            const uint64_t g = g0 + k;  // step g maps state g to state g+1
            if ((g + 1) % S_ == 0) {
                const uint64_t j = (g + 1) / S_ - 1;
                lam[a.trace_state].add(R(a.trace_bar[j * a.ld + src]));
            }
            R yt[n];
            const T* const row = seg + (uint64_t)k * (Keep && kept ? 4 * n : n) * a.sld;
            for (int i = 0; i < n; ++i)
                yt[i] = R(row[i * a.sld]);
            if constexpr (S == Explicit::GRL1)
                reverse_step_grl1<M, R>(yt, s_time[k], ldt, PR, a.PD, FR, lam, gF);
            else if constexpr (Keep)
                reverse_step_rk4<M, R>(yt, s_time[k], ldt, PR, a.PD, FR, lam, gF, kept ? row + n * a.sld : nullptr,
                                       a.sld);
            else
                reverse_step_rk4<M, R>(yt, s_time[k], ldt, PR, a.PD, FR, lam, gF, nullptr, 0);
            if constexpr (AdjointShape<R>::lockstep)
                __syncthreads();
        }
    }
    if (!active)
        return;
    for (int q = 0; q < M::num_field_params; ++q)
        a.fparams_bar[(uint64_t)q * a.ld + node] = gF[q];
    for (int i = 0; i < n; ++i)
        a.states_bar[(uint64_t)i * a.ld + node] = lam[i].store();
}

// Threads per block for the backward kernel: every thread carries one node
// through the whole trajectory, so the job runs in waves of (resident blocks
// x SMs) blocks and its time is about waves x resident warps per SM.  Choose
// the multiple of 32 (<= AdjointShape<T>::block) minimising that product (ties:
// the larger block).  A grid below one wave counts the blocks it puts on an SM,
// not those that would fit: 2,001 nodes in FP64 take blocks of 32 (one warp on
// each of 63 SMs) instead of 256 (eight on each of 8): GRL1 100 steps 1.80 ->
// 1.13 ms, 8,000 nodes (blocks of 64) 1.87 -> 1.19 ms.
template <class M, typename T, Explicit S, typename R = T>
inline unsigned adjoint_block(uint32_t num_nodes, size_t shm)
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        return AdjointShape<R>::block;
    unsigned best = AdjointShape<R>::block;
    uint64_t best_cost = ~0ull;
    for (unsigned b = AdjointShape<R>::block; b >= 32; b -= 32) {
        int active = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&active, adjoint_kernel<M, T, S, R>, (int)b, shm) !=
                cudaSuccess || active <= 0)
            continue;
        const uint64_t grid = (num_nodes + b - 1) / b;
        const uint64_t slots = (uint64_t)active * sms;
        const uint64_t waves = (grid + slots - 1) / slots;
        const uint64_t cost = (waves > 1 ? waves * (uint64_t)active : (grid + sms - 1) / sms) * b;
        if (cost < best_cost) {
            best_cost = cost;
            best = b;
        }
    }
    return best;
}

template <class M, typename T, Explicit S, typename R = T>
inline int launch_adjoint_t(const goss_adjoint_launch* L)
{
    AdjointArgs<M, T> a;
    a.states = L->states;
    a.fparams = L->field_params;
    a.checkpoints = L->checkpoints;
    a.trace = L->trace;
    a.trace_bar = L->trace_bar;
    a.scratch = static_cast<T*>(L->scratch);
    a.tape = static_cast<T*>(L->tape);
    a.taped_segments = L->taped_segments;
    if (L->keep_stages && (S != Explicit::RK4 || sizeof(T) != 8))
        return GOSS_ERR_ARGUMENT;
    a.fparams_bar = L->field_params_bar;
    a.states_bar = L->states_bar;
    a.flags = L->flags;
    a.ld = L->ld;
    a.N = L->num_nodes;
    a.num_intervals = L->num_intervals;
    a.steps_per_interval = L->steps_per_interval;
    a.checkpoint_every = L->checkpoint_every;
    a.trace_state = L->trace_state;
    a.t0 = L->t0;
    a.interval = L->interval;
    parameter_block<M>(L->params, a.PD);
    for (int i = 0; i < Dims<M>::np; ++i)
        a.P[i] = T(a.PD[i]);
    if (a.steps_per_interval == 0 || a.checkpoint_every == 0 || a.checkpoint_every % a.steps_per_interval ||
        a.trace_state >= (uint32_t)M::num_states)
        return GOSS_ERR_ARGUMENT;
    {
        const uint64_t total = (uint64_t)a.num_intervals * a.steps_per_interval;
        const uint64_t num_cp = (total + a.checkpoint_every - 1) / a.checkpoint_every;
        if (a.taped_segments > num_cp || (a.taped_segments && !a.tape))
            return GOSS_ERR_ARGUMENT;
    }
    // room for grid * block <= round_up(num_nodes, block) for any block <= 256
    a.sld = ((uint64_t)L->num_nodes + 255) / 256 * 256 + 256;
    if (L->num_nodes == 0)
        return 0;
    if (L->mode == 0) {
        const unsigned block = 128;
        const unsigned grid = (L->num_nodes + block - 1) / block;
        record_kernel<M, T, S><<<grid, block, 0, (cudaStream_t)L->stream>>>(a);
    } else {
        const size_t shm = sizeof(double) * a.checkpoint_every;
        if (shm > 48 * 1024)
            return GOSS_ERR_ARGUMENT;
        const unsigned block = L->block ? L->block : adjoint_block<M, T, S, R>(L->num_nodes, shm);
        if (block == 0 || block > AdjointShape<R>::block || block % 32)
            return GOSS_ERR_ARGUMENT;
        const unsigned grid = (L->num_nodes + block - 1) / block;
        constexpr bool can_keep = S == Explicit::RK4 && sizeof(T) == 8;
        if (can_keep && L->keep_stages)
            adjoint_kernel<M, T, S, R, can_keep><<<grid, block, shm, (cudaStream_t)L->stream>>>(a);
        else
            adjoint_kernel<M, T, S, R><<<grid, block, shm, (cudaStream_t)L->stream>>>(a);
    }
    return cudaPeekAtLastError() == cudaSuccess ? 0 : GOSS_ERR_CUDA;
}

template <class M>
inline int launch_adjoint(const goss_adjoint_launch* L)
{
    const bool f32 = L->precision == GOSS_FP32;
    const bool rev64 = L->reverse_precision == GOSS_FP64;
    if (!(L->reverse_precision == L->precision || (f32 && rev64 && L->solver == GOSS_GRL1)))
        return GOSS_ERR_UNSUPPORTED;
    switch (L->solver) {
    case GOSS_GRL1:
        if (f32 && rev64)
            return launch_adjoint_t<M, float, Explicit::GRL1, double>(L);
        return f32 ? launch_adjoint_t<M, float, Explicit::GRL1>(L) : launch_adjoint_t<M, double, Explicit::GRL1>(L);
    case GOSS_RK4:
        return f32 ? launch_adjoint_t<M, float, Explicit::RK4>(L) : launch_adjoint_t<M, double, Explicit::RK4>(L);
    default:
        return GOSS_ERR_UNSUPPORTED;
    }
}

}  // namespace goss_b200
#endif
