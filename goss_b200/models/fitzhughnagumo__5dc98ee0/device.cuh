// Generated by goss_b200.codegen from the 'fitzhughnagumo' model; do not edit.
// Device-side model: rhs and linearised rhs templated on the arithmetic type T.
#ifndef M_FITZHUGHNAGUMO__5DC98EE0_DEVICE_CUH
#define M_FITZHUGHNAGUMO__5DC98EE0_DEVICE_CUH
#include "goss_device_math.cuh"

namespace goss_b200 { namespace models {

struct M_fitzhughnagumo__5dc98ee0 {
  static constexpr const char* name = "fitzhughnagumo";
  static constexpr int num_states = 2;
  static constexpr int num_params = 11;
  static constexpr int num_field_params = 2;
  static constexpr int num_monitored = 0;
  static constexpr int num_derived = 8;
  // the reference generator's linear-term flags (RL1/RL2 use the exponential update for these)
  __host__ __device__ static constexpr bool linear_term(int i) { return i == 1; }

  // values = f(y, time)
  template <typename T>
  __device__ static __forceinline__ void rhs(const T* __restrict__ y, const double time, const T* __restrict__ P, const double* __restrict__ PD, const T* __restrict__ F, T* __restrict__ values)
  {
    const T s_V = y[0];
    const T s_s = y[1];
    const T v_V_th = (P[1] + (P[11]*F[0]));
    const T v_I = ((P[13]*s_s*(s_V + P[12])) + (P[14]*(s_V + P[12])*(s_V - ((v_V_th)))*(P[0] - ((s_V)))));
    const double v_i_Stim = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*time)))))))/(1.0 + exp((PD[15] + (5.0*time)))));
    values[0] = (v_I + T(v_i_Stim));
    values[1] = (F[1]*(s_V + P[12] + (P[17]*s_s)));
    (void)time; (void)P; (void)PD; (void)F;
  }

  // Newton matrix: 4 packed entries (the Jacobian's 4 structural
  // non-zeros, the diagonal and the LU fill-in; row-major over the structure)
  static constexpr int lu_nnz = 4;
  static constexpr bool has_jacobian = false;
  // J := scale*J + I
  template <class A>
  __device__ static __forceinline__ void lu_shift(A J, const double scale)
  {
    for (int k = 0; k < 4; ++k) J[k] = J[k] * scale;
    J[0] = J[0] + 1.0 * 1.0;
    J[3] = J[3] + 1.0 * 1.0;
  }
  // D := scale*S + I
  template <class A, class B>
  __device__ static __forceinline__ void lu_copy_shift(A S, B D, const double scale)
  {
    for (int k = 0; k < 4; ++k) D[k] = S[k] * scale;
    D[0] = D[0] + 1.0 * 1.0;
    D[3] = D[3] + 1.0 * 1.0;
  }
  // in-place Doolittle LU without pivoting over the structure
  template <class A>
  __device__ static __forceinline__ void lu_factorize(A J)
  {
    { const double s = 0.0; J[2] = (J[2] - s) / J[0]; }
    { double s = 0.0; s = s + J[2] * J[1]; J[3] -= s; }
  }
  // x = (LU)^-1 b, forward then backward substitution; b and x may alias
  template <class A>
  __device__ static __forceinline__ void lu_solve(A J, const double* b, double* x)
  {
    x[0] = b[0];
    { double s = 0.0; s = s + J[2] * x[0]; x[1] = b[1] - s; }
    x[1] = x[1] / J[3];
    { double s = 0.0; s = s + J[1] * x[1]; x[0] = (x[0] - s) / J[0]; }
  }
  // forward differences: zero the entries outside the Jacobian's structure
  template <class A>
  __device__ static __forceinline__ void fd_clear(A J)
  {
    (void)J;
  }
  // dense row-major copy: out(r*n + c, value) for every entry
  template <typename T, class Out>
  __device__ static __forceinline__ void lu_unpack(const T* J, Out&& out)
  {
    out(0, J[0]);
    out(1, J[1]);
    out(2, J[2]);
    out(3, J[3]);
  }

  // derived constants: parameter-only sub-expressions, evaluated once per
  // launch on the host in FP64 and stored after the parameters
  static void derived(const double* P, double* C)
  {
    const double v_V_amp = (P[0] - ((P[1])));
    C[0] = v_V_amp;
    C[1] = (-(P[1]));
    C[2] = (-(P[5]/v_V_amp));
    C[3] = (P[4]/(v_V_amp*v_V_amp));
    C[4] = ((-(5.0*P[8])) - ((5.0*P[10])));
    C[5] = (-(5.0*P[10]));
    C[6] = (-(P[6]));
    C[7] = (-(P[4]/(v_V_amp*v_V_amp)));
    (void)P; (void)C;
  }

  // rhs = f(y, time), linear[i] = d f_i / d y_i
  template <typename T>
  __device__ static __forceinline__ void linearized(const T* __restrict__ y, const double time, const T* __restrict__ P, const double* __restrict__ PD, const T* __restrict__ F, T* __restrict__ linear, T* __restrict__ rhs)
  {
    const T s_V = y[0];
    const T s_s = y[1];
    const T v_V_th = (P[1] + (P[11]*F[0]));
    const T v_I = ((P[13]*s_s*(s_V + P[12])) + (P[14]*(s_V + P[12])*(s_V - ((v_V_th)))*(P[0] - ((s_V)))));
    const double v_i_Stim = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*time)))))))/(1.0 + exp((PD[15] + (5.0*time)))));
    rhs[0] = (v_I + T(v_i_Stim));
    rhs[1] = (F[1]*(s_V + P[12] + (P[17]*s_s)));
    linear[1] = (P[17]*F[1]);
    const T v_dI_dV = ((P[13]*s_s) + (P[14]*(s_V + P[12])*(P[0] - ((s_V)))) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V)))) + (P[18]*(s_V + P[12])*(s_V - ((v_V_th)))));
    linear[0] = v_dI_dV;
    (void)time; (void)P; (void)PD; (void)F;
  }

  // linearized with every distinct transcendental and reciprocal of a state-dependent
  // operand evaluated once
  template <typename T>
  __device__ static __forceinline__ void linearized_split(const T* __restrict__ y, const double time, const T* __restrict__ P, const double* __restrict__ PD, const T* __restrict__ F, T* __restrict__ linear, T* __restrict__ rhs)
  {
    const T s_V = y[0];
    const T s_s = y[1];
    const T v_V_th = (P[1] + (P[11]*F[0]));
    const T v_I = ((s_V + P[12])*((P[13]*s_s) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
    const double v_i_Stim = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*time)))))))/(1.0 + exp((PD[15] + (5.0*time)))));
    const T v_dI_dV = ((P[14]*((P[0] - ((s_V)))*(P[12] - ((v_V_th)) + (T(2.0)*s_V)))) + ((P[13]*s_s) + (P[18]*(s_V + P[12])*(s_V - ((v_V_th))))));
    rhs[0] = (v_I + T(v_i_Stim));
    rhs[1] = (F[1]*(s_V + P[12] + (P[17]*s_s)));
    linear[1] = (P[17]*F[1]);
    linear[0] = v_dI_dV;
    (void)time; (void)P; (void)PD; (void)F;
  }

  // rhs in the same split form
  template <typename T>
  __device__ static __forceinline__ void rhs_split(const T* __restrict__ y, const double time, const T* __restrict__ P, const double* __restrict__ PD, const T* __restrict__ F, T* __restrict__ values)
  {
    const T s_V = y[0];
    const T s_s = y[1];
    const T v_V_th = (P[1] + (P[11]*F[0]));
    const T v_I = ((s_V + P[12])*((P[13]*s_s) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
    const double v_i_Stim = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*time)))))))/(1.0 + exp((PD[15] + (5.0*time)))));
    values[0] = (v_I + T(v_i_Stim));
    values[1] = (F[1]*(s_V + P[12] + (P[17]*s_s)));
    (void)time; (void)P; (void)PD; (void)F;
  }

  // forward-difference Jacobian of rhs_split at y into the packed Newton matrix (structural
  // entries; fd_clear sets the others); column i recomputes only the statements of its rows
  // that depend on state i.  f1 = f(y, time) (rhs_split) from the unperturbed statements
  template <typename T, class A>
  __device__ static __forceinline__ void rhs_fd_jacobian(const T* __restrict__ y, const double time, const T* __restrict__ P, const double* __restrict__ PD, const T* __restrict__ F, T* __restrict__ f1, A J)
  {
    const T s_V = y[0];
    const T s_s = y[1];
    const T v_V_th = (P[1] + (P[11]*F[0]));
    const T v_I = ((s_V + P[12])*((P[13]*s_s) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
    const double v_i_Stim = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*time)))))))/(1.0 + exp((PD[15] + (5.0*time)))));
    f1[0] = (v_I + T(v_i_Stim));
    f1[1] = (F[1]*(s_V + P[12] + (P[17]*s_s)));
    {
      const double d = sqrt(1e-15 * (1e-5 > fabs(double(y[0])) ? 1e-5 : fabs(double(y[0]))));
      const T v___yp0 = T(double(y[0]) + d);
      const T v_I__k0 = ((v___yp0 + P[12])*((P[13]*s_s) + (P[14]*(v___yp0 - ((v_V_th)))*(P[0] - ((v___yp0))))));
      J[0] = (((v_I__k0 + T(v_i_Stim))) - f1[0]) / d;
      J[2] = (((F[1]*(v___yp0 + P[12] + (P[17]*s_s)))) - f1[1]) / d;
    }
    {
      const double d = sqrt(1e-15 * (1e-5 > fabs(double(y[1])) ? 1e-5 : fabs(double(y[1]))));
      const T v___yp1 = T(double(y[1]) + d);
      const T v_I__k1 = ((s_V + P[12])*((v___yp1*P[13]) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
      J[1] = (((v_I__k1 + T(v_i_Stim))) - f1[0]) / d;
      J[3] = (((F[1]*(s_V + P[12] + (v___yp1*P[17])))) - f1[1]) / d;
    }
    (void)time; (void)P; (void)PD; (void)F; (void)f1; (void)J;
  }

  // f1 = f(y, time), and the forward-difference Jacobian only if want_jac (J is left as it
  // is otherwise): rhs_fd_jacobian with its columns selected at run time
  template <typename T, class A>
  __device__ static __forceinline__ void rhs_fd_jacobian_sel(const T* __restrict__ y, const double time, const T* __restrict__ P, const double* __restrict__ PD, const T* __restrict__ F, const bool want_jac,
      T* __restrict__ f1, A J)
  {
    const T s_V = y[0];
    const T s_s = y[1];
    const T v_V_th = (P[1] + (P[11]*F[0]));
    const T v_I = ((s_V + P[12])*((P[13]*s_s) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
    const double v_i_Stim = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*time)))))))/(1.0 + exp((PD[15] + (5.0*time)))));
    f1[0] = (v_I + T(v_i_Stim));
    f1[1] = (F[1]*(s_V + P[12] + (P[17]*s_s)));
    if (want_jac) {
    fd_clear(J);
    {
      const double d = sqrt(1e-15 * (1e-5 > fabs(double(y[0])) ? 1e-5 : fabs(double(y[0]))));
      const T v___yp0 = T(double(y[0]) + d);
      const T v_I__k0 = ((v___yp0 + P[12])*((P[13]*s_s) + (P[14]*(v___yp0 - ((v_V_th)))*(P[0] - ((v___yp0))))));
      J[0] = (((v_I__k0 + T(v_i_Stim))) - f1[0]) / d;
      J[2] = (((F[1]*(v___yp0 + P[12] + (P[17]*s_s)))) - f1[1]) / d;
    }
    {
      const double d = sqrt(1e-15 * (1e-5 > fabs(double(y[1])) ? 1e-5 : fabs(double(y[1]))));
      const T v___yp1 = T(double(y[1]) + d);
      const T v_I__k1 = ((s_V + P[12])*((v___yp1*P[13]) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
      J[1] = (((v_I__k1 + T(v_i_Stim))) - f1[0]) / d;
      J[3] = (((F[1]*(s_V + P[12] + (v___yp1*P[17])))) - f1[1]) / d;
    }
    }
    (void)time; (void)P; (void)PD; (void)F; (void)f1; (void)J;
  }

  // the same, also writing f0 = f(y, t0) (only the time-dependent statements again)
  template <typename T, class A>
  __device__ static __forceinline__ void rhs2_fd_jacobian(const T* __restrict__ y, const double time, const T* __restrict__ P, const double* __restrict__ PD, const T* __restrict__ F, const double t0,
      T* __restrict__ f0, T* __restrict__ f1, A J)
  {
    const T s_V = y[0];
    const T s_s = y[1];
    const T v_V_th = (P[1] + (P[11]*F[0]));
    const T v_I = ((s_V + P[12])*((P[13]*s_s) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
    const double v_i_Stim = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*time)))))))/(1.0 + exp((PD[15] + (5.0*time)))));
    f1[0] = (v_I + T(v_i_Stim));
    f1[1] = (F[1]*(s_V + P[12] + (P[17]*s_s)));
    const double v___tzero = t0;
    const double v_i_Stim__tz = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*v___tzero)))))))/(1.0 + exp((PD[15] + (5.0*v___tzero)))));
    f0[0] = (v_i_Stim__tz + v_I);
    f0[1] = f1[1];
    {
      const double d = sqrt(1e-15 * (1e-5 > fabs(double(y[0])) ? 1e-5 : fabs(double(y[0]))));
      const T v___yp0 = T(double(y[0]) + d);
      const T v_I__k0 = ((v___yp0 + P[12])*((P[13]*s_s) + (P[14]*(v___yp0 - ((v_V_th)))*(P[0] - ((v___yp0))))));
      J[0] = (((v_I__k0 + T(v_i_Stim))) - f1[0]) / d;
      J[2] = (((F[1]*(v___yp0 + P[12] + (P[17]*s_s)))) - f1[1]) / d;
    }
    {
      const double d = sqrt(1e-15 * (1e-5 > fabs(double(y[1])) ? 1e-5 : fabs(double(y[1]))));
      const T v___yp1 = T(double(y[1]) + d);
      const T v_I__k1 = ((s_V + P[12])*((v___yp1*P[13]) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
      J[1] = (((v_I__k1 + T(v_i_Stim))) - f1[0]) / d;
      J[3] = (((F[1]*(s_V + P[12] + (v___yp1*P[17])))) - f1[1]) / d;
    }
    (void)time; (void)t0; (void)P; (void)PD; (void)F; (void)f0; (void)f1; (void)J;
  }

  // vector-Jacobian product of linearized (reverse mode, generated): after the forward
  // sweep seed(linear, rhs, abar, bbar) supplies the cotangents of the outputs, then
  // ybar = abar^T d(linear)/dy + bbar^T d(rhs)/dy and Fbar likewise for the field parameters
  template <typename T, class Seed>
  __device__ static __forceinline__ void linearized_vjp(const T* __restrict__ y, const double time, const T* __restrict__ P, const double* __restrict__ PD, const T* __restrict__ F, Seed&& seed,
      T* __restrict__ ybar, T* __restrict__ Fbar)
  {
    const T s_V = y[0];
    const T s_s = y[1];
    const T v_V_th = (P[1] + (P[11]*F[0]));
    const T v_I = ((s_V + P[12])*((P[13]*s_s) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
    const double v_i_Stim = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*time)))))))/(1.0 + exp((PD[15] + (5.0*time)))));
    const T v_dI_dV = ((P[14]*((P[0] - ((s_V)))*(P[12] - ((v_V_th)) + (T(2.0)*s_V)))) + ((P[13]*s_s) + (P[18]*(s_V + P[12])*(s_V - ((v_V_th))))));
    T lin_v[2], abar[2], rhs_v[2], bbar[2];
    rhs_v[0] = (v_I + T(v_i_Stim));
    rhs_v[1] = (F[1]*(s_V + P[12] + (P[17]*s_s)));
    lin_v[1] = (P[17]*F[1]);
    lin_v[0] = v_dI_dV;
    seed(lin_v, rhs_v, abar, bbar);
    const T a_dI_dV = abar[0];
    const T a_I = bbar[0];
    const T a_V_th = ((a_dI_dV*((-(P[14]*(P[0] - ((s_V))))) - ((P[18]*(s_V + P[12]))))) - ((a_I*P[14]*(s_V + P[12])*(P[0] - ((s_V))))));
    ybar[0] = ((a_I*((P[14]*(((s_V - ((v_V_th)))*(P[0] - ((P[12])) - ((T(2.0)*s_V)))) + ((s_V + P[12])*(P[0] - ((s_V)))))) + (P[13]*s_s))) + (a_dI_dV*((P[14]*(v_V_th - ((P[12])) - ((T(2.0)*s_V)) + (T(2.0)*(P[0] - ((s_V)))))) + (P[18]*(P[12] - ((v_V_th)) + (T(2.0)*s_V))))) + (bbar[1]*F[1]));
    ybar[1] = ((P[13]*(a_dI_dV + (a_I*(s_V + P[12])))) + (P[17]*bbar[1]*F[1]));
    Fbar[0] = (a_V_th*P[11]);
    Fbar[1] = ((P[17]*abar[1]) + (bbar[1]*(s_V + P[12] + (P[17]*s_s))));
    (void)time; (void)P; (void)PD; (void)F; (void)abar; (void)bbar; (void)Fbar;
  }

  // vector-Jacobian product of rhs (reverse mode, generated): after the forward sweep
  // seed(values, bbar) supplies the cotangents of the values, then ybar = bbar^T df/dy
  // and Fbar = bbar^T df/dF
  template <typename T, class Seed>
  __device__ static __forceinline__ void rhs_vjp(const T* __restrict__ y, const double time, const T* __restrict__ P, const double* __restrict__ PD, const T* __restrict__ F, Seed&& seed,
      T* __restrict__ ybar, T* __restrict__ Fbar)
  {
    const T s_V = y[0];
    const T s_s = y[1];
    const T v_V_th = (P[1] + (P[11]*F[0]));
    const T v_I = ((s_V + P[12])*((P[13]*s_s) + (P[14]*(s_V - ((v_V_th)))*(P[0] - ((s_V))))));
    const double v_i_Stim = (PD[7]*(1.0 - ((1.0/(1.0 + exp((PD[16] + (5.0*time)))))))/(1.0 + exp((PD[15] + (5.0*time)))));
    T f_v[2], bbar[2];
    f_v[0] = (v_I + T(v_i_Stim));
    f_v[1] = (F[1]*(s_V + P[12] + (P[17]*s_s)));
    seed(f_v, bbar);
    const T a_I = bbar[0];
    const T a_V_th = (-(a_I*P[14]*(s_V + P[12])*(P[0] - ((s_V)))));
    ybar[0] = ((a_I*((P[14]*(((s_V - ((v_V_th)))*(P[0] - ((P[12])) - ((T(2.0)*s_V)))) + ((s_V + P[12])*(P[0] - ((s_V)))))) + (P[13]*s_s))) + (bbar[1]*F[1]));
    ybar[1] = ((a_I*P[13]*(s_V + P[12])) + (P[17]*bbar[1]*F[1]));
    Fbar[0] = (a_V_th*P[11]);
    Fbar[1] = (bbar[1]*(s_V + P[12] + (P[17]*s_s)));
    (void)time; (void)P; (void)PD; (void)F; (void)bbar; (void)Fbar;
  }
};

}}  // namespace goss_b200::models
#endif
