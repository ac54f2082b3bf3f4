// Species weights of the amplitudes (mp_sqom56.f90:901-936, :1338-1377), shared by the kernels that
// write cs(t, Q).
#pragma once

#include "mpsq_internal.h"

namespace mpsq {

// Parameters of the fused deconvolution / weighting.
struct WeightArgs {
  int ngroups;
  int pair[MPSQ_MAX_SPECIES];      // per group: 1 if it holds two species
  int sp_a[MPSQ_MAX_SPECIES];      // species in the real component (or the only one)
  int sp_b[MPSQ_MAX_SPECIES];      // species in the imaginary component
  int weight_mode;
  double b_coh[MPSQ_MAX_SPECIES];  // evaluated in the job's precision
  double xff[MPSQ_MAX_SPECIES][9];
  double kappa;                     // |Q|^2 -> exponent scale of the form factor
  double q0[3];
  double qs[3][3];
  double extra_sq;
  double wnorm;
  int store_species;
  int n_species;
  // FP32 copies (the FP32 path must not convert from double per element: FP64 pipe)
  float b_coh_f[MPSQ_MAX_SPECIES];
  float xff_f[MPSQ_MAX_SPECIES][9];
  float kappa_f, q0_f[3], qs_f[3][3], extra_f, wnorm_f;
  int even;   // |Q|^2 of -k equals that of k (mode (0,0,0) at Q = 0)
  float xb2_f[MPSQ_MAX_SPECIES][4];  // Cromer-Mann b_i log2(e): exp(-b_i s2) = 2^(-b_i log2(e) s2)
};

template <typename T>
struct WP;  // typed views of WeightArgs
template <>
struct WP<float> {
  static __device__ __forceinline__ float b(const WeightArgs& w, int s) { return w.b_coh_f[s]; }
  static __device__ __forceinline__ float x(const WeightArgs& w, int s, int i) { return w.xff_f[s][i]; }
  static __device__ __forceinline__ float kappa(const WeightArgs& w) { return w.kappa_f; }
  static __device__ __forceinline__ float q0(const WeightArgs& w, int b) { return w.q0_f[b]; }
  static __device__ __forceinline__ float qs(const WeightArgs& w, int k, int b) { return w.qs_f[k][b]; }
  static __device__ __forceinline__ float extra(const WeightArgs& w) { return w.extra_f; }
  static __device__ __forceinline__ float wnorm(const WeightArgs& w) { return w.wnorm_f; }
};
template <>
struct WP<double> {
  static __device__ __forceinline__ double b(const WeightArgs& w, int s) { return w.b_coh[s]; }
  static __device__ __forceinline__ double x(const WeightArgs& w, int s, int i) { return w.xff[s][i]; }
  static __device__ __forceinline__ double kappa(const WeightArgs& w) { return w.kappa; }
  static __device__ __forceinline__ double q0(const WeightArgs& w, int b) { return w.q0[b]; }
  static __device__ __forceinline__ double qs(const WeightArgs& w, int k, int b) { return w.qs[k][b]; }
  static __device__ __forceinline__ double extra(const WeightArgs& w) { return w.extra_sq; }
  static __device__ __forceinline__ double wnorm(const WeightArgs& w) { return w.wnorm; }
};

// 2^x on the special-function unit (PTX ex2.approx, relative error of order 2^-22; results
// below the normal range flush to zero).
__device__ __forceinline__ float ex2_sfu(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Species weight at s2 = kappa (|Q|^2 + extra) (mp_sqom56.f90:919-931): b_coh (neutron) or
// the Cromer-Mann factor c + sum_i a_i exp(-b_i s2) (X-ray).  The FP32 path takes each
// exponential as 2^(-(b_i log2 e) s2) on the SFU: one multiply and one SFU operation per term,
// with an error below the FP32 rounding of s2 that feeds it.
template <typename T>
__device__ __forceinline__ T species_weight(const WeightArgs& w, int s, T s2) {
  if (w.weight_mode == MPSQ_WEIGHT_NEUTRON) return WP<T>::b(w, s);
  if (w.weight_mode == MPSQ_WEIGHT_XRAY) {
    if constexpr (sizeof(T) == 4) {
      float f = w.xff_f[s][8];
#pragma unroll
      for (int i = 0; i < 4; ++i) f = fmaf(w.xff_f[s][2 * i], ex2_sfu(-w.xb2_f[s][i] * s2), f);
      return f;
    }
    T f = WP<T>::x(w, s, 8);
    for (int i = 0; i < 4; ++i) f += WP<T>::x(w, s, 2 * i) * exp(-WP<T>::x(w, s, 2 * i + 1) * s2);
    return f;
  }
  return (T)1;
}

}  // namespace mpsq
