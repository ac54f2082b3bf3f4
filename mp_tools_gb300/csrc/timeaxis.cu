// Time-axis kernels on the amplitude store cs(t, Q) of a job (frame-major, Q fastest):
//  * total S(Q) = sum_t |cs|^2 / nfile                      (mp_sqom56.f90:1381-1387)
//  * E=const map, sliding Hann window, one frequency bin     (:1437-1478, window :941-948)
//  * E(Q) dispersion cut, windowed DFT per start frame       (:1480-1517)
//  * Gaussian-window spectrum over the whole run (one FFT per Q in shared memory)
//  * I(Q,t) maps and path cuts (the j_sq /= 1 branch, :1467-1472, :1504-1510)
//  * atom-pair forms of the E=const map and E(Q) cut (raw sum of two species, :1460-1464)
// The ω-resolved forms subtract the elastic mean <cs>_t first (:1177-1185, :1359-1376) and
// optionally scale by 1/|Q| (:1373).  Sums over frames are compensated (FP32) or FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "dft.cuh"
#include "mpsq_internal.h"

namespace mpsq {

template <typename T> struct Acc;  // compensated accumulator
template <> struct Acc<float> {
  float s = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};
template <> struct Acc<double> {
  double s = 0.0;
  __device__ __forceinline__ void add(double v) { s += v; }
  __device__ __forceinline__ double value() const { return s; }
};

template <typename T>
__global__ void sq_total_kernel(const typename Cplx<T>::type* __restrict__ cs, int64_t nq,
                                int nt, double scale, float* __restrict__ out) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) return;
  Acc<T> a;
  for (int t = 0; t < nt; ++t) {
    const auto v = cs[(int64_t)t * nq + q];
    a.add(v.x * v.x + v.y * v.y);
  }
  out[q] = (float)(a.value() * scale);
}

// The time series a map is formed from: x(t, q) = a[t*stride + q] (+ b[t*stride + q]).  The
// job's weighted amplitudes (a = cs, stride n_Q, centred: the elastic mean is subtracted) or
// the raw sum of two stored species amplitudes (the atom-pair modes, not centred).
template <typename T>
struct Series {
  const typename Cplx<T>::type* a;
  const typename Cplx<T>::type* b;
  int64_t stride;
  int center;
};

// Loads a [nt x QT] tile of the series into shared memory, subtracts the column means (if
// centred) and applies the optional 1/|Q| factor.  Thread layout: column = tid % QT,
// part = tid / QT; a thread's elements are all of one column (QT a power of two, the block a
// multiple of it), so it sums them as it loads them and centres its own without index arithmetic.
// Sums are pairwise, within a thread's loads and over the parts: what the mean loses to rounding stays
// in every frame and adds up coherently in the lowest frequencies, and the 256 parts of a single column
// added one after the other raised the error of an E(Q) cut of 200 frames by a fifth.
template <typename T>
__device__ void load_centered_tile(Series<T> src, int64_t nq, int nt, int64_t q0, int QT,
                                   const float* __restrict__ q2n, typename Cplx<T>::type* xs,
                                   T* red_re, T* red_im) {
  using C = typename Cplx<T>::type;
  const int tid = threadIdx.x, NT = blockDim.x;
  const int col = tid & (QT - 1), nparts = NT / QT;
  const int64_t q = q0 + col;
  const bool in = q < nq;
  constexpr int LD = 8;               // loads in flight per thread
  T sr = 0, si = 0;
  for (int t0 = tid / QT; t0 < nt; t0 += LD * nparts) {
    C v[LD], u[LD];
#pragma unroll
    for (int k = 0; k < LD; ++k) {
      const int t = t0 + k * nparts;
      v[k].x = v[k].y = u[k].x = u[k].y = 0;
      if (t < nt && in) {
        v[k] = src.a[(int64_t)t * src.stride + q];
        if (src.b) u[k] = src.b[(int64_t)t * src.stride + q];
      }
    }
#pragma unroll
    for (int k = 0; k < LD; ++k) {
      const int t = t0 + k * nparts;
      v[k].x += u[k].x;
      v[k].y += u[k].y;
      if (t < nt) xs[t * QT + col] = v[k];
    }
#pragma unroll
    for (int n = LD / 2; n > 0; n /= 2)
#pragma unroll
      for (int k = 0; k < n; ++k) {
        v[k].x += v[k + n].x;
        v[k].y += v[k + n].y;
      }
    sr += v[0].x;
    si += v[0].y;
  }
  const T f = q2n && in ? (T)q2n[q] : (T)1;
  T mr = 0, mi = 0;
  if (src.center) {
    red_re[tid] = sr;
    red_im[tid] = si;
    __syncthreads();
    for (int n = nparts; n > 1;) {
      const int half = (n + 1) / 2;
      if (tid / QT + half < n) {
        red_re[tid] += red_re[tid + half * QT];
        red_im[tid] += red_im[tid + half * QT];
      }
      __syncthreads();
      n = half;
    }
    if (tid < QT) {
      red_re[NT + tid] = red_re[tid] / (T)nt;
      red_im[NT + tid] = red_im[tid] / (T)nt;
    }
    __syncthreads();
    mr = red_re[NT + col];
    mi = red_im[NT + col];
  }
  if (src.center || q2n)
    for (int t = tid / QT; t < nt; t += nparts) {
      C v = xs[t * QT + col];
      v.x = (v.x - mr) * f;
      v.y = (v.y - mi) * f;
      xs[t * QT + col] = v;
    }
  __syncthreads();
}

// Windowed sums of kStarts consecutive start frames t0 .. t0 + kStarts - 1 of one series:
// s[r] = sum_{i < n} w(i) y(r + i), y(i) = x(t0 + i) turned by exp(-2 pi i f (t0 + i) / n).  With the
// phase counted from frame 0 instead of from each window's start the sums keep their modulus and the
// coefficients are real, and the series slides through kStarts registers, so a coefficient and one
// new sample serve 2 kStarts multiply-adds; a sum per start frame with complex coefficients loads two
// values for 4 (420 us per map of 102,400 columns, 200 frames and a window of 101 there,
// shared-memory bound; complex coefficients on the sliding series 287 us; 176 us here).
constexpr int kStarts = 8;

// FP32 takes both parts of a product in one instruction (PTX fma.rn.f32x2, IEEE per lane).
struct SlideAcc32 {
  unsigned long long s = 0;
  __device__ __forceinline__ float2 value() const {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(s));
    return v;
  }
};
struct SlideAcc64 {
  double2 s = {0.0, 0.0};
  __device__ __forceinline__ double2 value() const { return s; }
};
template <typename T> struct SlideAccOf;
template <> struct SlideAccOf<float> { using type = SlideAcc32; };
template <> struct SlideAccOf<double> { using type = SlideAcc64; };
__device__ __forceinline__ void slide_add(SlideAcc32 (&s)[kStarts], float c, const float2 (&w)[kStarts], int u) {
  unsigned long long cc;
  asm("mov.b64 %0, {%1, %1};" : "=l"(cc) : "f"(c));
#pragma unroll
  for (int r = 0; r < kStarts; ++r) {
    const float2 v = w[(r + u) % kStarts];
    unsigned long long b;
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(v.x), "f"(v.y));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(s[r].s) : "l"(cc), "l"(b));
  }
}
__device__ __forceinline__ void slide_add(SlideAcc64 (&s)[kStarts], double c, const double2 (&w)[kStarts], int u) {
#pragma unroll
  for (int r = 0; r < kStarts; ++r) {
    const double2 v = w[(r + u) % kStarts];
    s[r].s.x = fma(c, v.x, s[r].s.x);
    s[r].s.y = fma(c, v.y, s[r].s.y);
  }
}

// y(i) is called for i = 0, 1, 2, ... in order, up to n - 1 + kStarts.
template <typename T, class Series_, class Coef>
__device__ __forceinline__ void sliding_sums(int n, Series_&& y, const Coef& coef,
                                             typename SlideAccOf<T>::type (&s)[kStarts]) {
  typename Cplx<T>::type w[kStarts];
#pragma unroll
  for (int r = 0; r < kStarts; ++r) w[r] = y(r);
  int i0 = 0;
  for (; i0 + kStarts <= n; i0 += kStarts) {
#pragma unroll
    for (int u = 0; u < kStarts; ++u) {
      slide_add(s, coef(i0 + u), w, u);
      w[u] = y(i0 + u + kStarts);
    }
  }
#pragma unroll
  for (int u = 0; u < kStarts - 1; ++u) {
    if (i0 + u < n) {                 // uniform
      slide_add(s, coef(i0 + u), w, u);
      w[u] = y(i0 + u + kStarts);
    }
  }
}

// E=const map: S(Q) = sum_{t0} | sum_i ph_i x(t0+i) |^2 with ph_i = t_wind_i exp(-2 pi i
// (j_freq-1)(i - n_int/2)/n_int) (0-based i), times scale.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) econst_kernel(Series<T> cs, int64_t nq, int nt,
                              int QT, int n_int, const float* __restrict__ t_wind, int jf,
                              const float* __restrict__ q2n, double scale, int win_smem,
                              float* __restrict__ out) {
  using C = typename Cplx<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NT = blockDim.x;
  C* xs = reinterpret_cast<C*>(smem_raw);
  C* ph = xs + (size_t)(nt + kStarts) * QT;                // exp(-2 pi i jf t / n_int), t < n_int
  T* red_re = reinterpret_cast<T*>(ph + n_int);
  T* red_im = red_re + NT + QT;
  T* win = red_im + NT + QT;                               // [n_int], where it fits
  const int64_t q0 = (int64_t)blockIdx.x * QT;
  const int tid = threadIdx.x;
  for (int e = tid; e < kStarts * QT; e += NT) xs[nt * QT + e].x = xs[nt * QT + e].y = 0;
  for (int i = tid; i < n_int; i += NT) {
    const int r = (int)(((long long)jf * i) % n_int);
    C v;
    if (sizeof(T) == 8) {
      double s_, c_;
      sincospi(-2.0 * (double)r / n_int, &s_, &c_);
      v.x = (T)c_;
      v.y = (T)s_;
    } else {
      float s_, c_;
      sincospif(-2.0f * (float)r / (float)n_int, &s_, &c_);
      v.x = (T)c_;
      v.y = (T)s_;
    }
    ph[i] = v;
    if (win_smem) win[i] = (T)t_wind[i];
  }
  load_centered_tile<T>(cs, nq, nt, q0, QT, q2n, xs, red_re, red_im);
  {  // turn every sample by its frame's phase
    const int step = NT / QT;
    int r = (tid / QT) % n_int;
    for (int t = tid / QT; t < nt; t += step) {
      C* const e = xs + t * QT + (tid & (QT - 1));
      const C v = *e, a = ph[r];
      e->x = a.x * v.x - a.y * v.y;
      e->y = a.x * v.y + a.y * v.x;
      r = (r + step) % n_int;
    }
  }
  __syncthreads();
  const int col = tid % QT, part = tid / QT, nparts = NT / QT;
  const int n0 = nt - n_int + 1;
  Acc<T> acc;
  if (part < nparts)
    for (int t0 = part * kStarts; t0 < n0; t0 += nparts * kStarts) {
      typename SlideAccOf<T>::type s[kStarts];
      const C* x = xs + t0 * QT + col;
      sliding_sums<T>(n_int, [&](int i) { return x[i * QT]; },
                      [&](int i) { return win_smem ? win[i] : (T)t_wind[i]; }, s);
#pragma unroll
      for (int r = 0; r < kStarts; ++r)
        if (t0 + r < n0) {
          const C v = s[r].value();
          acc.add(v.x * v.x + v.y * v.y);
        }
    }
  __syncthreads();
  red_re[tid] = (T)acc.value();
  __syncthreads();
  if (tid < QT) {
    double s = 0.0;
    for (int p = 0; p < nparts; ++p) s += (double)red_re[p * QT + tid];
    const int64_t q = q0 + tid;
    if (q < nq) out[q] = (float)(s * scale);
  }
}

constexpr int kSlots = 1024;          // partial sums of the E(Q) cut held at a time
// Dispersion: for path point p (one CTA), acc[f] = sum_{t0} |sum_i w_i x(t0+i) e^{-2 pi i f i/n}|^2.
// Thread (f, block of kStarts start frames), frequencies fastest; each block's sum goes to a slot of its
// own and the slots of a frequency are added in FP64 in the order of the start frames, so that a cut is
// the same in every run (a thread per frequency alone keeps 51 of 128 threads busy at 200 frames: 289 us
// for 320 points, 39 us here).
template <typename T>
__global__ void dispersion_kernel(Series<T> cs, int64_t nq,
                                  int nt, const int64_t* __restrict__ qidx, int n_int,
                                  const float* __restrict__ t_wind, int n_freq,
                                  const float* __restrict__ q2n, double scale, int sum_off,
                                  int win_smem, float* __restrict__ out) {
  using C = typename Cplx<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NT = blockDim.x, tid = threadIdx.x;
  C* xs = reinterpret_cast<C*>(smem_raw);
  C* tw = xs + nt + kStarts;
  T* red_re = reinterpret_cast<T*>(tw + n_int);
  T* red_im = red_re + NT + 1;
  T* win = red_im + NT + 1;                                      // [n_int], where it fits
  double* sum = reinterpret_cast<double*>(smem_raw + sum_off);   // [min(n_freq blocks, kSlots)]
  const int64_t q = qidx[blockIdx.x];
  if (q < 0 || q >= nq) {
    for (int f = tid; f < n_freq; f += NT) out[(int64_t)blockIdx.x * n_freq + f] = 0.0f;
    return;
  }
  if (tid < kStarts) xs[nt + tid].x = xs[nt + tid].y = 0;
  for (int i = tid; i < n_int; i += NT) {
    T sn, cn;
    if (sizeof(T) == 8) {
      double s_, c_;
      sincospi(-2.0 * (double)i / n_int, &s_, &c_);
      sn = (T)s_;
      cn = (T)c_;
    } else {
      float s_, c_;
      sincospif(-2.0f * (float)i / (float)n_int, &s_, &c_);
      sn = (T)s_;
      cn = (T)c_;
    }
    C v;
    v.x = cn;
    v.y = sn;
    tw[i] = v;
    if (win_smem) win[i] = (T)t_wind[i];
  }
  // the column of this path point (QT = 1 tile)
  load_centered_tile<T>(cs, nq, nt, q, 1, q2n, xs, red_re, red_im);
  const int n0 = nt - n_int + 1, blocks = (n0 + kStarts - 1) / kStarts;
  // frequencies at a time: those whose blocks fit the slots; a single one with more blocks than that
  // adds block b to slot b mod kSlots (always by the same thread, as NT divides kSlots)
  const int at_once = max(1, kSlots / blocks);
  for (int f0 = 0; f0 < n_freq; f0 += at_once) {
    const int nf = min(at_once, n_freq - f0);
    for (int e = tid; e < nf * blocks; e += NT) {
      const int b = e / nf, f = e - b * nf, t0 = b * kStarts;
      int r = (int)(((long long)(f0 + f) * t0) % n_int);   // f (t0 + i) mod n_int
      typename SlideAccOf<T>::type s[kStarts];
      sliding_sums<T>(n_int, [&](int i) {
        const C a = tw[r], v = xs[t0 + i];
        C y;
        y.x = a.x * v.x - a.y * v.y;
        y.y = a.x * v.y + a.y * v.x;
        r += f0 + f;
        if (r >= n_int) r -= n_int;
        return y;
      }, [&](int i) { return win_smem ? win[i] : (T)t_wind[i]; }, s);
      Acc<T> acc;
#pragma unroll
      for (int k = 0; k < kStarts; ++k)
        if (t0 + k < n0) {
          const C v = s[k].value();
          acc.add(v.x * v.x + v.y * v.y);
        }
      sum[e % kSlots] = e < kSlots ? acc.value() : sum[e % kSlots] + acc.value();
    }
    __syncthreads();
    const int slots = min(nf * blocks, kSlots);
    for (int f = tid; f < nf; f += NT) {
      double s = 0.0;
      for (int e = f; e < slots; e += nf) s += sum[e];
      out[(int64_t)blockIdx.x * n_freq + f0 + f] = (float)(s * scale);
    }
    __syncthreads();
  }
}

// Gaussian-window spectrum: per Q column, X_k = sum_t g_t (x_t - <x>) e^{-2 pi i k t/nt},
// out[k][q] = |X_k|^2 * scale for k < n_freq.  nt = 2^p <= 1024, radix-2 in shared memory.
template <typename T>
__global__ void gauss_fft_kernel(Series<T> cs, int64_t nq,
                                 int nt, int logn, int QT, const float* __restrict__ gwin,
                                 int n_freq, const float* __restrict__ q2n, double scale,
                                 float* __restrict__ out) {
  using C = typename Cplx<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NT = blockDim.x, tid = threadIdx.x;
  C* xs = reinterpret_cast<C*>(smem_raw);
  C* tw = xs + (size_t)nt * QT;
  T* red_re = reinterpret_cast<T*>(tw + nt / 2);
  T* red_im = red_re + NT + QT;
  const int64_t q0 = (int64_t)blockIdx.x * QT;
  for (int i = tid; i < nt / 2; i += NT) {
    T sn, cn;
    if (sizeof(T) == 8) {
      double s_, c_;
      sincospi(-2.0 * (double)i / nt, &s_, &c_);
      sn = (T)s_;
      cn = (T)c_;
    } else {
      float s_, c_;
      sincospif(-2.0f * (float)i / (float)nt, &s_, &c_);
      sn = (T)s_;
      cn = (T)c_;
    }
    C v;
    v.x = cn;
    v.y = sn;
    tw[i] = v;
  }
  load_centered_tile<T>(cs, nq, nt, q0, QT, q2n, xs, red_re, red_im);
  // window
  for (int e = tid; e < nt * QT; e += NT) {
    const T g = (T)gwin[e / QT];
    C v = xs[e];
    v.x *= g;
    v.y *= g;
    xs[e] = v;
  }
  __syncthreads();
  // bit reversal
  for (int e = tid; e < nt * QT; e += NT) {
    const int t = e / QT, c = e % QT;
    const int r = (int)(__brev((unsigned)t) >> (32 - logn));
    if (r > t) {
      const C a = xs[t * QT + c];
      xs[t * QT + c] = xs[r * QT + c];
      xs[r * QT + c] = a;
    }
  }
  __syncthreads();
  const int nb = (nt / 2) * QT;
  for (int s = 0; s < logn; ++s) {
    const int half = 1 << s;
    const int stride = nt >> (s + 1);  // twiddle index step
    for (int e = tid; e < nb; e += NT) {
      const int c = e % QT, b = e / QT;
      const int grp = b >> s, pos = b & (half - 1);
      const int i = (grp << (s + 1)) + pos, jj = i + half;
      const C wv = tw[pos * stride];
      const C u = xs[i * QT + c], v0 = xs[jj * QT + c];
      C v;
      v.x = v0.x * wv.x - v0.y * wv.y;
      v.y = v0.x * wv.y + v0.y * wv.x;
      C a, b2;
      a.x = u.x + v.x;
      a.y = u.y + v.y;
      b2.x = u.x - v.x;
      b2.y = u.y - v.y;
      xs[i * QT + c] = a;
      xs[jj * QT + c] = b2;
    }
    __syncthreads();
  }
  for (int e = tid; e < n_freq * QT; e += NT) {
    const int k = e / QT, c = e % QT;
    const int64_t q = q0 + c;
    if (q >= nq) continue;
    const C v = xs[k * QT + c];
    out[(int64_t)k * nq + q] = (float)((double)(v.x * v.x + v.y * v.y) * scale);
  }
}

// I(Q,t) map at lag `lag`: out[q] = Re sum_{i<n_int} x(i+lag) conj(x(i)) / n_int * scale.
template <typename T>
__global__ void iqt_kernel(Series<T> cs, int64_t nq, int nt, int QT, int n_int, int lag,
                           const float* __restrict__ q2n, double scale, float* __restrict__ out) {
  using C = typename Cplx<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NT = blockDim.x, tid = threadIdx.x;
  C* xs = reinterpret_cast<C*>(smem_raw);
  T* red_re = reinterpret_cast<T*>(xs + (size_t)nt * QT);
  T* red_im = red_re + NT + QT;
  const int64_t q0 = (int64_t)blockIdx.x * QT;
  load_centered_tile<T>(cs, nq, nt, q0, QT, q2n, xs, red_re, red_im);
  const int col = tid % QT, part = tid / QT, nparts = NT / QT;
  Acc<T> acc;
  if (part < nparts)
    for (int i = part; i < n_int; i += nparts) {
      const C a = xs[(i + lag) * QT + col], b = xs[i * QT + col];
      acc.add(a.x * b.x + a.y * b.y);   // Re(a conj b)
    }
  __syncthreads();
  red_re[tid] = (T)acc.value();
  __syncthreads();
  if (tid < QT) {
    double s = 0.0;
    for (int p = 0; p < nparts; ++p) s += (double)red_re[p * QT + tid];
    const int64_t q = q0 + tid;
    if (q < nq) out[q] = (float)(s / n_int * scale);
  }
}

// I(Q,t) along a path: one CTA per path point, out[p * n_lag + t] = Re sum_{i<n_int}
// x(t+i) conj(x(i)) * scale for t < n_lag = nt - n_int + 1.
template <typename T>
__global__ void iqt_dispersion_kernel(Series<T> cs, int64_t nq, int nt,
                                      const int64_t* __restrict__ qidx, int n_int,
                                      const float* __restrict__ q2n, double scale,
                                      float* __restrict__ out) {
  using C = typename Cplx<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NT = blockDim.x, tid = threadIdx.x;
  C* xs = reinterpret_cast<C*>(smem_raw);
  T* red_re = reinterpret_cast<T*>(xs + nt);
  T* red_im = red_re + NT + 1;
  const int n_lag = nt - n_int + 1;
  const int64_t q = qidx[blockIdx.x];
  if (q < 0 || q >= nq) {
    for (int t = tid; t < n_lag; t += NT) out[(int64_t)blockIdx.x * n_lag + t] = 0.0f;
    return;
  }
  load_centered_tile<T>(cs, nq, nt, q, 1, q2n, xs, red_re, red_im);
  for (int t = tid; t < n_lag; t += NT) {
    Acc<T> acc;
    for (int i = 0; i < n_int; ++i) {
      const C a = xs[t + i], b = xs[i];
      acc.add(a.x * b.x + a.y * b.y);
    }
    out[(int64_t)blockIdx.x * n_lag + t] = (float)(acc.value() * scale);
  }
}

// FP32 Gaussian-window spectrum of N = R0 R1 frames.  One CTA holds the N x 16 tile cs(t, q0 .. q0 + 15)
// in registers: thread (column c, j) loads frames j + R1 k (128-byte segments per frame), the columns'
// sums meet through shared memory, the elastic mean is subtracted and the window applied in
// registers, and the transform goes on as a radix-R0 butterfly, one exchange through shared memory
// and a radix-R1 one, whose outputs (frequency g + R0 k) leave as |X|^2.  All but the exchange and the
// sums stays off shared memory: loading the tile there and transforming it in place took 68 % of the
// load/store wavefronts and 1.80 ms for 512 frames of 96^3 modes (4.5 GB), this form 1.44 ms with a
// CTA per tile (waiting on loads, its phases hardly overlapping) and 1.24 ms with resident CTAs whose
// next tile loads under the second butterfly; tiles of 32 columns (one CTA per SM) measure the same.
// Issue slots are 58 % busy then, DRAM 46 %.
// HALF: only frequencies up to N / 2 are wanted, so the others are not computed.
constexpr int kGaussQ = 16;
template <int N>
struct GaussPlan {
  static constexpr int R0 = N == 64 ? 8 : (N >= 512 ? 32 : 16), R1 = N / R0;
  static constexpr int NT = kGaussQ * R1;
  static constexpr int kBlocks = N == 1024 ? 1 : (N == 512 ? 2 : (N == 64 ? 8 : 768 / NT));
  static constexpr bool kAhead = N < 1024;     // both butterflies' registers do not fit there
};

template <int N, bool HALF>
__global__ void __launch_bounds__(GaussPlan<N>::NT, GaussPlan<N>::kBlocks)
    gauss_kernel(const float2* __restrict__ cs, int64_t nq, const float* __restrict__ gwin,
                 const float2* __restrict__ tab, int n_freq, const float* __restrict__ q2n, float scale,
                 float* __restrict__ out) {
  using P = GaussPlan<N>;
  constexpr int R0 = P::R0, R1 = P::R1, Q = kGaussQ, NW = P::NT / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* const xs = reinterpret_cast<float2*>(smem_raw);      // [N][Q]
  __shared__ float2 part[NW][Q], mean[Q];
  const int tid = threadIdx.x, c = tid % Q, j = tid / Q, warp = tid >> 5, lane = tid & 31;
  const int64_t tiles = (nq + Q - 1) / Q;
  float2 v[R0];
  auto load = [&](int64_t tile) {
    const int64_t q = tile * Q + c;
#pragma unroll
    for (int k = 0; k < R0; ++k)
      v[k] = q < nq ? __ldcs(cs + (int64_t)(j + R1 * k) * nq + q) : make_float2(0.f, 0.f);
  };
  if (P::kAhead) load(blockIdx.x);
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    if (!P::kAhead) load(tile);
    // the elastic mean, then the mean of what it leaves: the rounding of a sum over N frames of a strong
    // elastic line would stay in the lowest frequencies
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      float2 s = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < R0; ++k) s = s + v[k];
      s.x += __shfl_xor_sync(0xffffffffu, s.x, 16);              // the warp's other frame
      s.y += __shfl_xor_sync(0xffffffffu, s.y, 16);
      if (lane < Q) part[warp][lane] = s;
      __syncthreads();
      if (tid < Q) {
        float2 m = make_float2(0.f, 0.f);
        for (int w = 0; w < NW; ++w) m = m + part[w][tid];
        mean[tid] = make_float2(m.x / (float)N, m.y / (float)N);
      }
      __syncthreads();
      const float2 m = mean[c];
#pragma unroll
      for (int k = 0; k < R0; ++k) v[k] = v[k] - m;
    }
#pragma unroll
    for (int k = 0; k < R0; ++k) {
      const float g = __ldg(gwin + j + R1 * k);
      v[k] = make_float2(v[k].x * g, v[k].y * g);
    }
    Dft<float2, R0>::run(v);
#pragma unroll
    for (int k = 0; k < R0; ++k) {
      const float2 t = __ldg(tab + k * R1 + j);                  // exp(-2 pi i j k / N)
      xs[(k * R1 + j) * Q + c] = make_float2(v[k].x * t.x - v[k].y * t.y, v[k].x * t.y + v[k].y * t.x);
    }
    __syncthreads();
    if (P::kAhead && tile + gridDim.x < tiles) load(tile + gridDim.x);        // in flight under the second butterfly
    const int64_t q = tile * Q + c;
    const float w2 = q2n && q < nq ? q2n[q] * q2n[q] : 1.0f;
    for (int g = j; g < R0; g += R1) {
      float2 u[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) u[k] = xs[(g * R1 + k) * Q + c];
      Dft<float2, R1>::run(u);
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        const int f = g + R0 * k;
        if ((!HALF || 2 * k <= R1) && f < n_freq && q < nq)
          __stcs(out + (int64_t)f * nq + q, (u[k].x * u[k].x + u[k].y * u[k].y) * scale * w2);
      }
    }
  }
}

// ------------------------------------------------------------------------------- host
static int tile_cols(int nt, size_t csz, size_t extra, size_t limit) {
  int qt = 32;
  while (qt > 1 && (size_t)nt * qt * csz + extra > limit) qt >>= 1;
  if ((size_t)nt * qt * csz + extra > limit) return 0;
  return qt;
}

// Where a map is computed: the caller's device array, or memory of the call that out_finish copies to the
// host.
static int out_prepare(MapMem& mem, float* out, int host, size_t n, float** dev) {
  if (!out) return fail(MPSQ_ERR_ARG, "null output pointer");
  *dev = out;
  return host ? mem.take(kScratchOut, n * sizeof(float), reinterpret_cast<void**>(dev)) : MPSQ_OK;
}
static int out_finish(float* out, int host, size_t n, const float* dev, cudaStream_t s) {
  if (host) {
    cudaError_t e = cudaMemcpyAsync(out, dev, n * sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(MPSQ_ERR_CUDA, "output copy: %s", cudaGetErrorString(e));
  }
  return MPSQ_OK;
}

// Small host array -> memory of the call, in the order of the job's stream (a call does not wait for the
// work queued before it).
template <typename X>
static int dev_copy(MapMem& mem, JobScratch slot, const X* h, size_t n, X** d, cudaStream_t s) {
  *d = nullptr;
  if (!h) return MPSQ_OK;
  const int rc = mem.take(slot, n * sizeof(X), reinterpret_cast<void**>(d));
  if (rc) return rc;
  MPSQ_CUDA_TRY(cudaMemcpyAsync(*d, h, n * sizeof(X), cudaMemcpyHostToDevice, s));
  return MPSQ_OK;
}

template <int N>
static int launch_gauss(MapMem& mem, const float2* cs, int64_t nq, const float* gwin, int n_freq,
                        const float* q2n, float scale, float* out, cudaStream_t s) {
  using P = GaussPlan<N>;
  std::vector<float2> t(N);
  for (int k = 0; k < P::R0; ++k)
    for (int i = 0; i < P::R1; ++i) {
      const double a = -2.0 * M_PI * (double)((i * k) % N) / N;
      t[k * P::R1 + i] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
  float2* tab = nullptr;
  const int rc = dev_copy(mem, kScratchPath, (const float2*)t.data(), t.size(), &tab, s);
  if (rc) return rc;
  const size_t smem = (size_t)N * kGaussQ * sizeof(float2);
  const int64_t tiles = (nq + kGaussQ - 1) / kGaussQ;
  int dev = 0, sms = 0;
  MPSQ_CUDA_TRY(cudaGetDevice(&dev));
  MPSQ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const unsigned nb = (unsigned)std::min<int64_t>(tiles, (int64_t)P::kBlocks * sms);
  auto kern = n_freq <= N / 2 + 1 ? gauss_kernel<N, true> : gauss_kernel<N, false>;
  MPSQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<nb, P::NT, smem, s>>>(cs, nq, gwin, tab, n_freq, q2n, scale, out);
  return MPSQ_OK;
}

}  // namespace mpsq

using namespace mpsq;

extern "C" int mpsq_job_sq_total(mpsq_job* j, double norm2, float* out, int host) {
  if (!j) return fail(MPSQ_ERR_ARG, "sq_total: null job");
  PhaseRange range("mpsq:reduce");
  MapMem mem(j);
  JobView v = job_view(j);
  float* dev = nullptr;
  int rc = out_prepare(mem, out, host, v.n_q, &dev);
  if (rc) return rc;
  const double scale = 1.0 / ((double)v.n_frames * (norm2 > 0 ? norm2 : 1.0));
  const unsigned nb = (unsigned)((v.n_q + 255) / 256);
  if (v.precision == MPSQ_FP64)
    sq_total_kernel<double><<<nb, 256, 0, v.s>>>((const double2*)v.cs, v.n_q, v.n_frames, scale, dev);
  else
    sq_total_kernel<float><<<nb, 256, 0, v.s>>>((const float2*)v.cs, v.n_q, v.n_frames, scale, dev);
  MPSQ_LAUNCH_CHECK();
  return out_finish(out, host, v.n_q, dev, v.s);
}

// q2_norm and t_wind are host arrays (n_Q and n_int floats).
namespace {
// Source of a map: the weighted amplitudes (centred) or the raw sum of two stored species.
struct SeriesArgs {
  const void* a;
  const void* b;
  int64_t stride;
  int center;
};
SeriesArgs weighted_series(const JobView& v) { return {v.cs, nullptr, v.n_q, 1}; }
int pair_series(const JobView& v, int32_t sp1, int32_t sp2, const char* where, SeriesArgs* out) {
  if (!v.store_species || !v.cs_species)
    return fail(MPSQ_ERR_STATE, "%s: the atom-pair modes need a job created with store_species = 1", where);
  if (sp1 < 0 || sp2 < 0 || sp1 >= v.n_species || sp2 >= v.n_species)
    return fail(MPSQ_ERR_ARG, "%s: species %d, %d outside 0..%d", where, sp1, sp2, v.n_species - 1);
  const size_t csz = v.precision == MPSQ_FP64 ? 16 : 8;
  const char* base = (const char*)v.cs_species;
  out->a = base + (size_t)sp1 * v.n_q * csz;
  out->b = base + (size_t)sp2 * v.n_q * csz;
  out->stride = (int64_t)v.n_species * v.n_q;
  out->center = 0;
  return MPSQ_OK;
}
template <typename T>
Series<T> typed(const SeriesArgs& s) {
  using C = typename Cplx<T>::type;
  return Series<T>{(const C*)s.a, (const C*)s.b, s.stride, s.center};
}

int econst_impl(mpsq_job* j, const SeriesArgs& src, int32_t n_int, const float* t_wind,
                int32_t j_freq, const float* q2_norm, double scale, float* out, int host) {
  MapMem mem(j);
  JobView v = job_view(j);
  if (n_int < 1 || n_int > v.n_frames)
    return fail(MPSQ_ERR_ARG, "sqw_econst: n_int %d outside 1..n_frames (%d)", n_int, v.n_frames);
  if (j_freq < 1) return fail(MPSQ_ERR_ARG, "sqw_econst: j_freq must be >= 1");
  const size_t csz = v.precision == MPSQ_FP64 ? 16 : 8;
  const size_t extra = (size_t)n_int * csz + (size_t)2 * (256 + 32) * (csz / 2);
  const int QT = tile_cols(v.n_frames, csz, extra, 200 * 1024);   // (limit without the kStarts rows)
  if (QT == 0) return fail(MPSQ_ERR_ARG, "sqw_econst: %d frames do not fit in shared memory", v.n_frames);
  // threads: one per column and block of kStarts start frames, in equal rounds of at most 256
  const int blocks = (v.n_frames - n_int + kStarts) / kStarts;
  const int rounds = (blocks * QT + 255) / 256;
  const int NT = std::max(32, (blocks + rounds - 1) / rounds * QT + 31 & ~31);
  const size_t least = (size_t)(v.n_frames + kStarts) * QT * csz + (size_t)n_int * csz +
                       (size_t)2 * (NT + QT) * (csz / 2), with_win = least + (size_t)n_int * (csz / 2);
  const int win = with_win <= 227 * 1024 ? 1 : 0;   // the window in shared memory too
  const size_t smem = win ? with_win : least;
  float *dw = nullptr, *dq = nullptr;
  int rc = dev_copy(mem, kScratchWindow, t_wind, n_int, &dw, v.s);
  if (!rc) rc = dev_copy(mem, kScratchQ2, q2_norm, q2_norm ? v.n_q : 0, &dq, v.s);
  float* dev = nullptr;
  if (!rc) rc = out_prepare(mem, out, host, v.n_q, &dev);
  if (rc) return rc;
  const unsigned nb = (unsigned)((v.n_q + QT - 1) / QT);
  const int jf = j_freq - 1;
  if (v.precision == MPSQ_FP64) {
    cudaFuncSetAttribute(econst_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    econst_kernel<double><<<nb, NT, smem, v.s>>>(typed<double>(src), v.n_q, v.n_frames, QT, n_int,
                                                 dw, jf, dq, scale, win, dev);
  } else {
    cudaFuncSetAttribute(econst_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    econst_kernel<float><<<nb, NT, smem, v.s>>>(typed<float>(src), v.n_q, v.n_frames, QT, n_int, dw,
                                                jf, dq, scale, win, dev);
  }
  count_launch();
  cudaError_t e = cudaGetLastError();
  rc = e == cudaSuccess ? out_finish(out, host, v.n_q, dev, v.s)
                        : fail(MPSQ_ERR_CUDA, "econst launch: %s", cudaGetErrorString(e));
  return rc;
}

int dispersion_impl(mpsq_job* j, const SeriesArgs& src, int32_t n_int, const float* t_wind,
                    int32_t n_path, const int64_t* q_index, int32_t n_freq,
                    const float* q2_norm, double scale, float* out, int host) {
  MapMem mem(j);
  JobView v = job_view(j);
  if (n_int < 1 || n_int > v.n_frames) return fail(MPSQ_ERR_ARG, "sqw_dispersion: bad n_int");
  if (n_path < 1 || n_freq < 1 || n_freq > n_int) return fail(MPSQ_ERR_ARG, "sqw_dispersion: bad sizes");
  const size_t csz = v.precision == MPSQ_FP64 ? 16 : 8;
  const int NT = 256;
  const size_t base = (size_t)v.n_frames * csz + (size_t)n_int * csz + (size_t)2 * (128 + 2) * (csz / 2);
  if (base > 200 * 1024) return fail(MPSQ_ERR_ARG, "sqw_dispersion: too many frames");
  const size_t least = (size_t)(v.n_frames + kStarts + n_int) * csz + (size_t)2 * (NT + 2) * (csz / 2);
  const size_t with_win = least + (size_t)n_int * (csz / 2);
  const int win = with_win + 8 + (size_t)kSlots * sizeof(double) <= 227 * 1024 ? 1 : 0;
  const size_t sum_off = ((win ? with_win : least) + 7) & ~size_t(7);
  const int64_t slots = (int64_t)n_freq * ((v.n_frames - n_int + kStarts) / kStarts);
  const size_t smem = sum_off + (size_t)std::min<int64_t>(slots, kSlots) * sizeof(double);
  float *dw = nullptr, *dq = nullptr;
  int64_t* di = nullptr;
  int rc = dev_copy(mem, kScratchWindow, t_wind, n_int, &dw, v.s);
  if (!rc) rc = dev_copy(mem, kScratchQ2, q2_norm, q2_norm ? v.n_q : 0, &dq, v.s);
  if (!rc) rc = dev_copy(mem, kScratchPath, q_index, n_path, &di, v.s);
  float* dev = nullptr;
  if (!rc) rc = out_prepare(mem, out, host, (size_t)n_path * n_freq, &dev);
  if (rc) return rc;
  if (v.precision == MPSQ_FP64) {
    cudaFuncSetAttribute(dispersion_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    dispersion_kernel<double><<<n_path, NT, smem, v.s>>>(typed<double>(src), v.n_q, v.n_frames, di,
                                                         n_int, dw, n_freq, dq, scale, (int)sum_off, win, dev);
  } else {
    cudaFuncSetAttribute(dispersion_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    dispersion_kernel<float><<<n_path, NT, smem, v.s>>>(typed<float>(src), v.n_q, v.n_frames, di,
                                                        n_int, dw, n_freq, dq, scale, (int)sum_off, win, dev);
  }
  count_launch();
  cudaError_t e = cudaGetLastError();
  rc = e == cudaSuccess ? out_finish(out, host, (size_t)n_path * n_freq, dev, v.s)
                        : fail(MPSQ_ERR_CUDA, "dispersion launch: %s", cudaGetErrorString(e));
  return rc;
}
}  // namespace

extern "C" int mpsq_job_sqw_econst(mpsq_job* j, int32_t n_int, const float* t_wind,
                                   int32_t j_freq, const float* q2_norm, double scale,
                                   float* out, int host) {
  PhaseRange range("mpsq:time");
  if (!j || !t_wind) return fail(MPSQ_ERR_ARG, "sqw_econst: null pointer");
  return econst_impl(j, weighted_series(job_view(j)), n_int, t_wind, j_freq, q2_norm, scale, out,
                     host);
}

extern "C" int mpsq_job_sqw_econst_pair(mpsq_job* j, int32_t n_int, const float* t_wind,
                                        int32_t j_freq, int32_t sp1, int32_t sp2, double scale,
                                        float* out, int host) {
  PhaseRange range("mpsq:time");
  if (!j || !t_wind) return fail(MPSQ_ERR_ARG, "sqw_econst_pair: null pointer");
  SeriesArgs src;
  const int rc = pair_series(job_view(j), sp1, sp2, "sqw_econst_pair", &src);
  if (rc) return rc;
  return econst_impl(j, src, n_int, t_wind, j_freq, nullptr, scale, out, host);
}

extern "C" int mpsq_job_sqw_dispersion(mpsq_job* j, int32_t n_int, const float* t_wind,
                                       int32_t n_path, const int64_t* q_index, int32_t n_freq,
                                       const float* q2_norm, double scale, float* out,
                                       int host) {
  PhaseRange range("mpsq:time");
  if (!j || !t_wind || !q_index) return fail(MPSQ_ERR_ARG, "sqw_dispersion: null pointer");
  return dispersion_impl(j, weighted_series(job_view(j)), n_int, t_wind, n_path, q_index, n_freq,
                         q2_norm, scale, out, host);
}

extern "C" int mpsq_job_sqw_dispersion_pair(mpsq_job* j, int32_t n_int, const float* t_wind,
                                            int32_t n_path, const int64_t* q_index,
                                            int32_t n_freq, int32_t sp1, int32_t sp2,
                                            double scale, float* out, int host) {
  PhaseRange range("mpsq:time");
  if (!j || !t_wind || !q_index) return fail(MPSQ_ERR_ARG, "sqw_dispersion_pair: null pointer");
  SeriesArgs src;
  const int rc = pair_series(job_view(j), sp1, sp2, "sqw_dispersion_pair", &src);
  if (rc) return rc;
  return dispersion_impl(j, src, n_int, t_wind, n_path, q_index, n_freq, nullptr, scale, out,
                         host);
}

extern "C" int mpsq_job_iqt(mpsq_job* j, int32_t n_int, int32_t lag, const float* q2_norm,
                            double scale, float* out, int host) {
  PhaseRange range("mpsq:time");
  if (!j) return fail(MPSQ_ERR_ARG, "iqt: null job");
  MapMem mem(j);
  JobView v = job_view(j);
  if (n_int < 1 || lag < 0 || lag + n_int > v.n_frames)
    return fail(MPSQ_ERR_ARG, "iqt: lag %d + n_int %d exceeds n_frames %d", lag, n_int, v.n_frames);
  const size_t csz = v.precision == MPSQ_FP64 ? 16 : 8;
  const int NT = 256;
  const size_t extra = (size_t)2 * (NT + 32) * (csz / 2);
  const int QT = tile_cols(v.n_frames, csz, extra, 200 * 1024);
  if (QT == 0) return fail(MPSQ_ERR_ARG, "iqt: %d frames do not fit in shared memory", v.n_frames);
  const size_t smem = (size_t)v.n_frames * QT * csz + (size_t)2 * (NT + QT) * (csz / 2);
  float* dq = nullptr;
  int rc = dev_copy(mem, kScratchQ2, q2_norm, q2_norm ? v.n_q : 0, &dq, v.s);
  float* dev = nullptr;
  if (!rc) rc = out_prepare(mem, out, host, v.n_q, &dev);
  if (rc) return rc;
  const unsigned nb = (unsigned)((v.n_q + QT - 1) / QT);
  const SeriesArgs src = weighted_series(v);
  if (v.precision == MPSQ_FP64) {
    cudaFuncSetAttribute(iqt_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    iqt_kernel<double><<<nb, NT, smem, v.s>>>(typed<double>(src), v.n_q, v.n_frames, QT, n_int, lag,
                                              dq, scale, dev);
  } else {
    cudaFuncSetAttribute(iqt_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    iqt_kernel<float><<<nb, NT, smem, v.s>>>(typed<float>(src), v.n_q, v.n_frames, QT, n_int, lag,
                                             dq, scale, dev);
  }
  count_launch();
  cudaError_t e = cudaGetLastError();
  rc = e == cudaSuccess ? out_finish(out, host, v.n_q, dev, v.s)
                        : fail(MPSQ_ERR_CUDA, "iqt launch: %s", cudaGetErrorString(e));
  return rc;
}

extern "C" int mpsq_job_iqt_dispersion(mpsq_job* j, int32_t n_int, int32_t n_path,
                                       const int64_t* q_index, const float* q2_norm,
                                       double scale, float* out, int host) {
  PhaseRange range("mpsq:time");
  if (!j || !q_index) return fail(MPSQ_ERR_ARG, "iqt_dispersion: null pointer");
  MapMem mem(j);
  JobView v = job_view(j);
  if (n_int < 1 || n_int > v.n_frames || n_path < 1)
    return fail(MPSQ_ERR_ARG, "iqt_dispersion: bad sizes");
  const int n_lag = v.n_frames - n_int + 1;
  const size_t csz = v.precision == MPSQ_FP64 ? 16 : 8;
  const int NT = 128;
  const size_t smem = (size_t)v.n_frames * csz + (size_t)2 * (NT + 2) * (csz / 2);
  if (smem > 200 * 1024) return fail(MPSQ_ERR_ARG, "iqt_dispersion: too many frames");
  float* dq = nullptr;
  int64_t* di = nullptr;
  int rc = dev_copy(mem, kScratchQ2, q2_norm, q2_norm ? v.n_q : 0, &dq, v.s);
  if (!rc) rc = dev_copy(mem, kScratchPath, q_index, n_path, &di, v.s);
  float* dev = nullptr;
  if (!rc) rc = out_prepare(mem, out, host, (size_t)n_path * n_lag, &dev);
  if (rc) return rc;
  const SeriesArgs src = weighted_series(v);
  if (v.precision == MPSQ_FP64) {
    cudaFuncSetAttribute(iqt_dispersion_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    iqt_dispersion_kernel<double><<<n_path, NT, smem, v.s>>>(typed<double>(src), v.n_q, v.n_frames,
                                                             di, n_int, dq, scale, dev);
  } else {
    cudaFuncSetAttribute(iqt_dispersion_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    iqt_dispersion_kernel<float><<<n_path, NT, smem, v.s>>>(typed<float>(src), v.n_q, v.n_frames,
                                                            di, n_int, dq, scale, dev);
  }
  count_launch();
  cudaError_t e = cudaGetLastError();
  rc = e == cudaSuccess ? out_finish(out, host, (size_t)n_path * n_lag, dev, v.s)
                        : fail(MPSQ_ERR_CUDA, "iqt_dispersion launch: %s", cudaGetErrorString(e));
  return rc;
}

extern "C" int mpsq_job_sqw_gauss(mpsq_job* j, double fwhm_frames, int32_t n_freq,
                                  const float* q2_norm, double scale, float* out, int host) {
  PhaseRange range("mpsq:time");
  if (!j) return fail(MPSQ_ERR_ARG, "sqw_gauss: null job");
  MapMem mem(j);
  JobView v = job_view(j);
  const int nt = v.n_frames;
  if (nt < 2 || nt > 1024 || (nt & (nt - 1)))
    return fail(MPSQ_ERR_ARG, "sqw_gauss: n_frames (%d) must be a power of two in 2..1024", nt);
  if (n_freq < 1 || n_freq > nt) return fail(MPSQ_ERR_ARG, "sqw_gauss: n_freq outside 1..n_frames");
  if (!(fwhm_frames > 0)) return fail(MPSQ_ERR_ARG, "sqw_gauss: fwhm must be > 0");
  int logn = 0;
  while ((1 << logn) < nt) ++logn;
  const size_t csz = v.precision == MPSQ_FP64 ? 16 : 8;
  const int NT = 256;
  const size_t extra = (size_t)(nt / 2) * csz + (size_t)2 * (NT + 32) * (csz / 2);
  const int QT = tile_cols(nt, csz, extra, 160 * 1024);
  if (QT == 0) return fail(MPSQ_ERR_ARG, "sqw_gauss: tile does not fit");
  const size_t smem = (size_t)nt * QT * csz + (size_t)(nt / 2) * csz + (size_t)2 * (NT + QT) * (csz / 2);
  std::vector<float> g(nt);
  const double tc = 0.5 * (nt - 1);
  for (int t = 0; t < nt; ++t) {
    const double u = (t - tc) / fwhm_frames;
    g[t] = (float)std::exp(-4.0 * std::log(2.0) * u * u);
  }
  float *dg = nullptr, *dq = nullptr;
  int rc = dev_copy(mem, kScratchWindow, (const float*)g.data(), nt, &dg, v.s);
  if (!rc) rc = dev_copy(mem, kScratchQ2, q2_norm, q2_norm ? v.n_q : 0, &dq, v.s);
  float* dev = nullptr;
  if (!rc) rc = out_prepare(mem, out, host, (size_t)n_freq * v.n_q, &dev);
  if (rc) return rc;
  const unsigned nb = (unsigned)((v.n_q + QT - 1) / QT);
  if (v.precision == MPSQ_FP64) {
    cudaFuncSetAttribute(gauss_fft_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    gauss_fft_kernel<double><<<nb, NT, smem, v.s>>>(typed<double>(weighted_series(v)), v.n_q, nt, logn, QT, dg,
                                                    n_freq, dq, scale, dev);
  } else if (nt >= 64) {
    const float2* cs = (const float2*)v.cs;
    const float sc = (float)scale;
    switch (nt) {
      case 64: rc = launch_gauss<64>(mem, cs, v.n_q, dg, n_freq, dq, sc, dev, v.s); break;
      case 128: rc = launch_gauss<128>(mem, cs, v.n_q, dg, n_freq, dq, sc, dev, v.s); break;
      case 256: rc = launch_gauss<256>(mem, cs, v.n_q, dg, n_freq, dq, sc, dev, v.s); break;
      case 512: rc = launch_gauss<512>(mem, cs, v.n_q, dg, n_freq, dq, sc, dev, v.s); break;
      default: rc = launch_gauss<1024>(mem, cs, v.n_q, dg, n_freq, dq, sc, dev, v.s); break;
    }
    if (rc) return rc;
  } else {
    cudaFuncSetAttribute(gauss_fft_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    gauss_fft_kernel<float><<<nb, NT, smem, v.s>>>(typed<float>(weighted_series(v)), v.n_q, nt, logn, QT, dg,
                                                   n_freq, dq, scale, dev);
  }
  count_launch();
  cudaError_t e = cudaGetLastError();
  rc = e == cudaSuccess ? out_finish(out, host, (size_t)n_freq * v.n_q, dev, v.s)
                        : fail(MPSQ_ERR_CUDA, "gauss launch: %s", cudaGetErrorString(e));
  return rc;
}

// ------------------------------------------------------------- spherical |Q| histogram
namespace mpsq {
// Fortran NORM2 of a 3-vector as the scaled sum of squares (the recurrence of BLAS snrm2):
// scale tracks the largest |component|, ssq the sum of squares relative to it.  Every
// operation is a separately rounded FP32 op (no contraction into fused multiply-adds).
__device__ __forceinline__ float norm2_scaled(float x, float y, float z) {
  float scale = 0.0f, ssq = 1.0f;
  const float c[3] = {x, y, z};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float a = fabsf(c[i]);
    if (a != 0.0f) {
      if (scale < a) {
        const float r = __fdiv_rn(scale, a);
        ssq = __fadd_rn(1.0f, __fmul_rn(ssq, __fmul_rn(r, r)));
        scale = a;
      } else {
        const float r = __fdiv_rn(a, scale);
        ssq = __fadd_rn(ssq, __fmul_rn(r, r));
      }
    }
  }
  return __fmul_rn(scale, __fsqrt_rn(ssq));
}

__device__ __forceinline__ float dot3_rn(float3 a, float v0, float v1, float v2) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a.x, v0), __fmul_rn(a.y, v1)), __fmul_rn(a.z, v2));
}

// Grid-stride over modes; a CTA accumulates its bins in shared memory (FP32 partial sums of a
// few thousand products) and flushes them to the FP64 output with atomics.
template <typename T>
__global__ void radial_hist_kernel(const typename Cplx<T>::type* __restrict__ amps, int s_stride,
                                   int S, int64_t nq, int nt, int m0, int m1, int m2, float3 r0,
                                   float3 r1, float3 r2, float3 dq, float q_step, float q_range,
                                   int n_hist, float scale2, int use_smem,
                                   double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* h = reinterpret_cast<float*>(smem_raw);
  const int nb = S * S * n_hist;
  if (use_smem) {
    for (int e = threadIdx.x; e < nb; e += blockDim.x) h[e] = 0.0f;
    __syncthreads();
  }
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nq;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % m0), j = (int)((q / m0) % m1), l = (int)(q / ((int64_t)m0 * m1));
    // v = k * d_q, Q = a_cell_inv v, |Q| = NORM2(Q), all in FP32 (mp_sql56.f90:1041)
    const float v0 = __fmul_rn((float)(i - m0 / 2), dq.x);
    const float v1 = __fmul_rn((float)(j - m1 / 2), dq.y);
    const float v2 = __fmul_rn((float)(l - m2 / 2), dq.z);
    const float qn = norm2_scaled(dot3_rn(r0, v0, v1, v2), dot3_rn(r1, v0, v1, v2),
                                  dot3_rn(r2, v0, v1, v2));
    if (!(qn <= q_range)) continue;
    const int bin = (int)roundf(__fdiv_rn(qn, q_step));   // NINT: half away from zero
    if (bin < 0 || bin >= n_hist) continue;
    for (int t = 0; t < nt; ++t) {
      for (int a = 0; a < S; ++a) {
        const auto A = amps[((int64_t)t * s_stride + a) * nq + q];
        for (int b = 0; b < S; ++b) {
          const auto B = amps[((int64_t)t * s_stride + b) * nq + q];
          const float v = (float)(A.x * B.x + A.y * B.y) * scale2;
          const int e = (a * S + b) * n_hist + bin;
          if (use_smem)
            atomicAdd(&h[e], v);
          else
            atomicAdd(&out[e], (double)v);
        }
      }
    }
  }
  if (use_smem) {
    __syncthreads();
    for (int e = threadIdx.x; e < nb; e += blockDim.x)
      if (h[e] != 0.0f) atomicAdd(&out[e], (double)h[e]);
  }
}
}  // namespace mpsq

extern "C" int mpsq_job_radial_hist(mpsq_job* j, const double* a_cell_inv, const double* d_q,
                                    double q_step, double q_range, int32_t n_hist,
                                    double amp_scale, double* out, int host) {
  if (!j || !a_cell_inv || !d_q || !out) return fail(MPSQ_ERR_ARG, "radial_hist: null pointer");
  MapMem mem(j);
  JobView v = job_view(j);
  if (v.slab) return fail(MPSQ_ERR_STATE, "radial_hist: needs the whole Q store (job has a q_slab)");
  if (n_hist < 1 || !(q_step > 0)) return fail(MPSQ_ERR_ARG, "radial_hist: bad bins");
  const void* amps = v.cs;
  int S = 1, s_stride = 1;
  if (v.store_species) {
    amps = v.cs_species;
    S = v.n_species;
    s_stride = v.n_species;
  } else if (v.n_species != 1) {
    return fail(MPSQ_ERR_STATE, "radial_hist: per-species amplitudes need store_species = 1");
  }
  const size_t nb = (size_t)S * S * n_hist;
  double* dev = nullptr;
  if (const int rc = mem.take(kScratchOut, nb * sizeof(double), reinterpret_cast<void**>(&dev))) return rc;
  MPSQ_CUDA_TRY(cudaMemsetAsync(dev, 0, nb * sizeof(double), v.s));
  const size_t smem = nb * sizeof(float);
  const int use_smem = smem <= 96 * 1024 ? 1 : 0;
  const double* A = a_cell_inv;
  const float3 r0 = make_float3((float)A[0], (float)A[1], (float)A[2]);
  const float3 r1 = make_float3((float)A[3], (float)A[4], (float)A[5]);
  const float3 r2 = make_float3((float)A[6], (float)A[7], (float)A[8]);
  const float3 dq = make_float3((float)d_q[0], (float)d_q[1], (float)d_q[2]);
  const float scale2 = (float)(amp_scale * amp_scale);
  const unsigned blocks = (unsigned)std::min<int64_t>((v.n_q + 255) / 256, 152 * 8);
  if (v.precision == MPSQ_FP64) {
    cudaFuncSetAttribute(radial_hist_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    radial_hist_kernel<double><<<blocks, 256, use_smem ? smem : 0, v.s>>>(
        (const double2*)amps, s_stride, S, v.n_q, v.n_frames, (int)v.m[0], (int)v.m[1], (int)v.m[2],
        r0, r1, r2, dq, (float)q_step, (float)q_range, n_hist, scale2, use_smem, dev);
  } else {
    cudaFuncSetAttribute(radial_hist_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    radial_hist_kernel<float><<<blocks, 256, use_smem ? smem : 0, v.s>>>(
        (const float2*)amps, s_stride, S, v.n_q, v.n_frames, (int)v.m[0], (int)v.m[1], (int)v.m[2],
        r0, r1, r2, dq, (float)q_step, (float)q_range, n_hist, scale2, use_smem, dev);
  }
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) {
    if (host) {
      e = cudaMemcpyAsync(out, dev, nb * sizeof(double), cudaMemcpyDeviceToHost, v.s);
    } else {
      e = cudaMemcpyAsync(out, dev, nb * sizeof(double), cudaMemcpyDeviceToDevice, v.s);
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(v.s);
  if (e != cudaSuccess) return fail(MPSQ_ERR_CUDA, "radial_hist: %s", cudaGetErrorString(e));
  return MPSQ_OK;
}
