// Pruned fine-grid transform of FP32 grids: passes X, Y and Z (passes.h).
//
// A line of length N = R0 R1 R2 (R1 = 1: two stages) is transformed by decimation in frequency.  The
// first stage works on registers straight from global memory (element j + (N/R0) k of a line in
// register k: neighbouring threads load neighbouring elements, or neighbouring lines), the last one
// leaves its kept frequencies straight from registers, and shared memory only carries the exchange
// between stages: one write and one read per point in two stages.  Loading a tile into shared memory,
// transforming in place and staging the output took five passes over shared memory, and its bandwidth
// (89 % of the load/store wavefronts) was what bounded pass X.  Measured before and after, per launch:
// one 384^3 grid X 160 -> 117 us (680 MB: 86 % of the copy rate), Y 91 -> 79, Z 88 -> 71; three 512^3
// grids X 1129 -> 857, Y 708 -> 549; three 1152^3 grids X, Y and Z together 42.4 -> 26.5 ms.
//
// After stage 0, block k0 of N/R0 elements holds the frequencies f = k0 (mod R0); stage 1 splits each
// block the same way; the last stage leaves frequency k0 + R0 (k1 + R1 k2).  Only f in [-N/4, N/4] is
// kept, so about half the outputs of the last stage are neither stored nor computed.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "dft.cuh"
#include "passes.h"

namespace mpsq {
namespace {

struct Split {
  int r0, r1, r2;
};
constexpr Split split_of(int n) {
  switch (n) {
    case 32: return {4, 1, 8};
    case 64: return {8, 1, 8};
    case 96: return {8, 1, 12};
    case 128: return {8, 1, 16};
    case 160: return {16, 1, 10};
    case 192: return {16, 1, 12};
    case 256: return {16, 1, 16};
    case 288: return {24, 1, 12};
    case 320: return {16, 1, 20};
    case 384: return {16, 1, 24};
    case 480: return {24, 1, 20};
    case 512: return {16, 1, 32};
    case 576: return {24, 1, 24};
    case 640: return {8, 8, 10};
    case 768: return {8, 8, 12};
    case 800: return {10, 8, 10};
    case 864: return {9, 8, 12};
    case 960: return {10, 8, 12};
    case 1024: return {8, 8, 16};
    case 1152: return {12, 8, 12};
    case 1280: return {16, 8, 10};
    case 1440: return {12, 10, 12};
    case 1536: return {12, 8, 16};
    case 1600: return {16, 10, 10};
    default: return {1, 1, 1};
  }
}
template <int N>
struct Plan {
  static constexpr int R0 = split_of(N).r0, R1 = split_of(N).r1, R2 = split_of(N).r2;
  static constexpr int M = N / R0;                 // block length after stage 0
  static_assert(R0 * R1 * R2 == N && R2 > 1, "no plan for this length");
};
constexpr int round32(int n) { return (n + 31) / 32 * 32; }

__device__ __forceinline__ float2 cmulf2(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// Whether output k of the last stage can be a kept frequency (|f| <= N / 4).
constexpr bool kept_output(int k, int r2) { return 4 * k <= r2 || 4 * k > 3 * r2 - 4; }
// Index of frequency f in [-h, h], or -1.
__device__ __forceinline__ int kept_index(int f, int N, int h) {
  return f <= h ? f + h : (f >= N - h ? f - N + h : -1);
}

// Twiddle tables of a length: stage 0 exp(-2 pi i j k0 / N) at [k0][j], j < M, then stage 1
// exp(-2 pi i j2 k1 / (R1 R2)) at [k1][j2].
template <int N>
__device__ __forceinline__ void twiddle0(float2* v, const float2* __restrict__ tab, int j) {
  using P = Plan<N>;
#pragma unroll
  for (int k = 1; k < P::R0; ++k) v[k] = cmulf2(v[k], __ldg(tab + k * P::M + j));
}
template <int N>
__device__ __forceinline__ void twiddle1(float2* v, const float2* __restrict__ tab, int j2) {
  using P = Plan<N>;
#pragma unroll
  for (int k = 1; k < P::R1; ++k) v[k] = cmulf2(v[k], __ldg(tab + N + k * P::R2 + j2));
}

// Pass X: L contiguous rows per CTA.  Row-major exchange buffer: element (k0, k1, j2) of a row at k0 PK +
// k1 P2 + j2 with odd pitches, which spread the last stage's reads over the banks.
template <int N>
constexpr int x_p2() { return Plan<N>::R2 | 1; }
template <int N>
constexpr int x_pk() { return (Plan<N>::R1 * x_p2<N>()) | 1; }
template <int N, int L>
constexpr int x_threads() {
  using P = Plan<N>;
  const int most = round32(L * (P::M > P::R0 * P::R1 ? P::M : P::R0 * P::R1));
  return most < 256 ? most : 256;
}
template <int N, int L>
constexpr int x_smem() {
  using P = Plan<N>;
  return L * P::R0 * x_pk<N>() * (int)sizeof(float2);
}
template <int N, int L>
__global__ void __launch_bounds__(x_threads<N, L>(), (Plan<N>::R2 > 24 || Plan<N>::R0 > 16 ? 512 : 768) / x_threads<N, L>())
    fftx_kernel(const float2* __restrict__ fine, int64_t n_rows, const float2* __restrict__ tab, int h0,
                int K0, float2* __restrict__ b1) {
  using P = Plan<N>;
  constexpr int NT = x_threads<N, L>(), R0 = P::R0, R1 = P::R1, R2 = P::R2, M = P::M, P2 = x_p2<N>(), PK = x_pk<N>();
  constexpr int LS = R0 * PK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* const xs = reinterpret_cast<float2*>(smem_raw);
  const int tid = threadIdx.x;
  const int64_t row0 = (int64_t)blockIdx.x * L;
  const int rows = (int)min((int64_t)L, n_rows - row0);
  const float2* const src = fine + row0 * N;
#pragma unroll
  for (int e0 = 0; e0 < L * M; e0 += NT) {
    const int e = e0 + tid, ln = e / M, j = e - ln * M;
    if (e < L * M && ln < rows) {
      float2 v[R0];
#pragma unroll
      for (int k = 0; k < R0; ++k) v[k] = __ldcs(src + ln * N + j + M * k);
      Dft<float2, R0>::run(v);
      twiddle0<N>(v, tab, j);
      float2* const q = xs + ln * LS + (j / R2) * P2 + j % R2;
#pragma unroll
      for (int k = 0; k < R0; ++k) q[k * PK] = v[k];
    }
  }
  __syncthreads();
  if constexpr (R1 > 1) {
    for (int e = tid; e < L * R0 * R2; e += NT) {
      const int ln = e / (R0 * R2), r = e - ln * (R0 * R2), k0 = r / R2, j2 = r - k0 * R2;
      float2* const q = xs + ln * LS + k0 * PK + j2;
      float2 v[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) v[k] = q[k * P2];
      Dft<float2, R1>::run(v);
      twiddle1<N>(v, tab, j2);
#pragma unroll
      for (int k = 0; k < R1; ++k) q[k * P2] = v[k];
    }
    __syncthreads();
  }
  for (int e = tid; e < L * R0 * R1; e += NT) {
    const int ln = e / (R0 * R1), u = e - ln * (R0 * R1), k0 = u % R0, k1 = u / R0;
    if (ln >= rows) break;
    const float2* const q = xs + ln * LS + k0 * PK + k1 * P2;
    float2 v[R2];
#pragma unroll
    for (int k = 0; k < R2; ++k) v[k] = q[k];
    Dft<float2, R2>::run(v);
    float2* const dst = b1 + (row0 + ln) * K0;
#pragma unroll
    for (int k = 0; k < R2; ++k)
      if (kept_output(k, R2)) {
        const int i = kept_index(u + R0 * R1 * k, N, h0);
        if (i >= 0) dst[i] = v[k];
      }
  }
}

// Passes Y and Z hold 16 lines, lines fastest: element at position p (after stage 0: k0 M + j) of
// line c at xs[16 p + c].
constexpr int kLines = 16;
template <int N>
constexpr int yz_threads() {
  using P = Plan<N>;
  const int most = 16 * (P::M > P::R0 * P::R1 ? P::M : P::R0 * P::R1);
  // few large CTAs where the tile leaves room for one or two per SM
  const int cap = N * 128 > 110 * 1024 ? 768 : (P::R2 > 24 || P::R0 > 16 ? 256 : 384);
  return round32(most < cap ? most : cap);
}
template <int N>
constexpr int yz_blocks() {   // CTAs per SM by registers (at most 80 or 128 a thread) and memory
  using P = Plan<N>;
  const int by_reg = (P::R2 > 24 || P::R0 > 16 ? 512 : 768) / yz_threads<N>();
  const int by_mem = 220 * 1024 / (N * 128 + 1024);
  const int b = by_reg < by_mem ? by_reg : by_mem;
  return b < 1 ? 1 : b;
}

// Stages 1 and last of 16 lines; store(f, line, value) takes the last stage's outputs that can be
// kept, in place at the position it is given.
template <int N, class Swz>
__device__ __forceinline__ void middle_stage16(float2* xs, const float2* __restrict__ tab, const Swz& at) {
  using P = Plan<N>;
  constexpr int R0 = P::R0, R1 = P::R1, R2 = P::R2;
  for (int e = threadIdx.x; e < kLines * R0 * R2; e += blockDim.x) {
    const int c = e % kLines, r = e / kLines, k0 = r / R2, j2 = r - k0 * R2;
    float2 v[R1];
#pragma unroll
    for (int k = 0; k < R1; ++k) v[k] = xs[at((k0 * R1 + k) * R2 + j2, c)];
    Dft<float2, R1>::run(v);
    twiddle1<N>(v, tab, j2);
#pragma unroll
    for (int k = 0; k < R1; ++k) xs[at((k0 * R1 + k) * R2 + j2, c)] = v[k];
  }
  __syncthreads();
}

// Pass Y: 16 consecutive x-columns (length N along y, stride K0) of one z-plane per CTA.
template <int N>
__global__ void __launch_bounds__(yz_threads<N>(), yz_blocks<N>())
    ffty_kernel(const float2* __restrict__ b1, int n2in, int n2, int zoff, int K0,
                const float2* __restrict__ tab, int h1, int K1, float2* __restrict__ b2) {
  using P = Plan<N>;
  constexpr int NT = yz_threads<N>(), R0 = P::R0, R1 = P::R1, R2 = P::R2, M = P::M;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* const xs = reinterpret_cast<float2*>(smem_raw);
  const int tid = threadIdx.x, c = tid % kLines;
  const int x = blockIdx.x * kLines + c, z = blockIdx.y, g = blockIdx.z;
  const bool live = x < K0;
  const float2* const src = b1 + ((int64_t)g * n2in + z) * (int64_t)N * K0 + x;
#pragma unroll
  for (int j0 = 0; j0 < M; j0 += NT / kLines) {
    const int j = j0 + tid / kLines;
    if (j < M && live) {
      float2 v[R0];
#pragma unroll
      for (int k = 0; k < R0; ++k) v[k] = __ldcs(src + (int64_t)(j + M * k) * K0);
      Dft<float2, R0>::run(v);
      twiddle0<N>(v, tab, j);
#pragma unroll
      for (int k = 0; k < R0; ++k) xs[(k * M + j) * kLines + c] = v[k];
    }
  }
  __syncthreads();
  if constexpr (R1 > 1) middle_stage16<N>(xs, tab, [](int p, int c) { return p * kLines + c; });
  if (!live) return;
  float2* const dst = b2 + ((int64_t)g * n2 + zoff + z) * (int64_t)K1 * K0 + x;
  for (int u = tid / kLines; u < R0 * R1; u += NT / kLines) {
    const int k0 = u % R0, k1 = u / R0;
    float2 v[R2];
#pragma unroll
    for (int k = 0; k < R2; ++k) v[k] = xs[((k0 * R1 + k1) * R2 + k) * kLines + c];
    Dft<float2, R2>::run(v);
#pragma unroll
    for (int k = 0; k < R2; ++k)
      if (kept_output(k, R2)) {
        const int i = kept_index(u + R0 * R1 * k, N, h1);
        if (i >= 0) dst[(int64_t)i * K0] = v[k];
      }
  }
}

// |Q|^2 as the exponent variable of the form factors at mode (kx, ky, kz) (0 without them).
__device__ __forceinline__ float q_square(const WeightArgs& w, int kx, int ky, int kz) {
  if (w.weight_mode != MPSQ_WEIGHT_XRAY) return 0.f;
  float qv[3];
#pragma unroll
  for (int b = 0; b < 3; ++b)
    qv[b] = w.q0_f[b] + (float)kx * w.qs_f[0][b] + (float)ky * w.qs_f[1][b] + (float)kz * w.qs_f[2][b];
  return w.kappa_f * (qv[0] * qv[0] + qv[1] * qv[1] + qv[2] * qv[2] + w.extra_f);
}

// Pass Z fused with the deconvolution.  CTA (x tile, ky index iy <= h1, frame) transforms, for every
// grid of the frame, the 8 z-columns P = (iy, x0 ..) and their mirrors M = (2 h1 - iy, 2 h0 - x), and
// forms both the modes k of the P columns and the modes -k of the M columns: either needs just P at
// frequency f and M at -f (the pair separation of k reads G(k) and G(-k)), and their weights are the
// same where |Q(-k)| = |Q(k)|.  A row that is its own mirror (iy = h1, and the single row of a plane)
// covers x > h0 as the M modes of x < h0.
template <int N>
__global__ void __launch_bounds__(yz_threads<N>(), yz_blocks<N>())
    fftz_deconv_kernel(const float2* __restrict__ b2, int K0, int K1, int m0, int m1, int m2, int z0,
                       int nz, int h0, int h1, int h2, int ngroups, const float2* __restrict__ tab,
                       const float* __restrict__ c0, const float* __restrict__ c1,
                       const float* __restrict__ c2, WeightArgs w, float2* __restrict__ cs_frame,
                       float2* __restrict__ cs_species_frame) {
  using P = Plan<N>;
  constexpr int NT = yz_threads<N>(), R0 = P::R0, R1 = P::R1, R2 = P::R2, M = P::M, T = kLines / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* const xs = reinterpret_cast<float2*>(smem_raw);
  // the halves of a row change places with the parity of its block and position, so that the output
  // loop's half-rows (8 P or 8 M lines of neighbouring frequencies) fall on different banks
  auto at = [](int p, int c) { return p * kLines + (c ^ (((p / M + p) & 1) << 3)); };
  const int tid = threadIdx.x, c = tid % kLines;
  const int x0 = blockIdx.x * T, iy = blockIdx.y, iym = 2 * h1 - iy;
  if (iym == iy && x0 > h0) return;                        // covered by the mirror modes
  const bool mrow = iym < m1;
  const int xp = iym == iy ? h0 + 1 : m0, xq = iym == iy ? h0 : (mrow ? K0 : 0);   // P modes x < xp, M modes x < xq
  const int64_t nm = (int64_t)m0 * m1 * nz;                // modes per frame in the store
  float2* const cs = cs_frame + (int64_t)blockIdx.z * nm;
  const int lx = x0 + (c & (T - 1));                       // this thread's line
  const bool mirror = c >= T;
  const int64_t col = mirror ? (int64_t)iym * K0 + (2 * h0 - lx) : (int64_t)iy * K0 + lx;
  for (int g = 0; g < ngroups; ++g) {
    const int pair = w.pair[g];
    const bool live = lx < K0 && (!mirror || pair || mrow);
    const float2* const src = b2 + ((int64_t)blockIdx.z * ngroups + g) * N * K1 * K0 + col;
    const int64_t step = (int64_t)K1 * K0;
    if (g > 0) __syncthreads();                            // the previous group's outputs have been read
#pragma unroll
    for (int j0 = 0; j0 < M; j0 += NT / kLines) {
      const int j = j0 + tid / kLines;
      if (j < M && live) {
        float2 v[R0];
#pragma unroll
        for (int k = 0; k < R0; ++k) v[k] = __ldcs(src + (j + M * k) * step);
        Dft<float2, R0>::run(v);
        twiddle0<N>(v, tab, j);
#pragma unroll
        for (int k = 0; k < R0; ++k) xs[at(k * M + j, c)] = v[k];
      }
    }
    __syncthreads();
    if constexpr (R1 > 1) middle_stage16<N>(xs, tab, at);
    if (live)
      for (int u = tid / kLines; u < R0 * R1; u += NT / kLines) {
        const int p0 = ((u % R0) * R1 + u / R0) * R2;
        float2 v[R2];
#pragma unroll
        for (int k = 0; k < R2; ++k) v[k] = xs[at(p0 + k, c)];
        Dft<float2, R2>::run(v);
#pragma unroll
        for (int k = 0; k < R2; ++k)
          if (kept_output(k, R2)) xs[at(p0 + k, c)] = v[k];
      }
    __syncthreads();
    const int sa = w.sp_a[g], sb = w.sp_b[g];
    for (int e = tid; e < T * (2 * h2 + 1); e += NT) {
      const int cc = e % T, i = e / T, im = 2 * h2 - i;
      const int x = x0 + cc, xm = 2 * h0 - x, f = i - h2;
      if (x >= K0) continue;
      const int lz = i - z0, lm = im - z0;
      const bool doP = x < xp && i < m2 && lz >= 0 && lz < nz;
      const bool doM = x < xq && xm < m0 && im < m2 && lm >= 0 && lm < nz;
      auto pos = [](int q) { return ((q % R0) * R1 + (q / R0) % R1) * R2 + q / (R0 * R1); };
      // G(k) and G(-k), times the deconvolution factor (even in every axis) and the window norm
      const float cr = c0[x < m0 ? x : xm] * c1[iy] * c2[i < m2 ? i : im] * w.wnorm_f;
      float2 A = xs[at(pos(f < 0 ? f + N : f), cc)];
      float2 B = pair || mrow ? xs[at(pos(f > 0 ? N - f : -f), T + cc)] : make_float2(0.f, 0.f);
      A = make_float2(A.x * cr, A.y * cr);
      B = make_float2(B.x * cr, B.y * cr);
      if (pair) {   // the species: A = (G(k) + G(-k)*) / 2, B = (G(k) - G(-k)*) / 2i; conjugates at -k
        const float2 u = make_float2(0.5f * (A.x + B.x), 0.5f * (A.y - B.y));
        B = make_float2(0.5f * (A.y + B.y), -0.5f * (A.x - B.x));
        A = u;
      }
      const int64_t qp = ((int64_t)lz * m1 + iy) * m0 + x, qm = ((int64_t)lm * m1 + iym) * m0 + xm;
      const float s2 = q_square(w, x - h0, iy - h1, f);
      float wa = species_weight<float>(w, sa, s2), wb = pair ? species_weight<float>(w, sb, s2) : 0.f;
      if (doP) {
        float2 u = make_float2(wa * A.x + wb * B.x, wa * A.y + wb * B.y);
        if (g > 0) {                                       // the earlier groups' sum, by this thread
          const float2 o = cs[qp];
          u = make_float2(u.x + o.x, u.y + o.y);
        }
        cs[qp] = u;
      }
      if (doM) {
        if (!w.even) {
          const float t2 = q_square(w, h0 - x, h1 - iy, -f);
          wa = species_weight<float>(w, sa, t2);
          wb = pair ? species_weight<float>(w, sb, t2) : 0.f;
        }
        float2 u = pair ? make_float2(wa * A.x + wb * B.x, -(wa * A.y + wb * B.y)) : make_float2(wa * B.x, wa * B.y);
        if (g > 0) {
          const float2 o = cs[qm];
          u = make_float2(u.x + o.x, u.y + o.y);
        }
        cs[qm] = u;
      }
      if (w.store_species) {
        float2* const sp = cs_species_frame + (int64_t)blockIdx.z * (nm * w.n_species);
        if (doP) sp[(int64_t)sa * nm + qp] = A;
        if (doP && pair) sp[(int64_t)sb * nm + qp] = B;
        if (doM) sp[(int64_t)sa * nm + qm] = pair ? make_float2(A.x, -A.y) : B;
        if (doM && pair) sp[(int64_t)sb * nm + qm] = make_float2(B.x, -B.y);
      }
    }
  }
  if (ngroups == 0)                                        // every species masked
    for (int e = tid; e < T * (2 * h2 + 1); e += NT) {
      const int i = e / T, im = 2 * h2 - i, x = x0 + e % T, xm = 2 * h0 - x, lz = i - z0, lm = im - z0;
      if (x >= K0) continue;
      if (x < xp && i < m2 && lz >= 0 && lz < nz) cs[((int64_t)lz * m1 + iy) * m0 + x] = make_float2(0.f, 0.f);
      if (x < xq && xm < m0 && im < m2 && lm >= 0 && lm < nz)
        cs[((int64_t)lm * m1 + iym) * m0 + xm] = make_float2(0.f, 0.f);
    }
}

// Long rows take half as many per CTA: at 1152 eight rows hold 80 KB and leave two CTAs per SM.
constexpr int x_rows(int n, int rows) { return n > 640 ? rows / 2 : rows; }
template <int N, int L>
int launch_x(const PruneLaunch& p) {
  // (grids follow one another: their rows are one list)
  const int64_t rows = (int64_t)p.ngrid * p.n[1] * p.fnz;
  if (p.n_fine != (int64_t)p.n[1] * p.fnz * N) return fail(MPSQ_ERR_ARG, "pass X: grids are not contiguous");
  if (const int rc = allow_smem(fftx_kernel<N, L>, x_smem<N, L>())) return rc;
  fftx_kernel<N, L><<<(unsigned)((rows + L - 1) / L), x_threads<N, L>(), x_smem<N, L>(), p.s>>>(
      p.fine, rows, p.tw[0], p.h[0], p.K[0], p.b1);
  MPSQ_LAUNCH_CHECK();
  return MPSQ_OK;
}
template <int N>
int launch_y(const PruneLaunch& p) {
  const size_t sm = (size_t)N * kLines * sizeof(float2);
  if (const int rc = allow_smem(ffty_kernel<N>, sm)) return rc;
  ffty_kernel<N><<<dim3((unsigned)((p.K[0] + kLines - 1) / kLines), (unsigned)p.fnz, (unsigned)p.ngrid),
                   yz_threads<N>(), sm, p.s>>>(p.b1, p.fnz, p.n[2], p.fz0, p.K[0], p.tw[1], p.h[1], p.K[1],
                                               p.b2);
  MPSQ_LAUNCH_CHECK();
  return MPSQ_OK;
}
template <int N>
int launch_z(const PruneLaunch& p, const WeightArgs& w, float2* csf, float2* css) {
  const size_t sm = (size_t)N * kLines * sizeof(float2);
  if (const int rc = allow_smem(fftz_deconv_kernel<N>, sm)) return rc;
  const int rows = std::min(p.m[1], p.h[1] + 1);   // ky rows iy <= h1; each also forms 2 h1 - iy
  // x tiles cover the K0 = 2 h0 + 1 kept columns: column 2 h0 is the mirror of mode column 0
  const int T = kLines / 2;
  fftz_deconv_kernel<N><<<dim3((unsigned)((p.K[0] + T - 1) / T), (unsigned)rows, (unsigned)p.frames),
                          yz_threads<N>(), sm, p.s>>>(
      p.b2, p.K[0], p.K[1], p.m[0], p.m[1], p.m[2], p.z0, p.nz, p.h[0], p.h[1], p.h[2], p.ngroups, p.tw[2],
      p.c[0], p.c[1], p.c[2], w, csf, css);
  MPSQ_LAUNCH_CHECK();
  return MPSQ_OK;
}

}  // namespace

bool fft_size_compiled(int n) {
  switch (n) {
#define MPSQ_CASE(N) case N:
    MPSQ_FFT_SIZES(MPSQ_CASE)
#undef MPSQ_CASE
    return true;
    default:
      return false;
  }
}
bool fft_plane_size_compiled(int n) {
  switch (n) {
#define MPSQ_CASE(N) case N:
    MPSQ_FFT_PLANE_SIZES(MPSQ_CASE)
#undef MPSQ_CASE
    return true;
    default:
      return false;
  }
}
int64_t compiled_fft_size_at_least(int64_t n) {
  int64_t best = 0;
#define MPSQ_MIN(N) if (N >= n && (best == 0 || N < best)) best = N;
  MPSQ_FFT_SIZES(MPSQ_MIN)
#undef MPSQ_MIN
  return best;
}

namespace {
// Gain of an FP32 rotation: the part along the exact one, exp(-2 pi i num / den), less 1.
double rotation_gain(int num, int den) {
  const double t = 2.0 * M_PI * (double)(num % den) / den, c = std::cos(t), s = std::sin(t);
  return c * ((double)(float)c - c) + s * ((double)(float)s - s);
}
// Gain of each output of a butterfly (dft.cuh): the mean of the above over the inputs, for its matrix with
// the constants of FP32.
std::vector<double> butterfly_gains(int r) {
  std::vector<double> g(r, 0.0);
  // Cooley-Tukey a x b (output k1 + a k2, twiddles between) and coprime factors (no twiddles)
  auto composite = [&](int a, int b, bool twiddles) {
    const std::vector<double> ga = butterfly_gains(a), gb = butterfly_gains(b);
    for (int k = 0; k < r; ++k) {
      g[k] = ga[k % a] + gb[twiddles ? k / a : k % b];
      for (int j = 0; j < b && twiddles; ++j) g[k] += rotation_gain(j * (k % a), r) / b;
    }
  };
  switch (r) {
    case 3: case 5:                        // every input but the first by a rotation, no output but the first
      for (int k = 1; k < r; ++k)
        for (int j = 1; j < r; ++j) {
          const double c = std::cos(2.0 * M_PI * j / r), s = std::sin(2.0 * M_PI * j / r);
          const double cf = r == 3 ? c : (double)(float)c;                       // (-1/2 is exact)
          g[k] += (c * (cf - c) + s * ((double)(float)s - s)) / r;
        }
      break;
    case 8:                                // odd outputs take the odd inputs times sqrt(1/2)
      for (int k = 1; k < 8; k += 2) g[k] = 0.5 * ((double)(float)std::sqrt(0.5) / std::sqrt(0.5) - 1.0);
      break;
    case 9: composite(3, 3, true); break;
    case 16: composite(4, 4, true); break;
    case 32: composite(8, 4, true); break;
    case 6: composite(2, 3, false); break;
    case 10: composite(2, 5, false); break;
    case 12: composite(4, 3, false); break;
    case 15: composite(3, 5, false); break;
    case 18: composite(2, 9, false); break;
    case 20: composite(4, 5, false); break;
    case 24: composite(8, 3, false); break;
    default: break;                        // 2 and 4 have no constants
  }
  return g;
}
}  // namespace

std::vector<float2> pass_twiddles(int n, std::vector<double>* gains) {
  const Split s = split_of(n);
  const int m = n / s.r0;
  std::vector<float2> t;
  std::vector<double> rows;                // mean gain of each row of twiddles
  auto add = [&](int row, int count, int den) {
    double sum = 0.0;
    for (int j = 0; j < count; ++j) {
      const double a = -2.0 * M_PI * (double)(j * row % den) / (double)den, c = std::cos(a), d = std::sin(a);
      t.push_back(make_float2((float)c, (float)d));
      sum += c * ((double)t.back().x - c) + d * ((double)t.back().y - d);
    }
    rows.push_back(sum / count);
  };
  for (int k = 0; k < s.r0; ++k) add(k, m, n);
  if (s.r1 > 1)
    for (int k = 0; k < s.r1; ++k) add(k, s.r2, s.r1 * s.r2);
  if (gains) {
    const std::vector<double> g0 = butterfly_gains(s.r0), g1 = butterfly_gains(s.r1), g2 = butterfly_gains(s.r2);
    auto gain = [&](int f) {               // f = k0 + r0 (k1 + r1 k2)
      const int k0 = f % s.r0, k1 = f / s.r0 % s.r1, k2 = f / (s.r0 * s.r1);
      return g0[k0] + rows[k0] + g2[k2] + (s.r1 > 1 ? g1[k1] + rows[s.r0 + k1] : 0.0);
    };
    gains->resize(n / 4 + 1);
    for (int f = 0; f <= n / 4; ++f) (*gains)[f] = 1.0 + 0.5 * (gain(f) + gain((n - f) % n));
  }
  return t;
}

int run_pruned_x(const PruneLaunch& p) {
  switch (p.n[0]) {
#define MPSQ_CASE(N) case N: return p.xrows == 4 ? launch_x<N, x_rows(N, 4)>(p) : launch_x<N, x_rows(N, 8)>(p);
    MPSQ_FFT_SIZES(MPSQ_CASE)
    MPSQ_FFT_PLANE_SIZES(MPSQ_CASE)
#undef MPSQ_CASE
  }
  return fail(MPSQ_ERR_ARG, "pass X: length %d is not compiled", p.n[0]);
}
int run_pruned_xy(const PruneLaunch& p) {
  const int rc = run_pruned_x(p);
  if (rc) return rc;
  switch (p.n[1]) {
#define MPSQ_CASE(N) case N: return launch_y<N>(p);
    MPSQ_FFT_SIZES(MPSQ_CASE)
#undef MPSQ_CASE
  }
  return fail(MPSQ_ERR_ARG, "pass Y: length %d is not compiled", p.n[1]);
}
int run_pruned_z(const PruneLaunch& p, const WeightArgs& w, float2* csf, float2* css) {
  switch (p.n[2]) {
#define MPSQ_CASE(N) case N: return launch_z<N>(p, w, csf, css);
    MPSQ_FFT_SIZES(MPSQ_CASE)
    MPSQ_FFT_PLANE_SIZES(MPSQ_CASE)
#undef MPSQ_CASE
  }
  return fail(MPSQ_ERR_ARG, "pass Z: length %d is not compiled", p.n[2]);
}

}  // namespace mpsq
