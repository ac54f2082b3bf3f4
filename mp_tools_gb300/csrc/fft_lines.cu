// Line transforms of the fine grids, FP64 and FP32, pruned to the kept frequencies.
//
// GB300 runs 2 FP64 lanes per clock and SM, so the number of FP64 instructions is the time of an FP64
// transform.  A line of length N = 2^a 3^b 5^c is transformed in shared memory by two or three large
// radices: composite butterflies of coprime factors carry no twiddles inside (Good-Thomas), the
// others few, so 320 = 16 x 20 takes 25 FP64 instructions per point (3.0 N log2 N; cuFFT's Z2Z time
// of 6.36 ms for 307,200 rows of 320 is that of 4.9 N log2 N).  The three axes run one after the
// other, each keeping only the 2h + 1 frequencies of [-h, h] that the modes and their mirrors read,
// so the second and third pass work on about 1/2 and 1/4 of the grid.  Radices are chosen at run time
// (index arithmetic is free next to the FP64 pipe), so every 2,3,5-smooth length is covered by one
// kernel.  Three 320^3 grids: cuFFT 13.0 ms, these passes 6.8 ms with the FP64 pipe 82 % busy.
//
// FP32 plans of larger volumes take float passes of the same plans: DRAM is the bound there, and of the 6
// times the grid that three full passes move the kept ones move 2.6 (two grids of 256 x 240 x 240:
// cuFFT 324 us and 29 us of deconvolution, these passes 160 us and 17 us).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "dft.cuh"
#include "mpsq_internal.h"

namespace mpsq {
namespace {

// FP64 instructions of each compiled radix (an FMA counts one).
constexpr struct { int r, cost; } kRadix[] = {{2, 4}, {3, 12}, {4, 16}, {5, 36}, {6, 36}, {8, 52}, {9, 88}, {10, 92},
                                              {12, 96}, {15, 168}, {16, 160}, {18, 212}, {20, 224}, {24, 252}};

// One stage of the in-place decimation-in-frequency transform of L = 2^lg lines (line l at xs + l
// (N + 1): the odd pitch puts a quarter-warp's eight 16-byte accesses of one position on eight
// different bank groups): groups {base + M k} by a radix-R DFT, output k' times
// exp(-2 pi i j k' / B), B = M R, j = base mod M.
//
// LAST (M = 1): output k of group g is frequency g + (N / R) k of which only [-N/4, N/4] is read, so
// the others are not stored and what only they need is not computed.
template <int R, bool LAST>
__device__ __forceinline__ void stage(double2* __restrict__ xs, const double2* __restrict__ tw, int lg, int N, int B) {
  const int M = B / R, step = N / B;
  for (int e = threadIdx.x; e < (N / R) << lg; e += blockDim.x) {
    const int ln = e & ((1 << lg) - 1), g = e >> lg;
    const int q = g / M, j = g - q * M;
    double2* const p = xs + ln * (N + 1) + q * B + j;
    double2 v[R];
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = p[k * M];
    Dft<double2, R>::run(v);
    if constexpr (LAST) {
#pragma unroll
      for (int k = 0; k < R; ++k)
        if (4 * k <= R || 4 * k > 3 * R - 4) p[k] = v[k];
    } else {
#pragma unroll
      for (int k = 1; k < R; ++k) {
        const double2 w = tw[step * j * k];
        v[k] = make_double2(fma(v[k].x, w.x, -v[k].y * w.y), fma(v[k].x, w.y, v[k].y * w.x));
      }
#pragma unroll
      for (int k = 0; k < R; ++k) p[k * M] = v[k];
    }
  }
}

template <bool LAST>
__device__ __forceinline__ void any_stage(int radix, double2* xs, const double2* tw, int lg, int N, int B) {
  switch (radix) {
    case 2: stage<2, LAST>(xs, tw, lg, N, B); break;
    case 3: stage<3, LAST>(xs, tw, lg, N, B); break;
    case 4: stage<4, LAST>(xs, tw, lg, N, B); break;
    case 5: stage<5, LAST>(xs, tw, lg, N, B); break;
    case 6: stage<6, LAST>(xs, tw, lg, N, B); break;
    case 8: stage<8, LAST>(xs, tw, lg, N, B); break;
    case 9: stage<9, LAST>(xs, tw, lg, N, B); break;
    case 10: stage<10, LAST>(xs, tw, lg, N, B); break;
    case 12: stage<12, LAST>(xs, tw, lg, N, B); break;
    case 15: stage<15, LAST>(xs, tw, lg, N, B); break;
    case 16: stage<16, LAST>(xs, tw, lg, N, B); break;
    case 18: stage<18, LAST>(xs, tw, lg, N, B); break;
    case 20: stage<20, LAST>(xs, tw, lg, N, B); break;
    default: stage<24, LAST>(xs, tw, lg, N, B); break;
  }
}

// One axis of a set of grids: line l of outer block o (blockIdx.y) of grid g (from blockIdx.z) starts at in
// + g in_grid + o in_outer + l in_line and its elements are in_elem apart; its kept frequency i (f =
// i - h) goes to out + g out_grid + o out_outer + l out_line + i out_elem.  One CTA takes 2^lg
// lines; contiguous ones (in_elem 1) go warp by warp.  swap: real and imaginary parts exchanged on
// reading (with the same exchange of the results this turns the forward transform into the backward one).
template <bool CONTIG, bool REAL>
__global__ void __launch_bounds__(128, 3)
    lines_f64_kernel(LinePass p, int lg) {
  constexpr int NT = 128, NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = 1 << lg, N = p.plan.n;
  double2* const xs = reinterpret_cast<double2*>(smem_raw);
  double2* const tw = xs + L * (N + 1);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t l0 = (int64_t)blockIdx.x * L;
  const int lines = (int)min((int64_t)L, p.n_lines - l0);
  const int64_t grid = (blockIdx.z / p.per) * p.skip + blockIdx.z % p.per + p.first;
  const double2* const src =
      static_cast<const double2*>(p.in) + grid * p.in_grid + blockIdx.y * p.in_outer + l0 * (REAL ? 2 : 1) * p.in_line;
  for (int i = tid; i < N; i += NT) tw[i] = static_cast<const double2*>(p.plan.tw)[i];
  auto put = [&](int at, double2 v) { xs[at] = p.swap ? make_double2(v.y, v.x) : v; };
  if constexpr (CONTIG) {
    for (int ln = warp; ln < L; ln += NW) {
      const double2* const row = src + (REAL ? 2 : 1) * ln * p.in_line;
#pragma unroll 4
      for (int x = lane; x < N; x += 32) {
        double2 v = make_double2(0.0, 0.0);
        if constexpr (REAL) {
          if (ln < lines) v = make_double2(__ldcs(row + x).x, __ldcs(row + p.in_line + x).x);
        } else {
          if (ln < lines) v = __ldcs(row + x);
        }
        put(ln * (N + 1) + x, v);
      }
    }
  } else {
#pragma unroll 8
    for (int e = tid; e < N << lg; e += NT) {
      const int ln = e & (L - 1), x = e >> lg;
      put(ln * (N + 1) + x, ln < lines ? __ldcs(src + ln * p.in_line + x * p.in_elem) : make_double2(0.0, 0.0));
    }
  }
  __syncthreads();
  int B = N;
  for (int s = 0; s + 1 < p.plan.stages; ++s) {
    any_stage<false>(p.plan.radix[s], xs, tw, lg, N, B);
    B /= p.plan.radix[s];
    __syncthreads();
  }
  any_stage<true>(B, xs, tw, lg, N, B);
  __syncthreads();
  if constexpr (REAL) {                      // rows 2 l, 2 l + 1 from Z = A + i B: A(f) = (Z(f) + Z(-f)*) / 2
    double2* const dst = static_cast<double2*>(p.out) + grid * p.out_grid + 2 * l0 * p.out_line;
    for (int ln = warp; ln < lines; ln += NW)
      for (int f = lane; f <= p.h; f += 32) {
        const double2 u = xs[ln * (N + 1) + p.plan.pos[f]], v = xs[ln * (N + 1) + p.plan.pos[f ? N - f : 0]];
        dst[2 * ln * p.out_line + f] = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
        dst[(2 * ln + 1) * p.out_line + f] = make_double2(0.5 * (u.y + v.y), 0.5 * (v.x - u.x));
      }
  } else {
    double2* const dst = static_cast<double2*>(p.out) + grid * p.out_grid + blockIdx.y * p.out_outer + l0 * p.out_line;
    const int K = 2 * p.h + 1;
    auto at = [&](int i) { return p.plan.pos[i < p.h ? i - p.h + N : i - p.h]; };
    if constexpr (CONTIG) {
      for (int ln = warp; ln < lines; ln += NW)
        for (int i = lane; i < K; i += 32) dst[ln * p.out_line + (int64_t)i * p.out_elem] = xs[ln * (N + 1) + at(i)];
    } else {
      for (int e = tid; e < K << lg; e += NT) {
        const int ln = e & (L - 1), i = e >> lg;
        if (ln < lines) dst[ln * p.out_line + (int64_t)i * p.out_elem] = xs[ln * (N + 1) + at(i)];
      }
    }
  }
}

// The same for float2: DRAM and latency are the bound there, so the first butterfly reads its elements
// straight from the grid and the last one writes its kept frequencies, and only the exchange between
// the stages goes through shared memory (padded by one element in 16 so that neither the lines nor
// the groups of a line meet in a bank).
__device__ __forceinline__ int at32(int p) { return p + (p >> 4); }
int pitch32(int n) { return (n + n / 16 + 1) | 1; }

template <int R, bool CONTIG>
__device__ __forceinline__ void first32(const LinePass& p, const float2* __restrict__ src, float2* __restrict__ xs,
                                        const float2* __restrict__ tw, int lg, int lines, int pitch) {
  const int N = p.plan.n, M = N / R;
  for (int e = threadIdx.x; e < M << lg; e += blockDim.x) {
    const int ln = CONTIG ? e / M : e & ((1 << lg) - 1), j = CONTIG ? e - ln * M : e >> lg;
    const float2* const q = src + ln * p.in_line + j * p.in_elem;
    float2 v[R];
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = ln < lines ? __ldcs(q + k * M * p.in_elem) : make_float2(0.f, 0.f);
    if (p.swap) {
#pragma unroll
      for (int k = 0; k < R; ++k) v[k] = make_float2(v[k].y, v[k].x);
    }
    Dft<float2, R>::run(v);
    float2* const x = xs + ln * pitch;
    x[at32(j)] = v[0];
#pragma unroll
    for (int k = 1; k < R; ++k) {
      const float2 w = tw[j * k];
      x[at32(j + M * k)] = make_float2(v[k].x * w.x - v[k].y * w.y, v[k].x * w.y + v[k].y * w.x);
    }
  }
}

template <int R>
__device__ __forceinline__ void middle32(float2* __restrict__ xs, const float2* __restrict__ tw, int lg, int N, int B,
                                         int pitch) {
  const int M = B / R, step = N / B;
  for (int e = threadIdx.x; e < (N / R) << lg; e += blockDim.x) {
    const int ln = e & ((1 << lg) - 1), g = e >> lg;
    const int q = g / M, j = g - q * M;
    float2* const x = xs + ln * pitch;
    float2 v[R];
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = x[at32(q * B + j + k * M)];
    Dft<float2, R>::run(v);
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const float2 w = tw[step * j * k];
      x[at32(q * B + j + k * M)] = make_float2(v[k].x * w.x - v[k].y * w.y, v[k].x * w.y + v[k].y * w.x);
    }
  }
}

template <int R, bool CONTIG>
__device__ __forceinline__ void last32(const LinePass& p, float2* __restrict__ dst, const float2* __restrict__ xs,
                                       int lg, int lines, int pitch) {
  const int N = p.plan.n, G = N / R;
  for (int e = threadIdx.x; e < G << lg; e += blockDim.x) {
    const int ln = CONTIG ? e / G : e & ((1 << lg) - 1), g = CONTIG ? e - ln * G : e >> lg;
    if (ln >= lines) continue;
    const int q = p.plan.pos[g];           // where the group of frequencies g + G k starts
    float2 v[R];
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = xs[ln * pitch + at32(q + k)];
    Dft<float2, R>::run(v);
    float2* const o = dst + ln * p.out_line;
#pragma unroll
    for (int k = 0; k < R; ++k) {
      if (4 * k > R && 4 * k <= 3 * R - 4) continue;           // h < N / 4
      const int f = g + G * k, i = f <= p.h ? f + p.h : f - N + p.h;
      if (i >= 0) o[i * p.out_elem] = v[k];
    }
  }
}

template <bool CONTIG>
__global__ void __launch_bounds__(256, 3)
    lines_f32_kernel(LinePass p, int lg, int pitch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = 1 << lg, N = p.plan.n;
  float2* const xs = reinterpret_cast<float2*>(smem_raw);
  float2* const tw = xs + L * pitch;
  const int64_t l0 = (int64_t)blockIdx.x * L;
  const int lines = (int)min((int64_t)L, p.n_lines - l0);
  const int64_t grid = (blockIdx.z / p.per) * p.skip + blockIdx.z % p.per + p.first;
  const float2* const src =
      static_cast<const float2*>(p.in) + grid * p.in_grid + blockIdx.y * p.in_outer + l0 * p.in_line;
  float2* const dst = static_cast<float2*>(p.out) + grid * p.out_grid + blockIdx.y * p.out_outer + l0 * p.out_line;
  for (int i = threadIdx.x; i < N; i += 256) tw[i] = static_cast<const float2*>(p.plan.tw)[i];
  __syncthreads();
#define MPSQ_RADIX32(X) \
  X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10) X(12) X(15) X(16)
  switch (p.plan.radix[0]) {
#define MPSQ_STAGE(R) case R: first32<R, CONTIG>(p, src, xs, tw, lg, lines, pitch); break;
    MPSQ_RADIX32(MPSQ_STAGE)
#undef MPSQ_STAGE
  }
  int B = N / p.plan.radix[0];
  __syncthreads();
  for (int s = 1; s + 1 < p.plan.stages; ++s) {
    switch (p.plan.radix[s]) {
#define MPSQ_STAGE(R) case R: middle32<R>(xs, tw, lg, N, B, pitch); break;
      MPSQ_RADIX32(MPSQ_STAGE)
#undef MPSQ_STAGE
    }
    B /= p.plan.radix[s];
    __syncthreads();
  }
  switch (B) {
#define MPSQ_STAGE(R) case R: last32<R, CONTIG>(p, dst, xs, lg, lines, pitch); break;
    MPSQ_RADIX32(MPSQ_STAGE)
#undef MPSQ_STAGE
  }
#undef MPSQ_RADIX32
}

// (the size depends on the line's length)
size_t most_smem(size_t sm) { return sm > 48 * 1024 ? 227 * 1024 : sm; }

template <bool CONTIG, bool REAL>
int launch_f64(const LinePass& p, int lg, dim3 grid, size_t sm, cudaStream_t s) {
  if (const int rc = allow_smem(lines_f64_kernel<CONTIG, REAL>, most_smem(sm))) return rc;
  lines_f64_kernel<CONTIG, REAL><<<grid, 128, sm, s>>>(p, lg);
  MPSQ_LAUNCH_CHECK();
  return MPSQ_OK;
}
template <bool CONTIG>
int launch_f32(const LinePass& p, int lg, dim3 grid, size_t sm, cudaStream_t s) {
  if (const int rc = allow_smem(lines_f32_kernel<CONTIG>, most_smem(sm))) return rc;
  lines_f32_kernel<CONTIG><<<grid, 256, sm, s>>>(p, lg, pitch32(p.plan.n));
  MPSQ_LAUNCH_CHECK();
  return MPSQ_OK;
}

size_t line_smem(int n, int lines, int bytes) {
  return (size_t)bytes * ((size_t)lines * (bytes == 16 ? n + 1 : pitch32(n)) + n);
}

}  // namespace

bool line_radices(int64_t n, int bytes, LinePlan* plan, int max_radix) {
  if (n < 2 || line_smem((int)std::min<int64_t>(n, 1 << 20), 1, bytes) > 227 * 1024) return false;
  // cheapest factorisation: instructions per point of every stage and of the twiddles between them
  // (4 per point), each further stage also a pass over shared memory (counted 2 per point)
  std::vector<double> best(n + 1, 1e30);
  std::vector<int> first(n + 1, 0);
  best[1] = 0.0;
  for (int64_t m = 2; m <= n; ++m) {
    if (n % m) continue;
    for (const auto& k : kRadix) {
      if (m % k.r || k.r > max_radix || (bytes == 8 && k.r > 16)) continue;   // (80 registers in FP32)
      const double c = best[m / k.r] + (double)k.cost / k.r + (m > k.r ? 6.0 : 0.0);
      if (c < best[m]) {
        best[m] = c;
        first[m] = k.r;
      }
    }
  }
  if (best[n] > 1e29 || (bytes == 8 && first[n] == n)) return false;      // (FP32: two stages at least)
  LinePlan q;
  q.n = (int)n;
  for (int64_t m = n; m > 1; m /= first[m]) {
    if (q.stages == kLineStages) return false;
    q.radix[q.stages++] = first[m];
  }
  if (plan) *plan = q;
  return true;
}

void line_tables(const LinePlan& plan, std::vector<double2>* tw, std::vector<int>* pos) {
  tw->resize(plan.n);
  pos->resize(plan.n);
  for (int i = 0; i < plan.n; ++i) {
    // from the angle to the nearest axis, at most 1/8 turn, so that 0 and 1 come out exact
    const int n = plan.n, o = (int)((8LL * i) / n);
    double c = 0, s = 0;
    const double quarter = 0.25 * n;
    const double d = (double)i - quarter * ((o + 1) / 2);            // distance to the nearest axis
    const double ca = std::cos(2.0 * M_PI * d / n), sa = std::sin(2.0 * M_PI * d / n);
    switch (((o + 1) / 2) & 3) {
      case 0: c = ca; s = sa; break;
      case 1: c = -sa; s = ca; break;
      case 2: c = -ca; s = -sa; break;
      default: c = sa; s = -ca; break;
    }
    (*tw)[i] = make_double2(c, -s);
    int f = i, block = n, p = 0;
    for (int k = 0; k < plan.stages; ++k) {
      block /= plan.radix[k];
      p += (f % plan.radix[k]) * block;
      f /= plan.radix[k];
    }
    (*pos)[i] = p;
  }
}

int launch_lines(const LinePass& p, int outer, cudaStream_t s) {
  if (outer > 65535 || p.grids > 65535) return fail(MPSQ_ERR_ARG, "line transform: too many grids");
  // 128-byte segments across lines: eight per CTA in FP64, sixteen in FP32 (eight where sixteen
  // would leave fewer than three CTAs per SM), fewer where that leaves SMs without a CTA or they do not fit
  int lg = p.bytes == 16 ? 3 : 4;
  if (lg == 4 && line_smem(p.plan.n, 16, p.bytes) > 75 * 1024) lg = 3;
  while (lg > 0 && (line_smem(p.plan.n, 1 << lg, p.bytes) > 227 * 1024 ||
                    ((p.n_lines + (1 << lg) - 1) >> lg) * outer * p.grids < 2 * 152))
    --lg;
  const size_t sm = line_smem(p.plan.n, 1 << lg, p.bytes);
  const dim3 grid((unsigned)((p.n_lines + (1 << lg) - 1) >> lg), (unsigned)outer, (unsigned)p.grids);
  const bool contig = p.in_elem == 1;
  if (p.bytes == 8) return contig ? launch_f32<true>(p, lg, grid, sm, s) : launch_f32<false>(p, lg, grid, sm, s);
  if (p.real) return launch_f64<true, true>(p, lg, grid, sm, s);
  return contig ? launch_f64<true, false>(p, lg, grid, sm, s) : launch_f64<false, false>(p, lg, grid, sm, s);
}

bool grid_lines_ok(const GridGeom& g, int precision) {
  const int bytes = precision == MPSQ_FP64 ? 16 : 8;
  for (int k = 0; k < g.dim; ++k)
    if (!line_radices(g.nf[k], bytes, nullptr)) return false;
  return true;
}

void grid_lines_plan(const GridGeom& g, int precision, int64_t ngrid, GridLines* gl, std::vector<char>* tables) {
  GridLines r;
  r.dim = g.dim;
  r.bytes = precision == MPSQ_FP64 ? 16 : 8;
  tables->clear();
  for (int k = 0; k < g.dim; ++k) {
    // An SM's four schedulers each hold a quarter of its FP64 lanes, so a line or two per SM in
    // radix-16 and -20 butterflies (20 threads) run on one of them: below 16 lines per SM the
    // radices stay at 5 (one 320^2 grid, per pass: 26 -> 15 us).
    const bool few = r.bytes == 16 && ngrid * (g.n_fine / g.nf[k]) < 16 * 152;
    if (!few || !line_radices(g.nf[k], r.bytes, &r.plan[k], 5)) line_radices(g.nf[k], r.bytes, &r.plan[k]);
    r.n[k] = g.nf[k];
    r.h[k] = (int)(g.m[k] / 2);
    r.K[k] = 2 * r.h[k] + 1;
    std::vector<double2> tw;
    std::vector<int> pos;
    line_tables(r.plan[k], &tw, &pos);
    std::vector<float2> twf(tw.size());
    for (size_t i = 0; i < tw.size(); ++i) twf[i] = make_float2((float)tw[i].x, (float)tw[i].y);
    const char* a = r.bytes == 16 ? reinterpret_cast<const char*>(tw.data()) : reinterpret_cast<const char*>(twf.data());
    const char* b = reinterpret_cast<const char*>(pos.data());
    tables->insert(tables->end(), a, a + tw.size() * r.bytes);
    tables->insert(tables->end(), b, b + pos.size() * sizeof(int));
    tables->resize((tables->size() + 255) & ~size_t(255));
  }
  *gl = r;
}

void grid_lines_bind(GridLines* gl, const void* tables) {
  const char* p = static_cast<const char*>(tables);
  size_t off = 0;
  for (int k = 0; k < gl->dim; ++k) {
    const int64_t n = gl->n[k];
    gl->plan[k].tw = p + off;
    gl->plan[k].pos = reinterpret_cast<const int*>(p + off + n * gl->bytes);
    off = (off + n * (gl->bytes + sizeof(int)) + 255) & ~size_t(255);
  }
}

int run_grid_lines(const GridLines& gl, int ngrid, int group, bool last_real, void* fine, void* tmp, bool swap,
                   cudaStream_t s) {
  const int64_t n0 = gl.n[0], n1 = gl.n[1], n2 = gl.n[2], n_fine = gl.n_fine();
  const bool turns = gl.at_once(ngrid) < ngrid;      // one grid at a time through tmp
  // the three passes over grids z -> (z / per) skip + z % per + first, z < count
  auto passes = [&](int count, int per, int skip, int first, bool real) -> int {
    const int64_t K0 = real ? gl.h[0] + 1 : gl.K[0], K1 = gl.K[1], K2 = gl.K[2];
    const int64_t tmp_grid = turns ? 0 : gl.tmp_grid();
    LinePass x{};
    x.bytes = gl.bytes;
    x.plan = gl.plan[0];
    x.in = fine;
    x.out = tmp;
    x.n_lines = n2 * n1 / (real ? 2 : 1);
    x.in_line = n0;
    x.in_elem = 1;
    x.in_grid = n_fine;
    x.out_line = K0;
    x.out_elem = 1;
    x.out_grid = tmp_grid;
    x.grids = count;
    x.per = per;
    x.skip = skip;
    x.first = first;
    x.h = gl.h[0];
    x.swap = swap ? 1 : 0;
    x.real = real ? 1 : 0;
    int rc = launch_lines(x, 1, s);
    if (rc) return rc;
    LinePass y = x;
    y.plan = gl.plan[1];
    y.in = tmp;
    y.out = fine;
    y.n_lines = K0;
    y.in_line = y.out_line = 1;
    y.in_elem = y.out_elem = K0;
    y.in_outer = n1 * K0;
    y.in_grid = tmp_grid;
    y.out_outer = K1 * K0;
    y.out_grid = n_fine;
    y.h = gl.h[1];
    y.swap = y.real = 0;
    rc = launch_lines(y, (int)n2, s);
    if (rc || gl.dim == 2) return rc;
    LinePass z = y;
    z.plan = gl.plan[2];
    z.in = fine;
    z.out = static_cast<char*>(fine) + gl.kept() * gl.bytes;
    z.n_lines = K1 * K0;
    z.in_elem = z.out_elem = K1 * K0;
    z.in_outer = z.out_outer = 0;
    z.in_grid = n_fine;
    z.h = gl.h[2];
    return launch_lines(z, 1, s);
  };
  const int full = last_real ? group - 1 : group;    // complex grids per group
  if (turns) {
    for (int g = 0; g < ngrid; ++g) {
      const int rc = passes(1, 1, 0, g, g % group >= full);
      if (rc) return rc;
    }
    return MPSQ_OK;
  }
  const int groups = ngrid / group;
  int rc = MPSQ_OK;
  if (full > 0) rc = passes(groups * full, full, group, 0, false);
  if (!rc && last_real) rc = passes(groups, 1, group, group - 1, true);
  return rc;
}

}  // namespace mpsq
