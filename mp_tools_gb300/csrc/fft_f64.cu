// FP64 line transforms of the fine grids, pruned to the kept frequencies.
//
// GB300 runs 2 FP64 lanes per clock and SM, so the number of FP64 instructions is the time of an FP64
// transform.  A line of length N = 2^a 3^b 5^c is transformed in shared memory by two or three large
// radices: composite butterflies of coprime factors carry no twiddles inside (Good-Thomas), the
// others few, so 320 = 16 x 20 takes 25 FP64 instructions per point (3.0 N log2 N; cuFFT's Z2Z time
// of 6.36 ms for 307,200 rows of 320 is that of 4.9 N log2 N).  The three axes run one after the
// other, each keeping only the 2h + 1 frequencies of [-h, h] that the modes and their mirrors read,
// so the second and third pass work on about 1/2 and 1/4 of the grid.  Radices are chosen at run time
// (index arithmetic is free next to the FP64 pipe), so every 2,3,5-smooth length is covered by one
// kernel.
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

// One stage of the in-place decimation-in-frequency transform of L = 2^LG lines (line l at xs + l
// (N + 1): the odd pitch puts a quarter-warp's eight 16-byte accesses of one position on eight
// different bank groups): groups {base + M k} by a radix-R DFT, output k' times
// exp(-2 pi i j k' / B), B = M R, j = base mod M.
//
// LAST (M = 1): output k of group g is frequency g + (N / R) k of which only [-N/4, N/4] is read, so
// the others are not stored and what only they need is not computed.
template <int R, int LG, bool LAST>
__device__ __forceinline__ void stage(double2* __restrict__ xs, const double2* __restrict__ tw, int N,
                                      int B) {
  const int M = B / R, step = N / B;
  for (int e = threadIdx.x; e < (N / R) << LG; e += blockDim.x) {
    const int ln = e & ((1 << LG) - 1), g = e >> LG;
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

template <int LG, bool LAST>
__device__ __forceinline__ void any_stage(int radix, double2* xs, const double2* tw, int N, int B) {
  switch (radix) {
    case 2: stage<2, LG, LAST>(xs, tw, N, B); break;
    case 3: stage<3, LG, LAST>(xs, tw, N, B); break;
    case 4: stage<4, LG, LAST>(xs, tw, N, B); break;
    case 5: stage<5, LG, LAST>(xs, tw, N, B); break;
    case 6: stage<6, LG, LAST>(xs, tw, N, B); break;
    case 8: stage<8, LG, LAST>(xs, tw, N, B); break;
    case 9: stage<9, LG, LAST>(xs, tw, N, B); break;
    case 10: stage<10, LG, LAST>(xs, tw, N, B); break;
    case 12: stage<12, LG, LAST>(xs, tw, N, B); break;
    case 15: stage<15, LG, LAST>(xs, tw, N, B); break;
    case 16: stage<16, LG, LAST>(xs, tw, N, B); break;
    case 18: stage<18, LG, LAST>(xs, tw, N, B); break;
    case 20: stage<20, LG, LAST>(xs, tw, N, B); break;
    default: stage<24, LG, LAST>(xs, tw, N, B); break;
  }
}

// One axis of a set of grids: line l of outer block o (blockIdx.y) of grid g (from blockIdx.z) starts at in
// + g in_grid + o in_outer + l in_line and its elements are in_elem apart; its kept frequency i (f =
// i - h) goes to out + g out_grid + o out_outer + l out_line + i out_elem.  One CTA takes 2^LG lines.  swap: real and imaginary parts exchanged on reading
// (with the same exchange of the results this turns the forward transform into the backward one).
template <int LG, bool CONTIG, bool REAL>
__global__ void __launch_bounds__(128, 3)
    lines_f64_kernel(LinePass p) {
  constexpr int L = 1 << LG;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = p.plan.n;
  double2* const xs = reinterpret_cast<double2*>(smem_raw);
  double2* const tw = xs + L * (N + 1);
  const int tid = threadIdx.x;
  const int64_t l0 = (int64_t)blockIdx.x * L;
  const int lines = (int)min((int64_t)L, p.n_lines - l0);
  const int64_t grid = (blockIdx.z / p.per) * p.skip + blockIdx.z % p.per + p.first;
  const double2* const src = p.in + grid * p.in_grid + blockIdx.y * p.in_outer + l0 * (REAL ? 2 : 1) * p.in_line;
  for (int i = tid; i < N; i += 128) tw[i] = p.plan.tw[i];
#pragma unroll 4
  for (int e = tid; e < L * N; e += 128) {
    const int ln = CONTIG ? e / N : e & (L - 1), x = CONTIG ? e - ln * N : e >> LG;
    double2 v = make_double2(0.0, 0.0);
    if constexpr (REAL) {
      if (ln < lines) v = make_double2(__ldcs(src + 2 * ln * p.in_line + x).x, __ldcs(src + (2 * ln + 1) * p.in_line + x).x);
    } else {
      if (ln < lines) v = __ldcs(src + ln * p.in_line + x * p.in_elem);
    }
    xs[ln * (N + 1) + x] = p.swap ? make_double2(v.y, v.x) : v;
  }
  __syncthreads();
  int B = N;
  for (int s = 0; s + 1 < p.plan.stages; ++s) {
    any_stage<LG, false>(p.plan.radix[s], xs, tw, N, B);
    B /= p.plan.radix[s];
    __syncthreads();
  }
  any_stage<LG, true>(B, xs, tw, N, B);
  __syncthreads();
  if constexpr (REAL) {                      // rows 2 l, 2 l + 1 from Z = A + i B: A(f) = (Z(f) + Z(-f)*) / 2
    double2* const dst = p.out + grid * p.out_grid + 2 * l0 * p.out_line;
    const int K = p.h + 1;
    for (int e = tid; e < L * K; e += 128) {
      const int ln = e / K, f = e - ln * K;
      if (ln >= lines) continue;
      const double2 u = xs[ln * (N + 1) + p.plan.pos[f]], v = xs[ln * (N + 1) + p.plan.pos[f ? N - f : 0]];
      dst[2 * ln * p.out_line + f] = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
      dst[(2 * ln + 1) * p.out_line + f] = make_double2(0.5 * (u.y + v.y), 0.5 * (v.x - u.x));
    }
  } else {
    double2* const dst = p.out + grid * p.out_grid + blockIdx.y * p.out_outer + l0 * p.out_line;
    const int K = 2 * p.h + 1;
    for (int e = tid; e < L * K; e += 128) {
      const int ln = CONTIG ? e / K : e & (L - 1), i = CONTIG ? e - ln * K : e >> LG;
      const int f = i - p.h;
      if (ln < lines) dst[ln * p.out_line + (int64_t)i * p.out_elem] = xs[ln * (N + 1) + p.plan.pos[f < 0 ? f + N : f]];
    }
  }
}

template <int LG>
cudaError_t raise_smem() {
  constexpr int most = 227 * 1024;
  cudaError_t e = cudaFuncSetAttribute(lines_f64_kernel<LG, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(lines_f64_kernel<LG, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(lines_f64_kernel<LG, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  return e;
}

size_t line_smem(int n, int lines) { return sizeof(double2) * ((size_t)lines * (n + 1) + n); }

}  // namespace

bool line_radices(int64_t n, LinePlan* plan, int max_radix) {
  if (n < 2 || line_smem((int)std::min<int64_t>(n, 1 << 20), 1) > 227 * 1024) return false;
  // cheapest factorisation: instructions per point of every stage and of the twiddles between them
  // (4 per point), each further stage also a pass over shared memory (counted 2 per point)
  std::vector<double> best(n + 1, 1e30);
  std::vector<int> first(n + 1, 0);
  best[1] = 0.0;
  for (int64_t m = 2; m <= n; ++m) {
    if (n % m) continue;
    for (const auto& k : kRadix) {
      if (m % k.r || k.r > max_radix) continue;
      const double c = best[m / k.r] + (double)k.cost / k.r + (m > k.r ? 6.0 : 0.0);
      if (c < best[m]) {
        best[m] = c;
        first[m] = k.r;
      }
    }
  }
  if (best[n] > 1e29) return false;
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
  static const cudaError_t attr = [] {
    cudaError_t e = raise_smem<0>();
    if (e == cudaSuccess) e = raise_smem<1>();
    if (e == cudaSuccess) e = raise_smem<2>();
    if (e == cudaSuccess) e = raise_smem<3>();
    return e;
  }();
  if (attr != cudaSuccess) return fail(MPSQ_ERR_CUDA, "line transform attribute: %s", cudaGetErrorString(attr));
  // eight lines per CTA (128-byte segments across lines), fewer where that leaves SMs without a CTA
  // or where they do not fit
  int lg = 3;
  while (lg > 0 && (line_smem(p.plan.n, 1 << lg) > 227 * 1024 ||
                    ((p.n_lines + (1 << lg) - 1) >> lg) * outer * p.grids < 2 * 152))
    --lg;
  const size_t sm = line_smem(p.plan.n, 1 << lg);
  const dim3 grid((unsigned)((p.n_lines + (1 << lg) - 1) >> lg), (unsigned)outer, (unsigned)p.grids);
#define MPSQ_LINES(G)                                                     \
  if (p.real)                                                             \
    lines_f64_kernel<G, true, true><<<grid, 128, sm, s>>>(p);             \
  else if (p.in_elem == 1)                                                \
    lines_f64_kernel<G, true, false><<<grid, 128, sm, s>>>(p);            \
  else                                                                    \
    lines_f64_kernel<G, false, false><<<grid, 128, sm, s>>>(p)
  switch (lg) {
    case 0: MPSQ_LINES(0); break;
    case 1: MPSQ_LINES(1); break;
    case 2: MPSQ_LINES(2); break;
    default: MPSQ_LINES(3); break;
  }
#undef MPSQ_LINES
  MPSQ_LAUNCH_CHECK();
  return MPSQ_OK;
}

bool grid_lines_ok(const GridGeom& g) {
  for (int k = 0; k < g.dim; ++k)
    if (!line_radices(g.nf[k], nullptr)) return false;
  return true;
}

void grid_lines_plan(const GridGeom& g, int64_t ngrid, GridLines* gl, std::vector<char>* tables) {
  GridLines r;
  r.dim = g.dim;
  tables->clear();
  for (int k = 0; k < g.dim; ++k) {
    // An SM's four schedulers each hold a quarter of its FP64 lanes, so a line or two per SM in
    // radix-16 and -20 butterflies (20 threads) run on one of them: below 16 lines per SM the
    // radices stay at 5 (one 320^2 grid, per pass: 26 -> 15 us).
    const bool few = ngrid * (g.n_fine / g.nf[k]) < 16 * 152;
    if (!few || !line_radices(g.nf[k], &r.plan[k], 5)) line_radices(g.nf[k], &r.plan[k]);
    r.n[k] = g.nf[k];
    r.h[k] = (int)(g.m[k] / 2);
    r.K[k] = 2 * r.h[k] + 1;
    std::vector<double2> tw;
    std::vector<int> pos;
    line_tables(r.plan[k], &tw, &pos);
    const char* a = reinterpret_cast<const char*>(tw.data());
    const char* b = reinterpret_cast<const char*>(pos.data());
    tables->insert(tables->end(), a, a + tw.size() * sizeof(double2));
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
    gl->plan[k].tw = reinterpret_cast<const double2*>(p + off);
    gl->plan[k].pos = reinterpret_cast<const int*>(p + off + n * sizeof(double2));
    off = (off + n * (sizeof(double2) + sizeof(int)) + 255) & ~size_t(255);
  }
}

int run_grid_lines(const GridLines& gl, int ngrid, int group, bool last_real, double2* fine,
                   double2* tmp, bool swap, cudaStream_t s) {
  const int64_t n0 = gl.n[0], n1 = gl.n[1], n2 = gl.n[2], n_fine = gl.n_fine();
  const bool turns = gl.at_once(ngrid) < ngrid;      // one grid at a time through tmp
  // the three passes over grids z -> (z / per) skip + z % per + first, z < count
  auto passes = [&](int count, int per, int skip, int first, bool real) -> int {
    const int64_t K0 = real ? gl.h[0] + 1 : gl.K[0], K1 = gl.K[1], K2 = gl.K[2];
    const int64_t tmp_grid = turns ? 0 : gl.tmp_grid();
    LinePass x{};
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
    z.out = fine + gl.kept();
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
