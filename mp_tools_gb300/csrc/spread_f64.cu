// FP64 spreading (planes and volumes, any width, complex strengths or packed real pairs).
//
// GB300 issues two FP64 lanes per clock and SM (one warp instruction in 16 clocks), so FP64
// instructions are what a spread costs.  Two things hold them down:
//  * kernel values.  The ES kernel phi(z) = exp(beta (sqrt(1 - z^2) - 1)) is even, so the cells i
//    and w-1-i of a support are p(v) = E(v^2) + v O(v^2) and p(-v) of one polynomial in v = 2u - 1
//    (u the point's offset in its cell): 21 multiply-adds for two values at degree 20, good to
//    2e-16 of the kernel's peak (sqrt and exp: up to 3e-15) in every cell but the two at the support's
//    ends.  There phi has its square-root singularity and is taken from sqrt and exp.
//    The lanes of a warp share the values of 16 records, so that all of them work (one record per
//    warp kept 14 of 32 lanes busy with exp and sqrt at width 7 on a plane).
//  * sums.  No atomics (a shared-memory FP64 add is a compare-and-swap loop): on a plane every warp
//    adds into a copy of the tile of its own, one support row of a record per w lanes; in a volume
//    every warp owns two planes of the tile.
#include <cuda_runtime.h>

#include <mutex>

#include "es_pairs.h"
#include "mpsq_internal.h"

namespace mpsq {
namespace {

EsPairs pairs_for(int w, double beta) {
  static std::mutex mu;
  static EsPairs kept[17];
  static double kept_beta[17] = {};
  std::lock_guard<std::mutex> lock(mu);
  if (kept_beta[w] != beta) {
    kept[w] = make_pairs(w, beta);
    kept_beta[w] = beta;
  }
  return kept[w];
}

__device__ __forceinline__ double es_end(double d, int i, double two_over_w, double beta) {
  const double z = (d + (double)i) * two_over_w;
  return exp(beta * (sqrt(fmax(1.0 - z * z, 0.0)) - 1.0));
}

// The two cells of interior pair p from their point's offset d.
__device__ __forceinline__ void eval_pair(const EsPairs& tab, int p, int w, double d,
                                          double* __restrict__ row) {
  const double v = fma(2.0, d, (double)(w - 1)), v2 = v * v;
  double e = tab.e[p][kEven - 1], o = tab.o[p][kOdd - 1];
#pragma unroll
  for (int k = kEven - 2; k >= 0; --k) e = fma(e, v2, tab.e[p][k]);
#pragma unroll
  for (int k = kOdd - 2; k >= 0; --k) o = fma(o, v2, tab.o[p][k]);
  row[p + 1] = fma(v, o, e);
  row[w - 2 - p] = fma(-v, o, e);
}

constexpr int kR = 16;               // records a warp evaluates together
// doubles per record: DIM rows of 16 values, odd, so that a half-warp's stores hit all banks
template <int DIM>
constexpr int kRec = DIM * 16 + 1;

// Kernel values of up to kR records of a plane, lane l < kR holding record l's offsets: ker[r kRec
// + 16 axis + cell].  All lanes of the warp call it (past the last record they evaluate a fixed offset).
__device__ __forceinline__ void eval_records(const EsPairs& tab, int w, double beta, double d0,
                                             double d1, double* __restrict__ ker) {
  constexpr int DIM = 2;
  const int lane = threadIdx.x & 31, r = lane & (kR - 1), half = lane >> 4;
  const double two_over_w = 2.0 / w;
  const double dx = __shfl_sync(0xffffffffu, d0, r), dy = __shfl_sync(0xffffffffu, d1, r);
#pragma unroll 1
  for (int ax = 0; ax < DIM; ++ax) {            // the two end cells, one per half-warp
    const double d = ax == 0 ? dx : dy;
    const int i = half ? w - 1 : 0;
    ker[r * kRec<DIM> + ax * 16 + i] = es_end(d, i, two_over_w, beta);
  }
  const int np = (w + 1) / 2 - 1;               // interior pairs (a middle cell counts as one)
#pragma unroll 1
  for (int c0 = 0; c0 < DIM * np; c0 += 2) {
    const int c = c0 + half;
    if (c < DIM * np) {
      const int ax = c / np, p = c - ax * np;
      const double d = ax == 0 ? dx : dy;
      eval_pair(tab, p, w, d, ker + r * kRec<DIM> + ax * 16);
    }
  }
}

__device__ __forceinline__ double2 strength_of(const int* idx, const double2* cv, int64_t off, int r) {
  return cv ? (idx ? cv[off + idx[r]] : cv[r]) : make_double2(1.0, 0.0);
}

// ------------------------------------------------------------------------------ planes
constexpr int kT2 = 32, kPitch2 = 36;    // tile edge, row pitch in cells (rows shift by 64 B of banks)

struct Plane64Smem {
  EsPairs tab;
  double ker[8][kR * kRec<2>];
  double2 acc[8][kT2 * kPitch2];         // one copy of the tile per warp
};

__global__ void __launch_bounds__(256)
    spread2_f64_kernel(SpreadArgs a, const RecD* __restrict__ recs, const int* __restrict__ idx,
                       const double2* __restrict__ cv, int64_t c_stride,
                       const int* __restrict__ starts, int real_pair, double2* __restrict__ fine,
                       const EsPairs tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Plane64Smem& sm = *reinterpret_cast<Plane64Smem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, w = a.w;
  const int64_t key = blockIdx.x, keygrid = (unsigned)key / (unsigned)a.n_tiles;
  const int tile = (int)(key - keygrid * a.n_tiles);
  const int tx = tile % a.ntile[0], ty = tile / a.ntile[0];
  const int trans = blockIdx.y;
  const int r0 = starts[key], r1 = starts[key + 1];
  const int copies = min(8, (r1 - r0 + kR - 1) / kR);     // warps with records
  for (int e = tid; e < (int)(sizeof(EsPairs) / 8); e += 256)
    reinterpret_cast<double*>(&sm.tab)[e] = reinterpret_cast<const double*>(&tab)[e];
  for (int e = tid; e < copies * kT2 * kPitch2; e += 256)
    sm.acc[0][e] = make_double2(0.0, 0.0);
  __syncthreads();
  double* const ker = sm.ker[warp];
  double2* const acc = sm.acc[warp];
  const int rows = 32 / w, li = lane % w, lj = lane / w;   // lanes with lj >= rows stay idle
  for (int b = r0 + warp * kR; b < r1; b += 8 * kR) {
    const int n = min(kR, r1 - b);
    double d0 = -0.5 * w, d1 = d0;
    int packed = 0;
    double2 c = make_double2(0.0, 0.0);
    if (lane < n) {
      const RecD q = recs[b + lane];
      d0 = q.dx;
      d1 = q.dy;
      packed = q.packed;
      c = strength_of(idx, cv, (int64_t)trans * c_stride, b + lane);
    }
    eval_records(sm.tab, w, a.beta, d0, d1, ker);
    __syncwarp();
    for (int r = 0; r < n; ++r) {
      const int pk = __shfl_sync(0xffffffffu, packed, r);
      const double cx = __shfl_sync(0xffffffffu, c.x, r), cy = __shfl_sync(0xffffffffu, c.y, r);
      const int x = (pk & 0xff) - 64 + li, ly = ((pk >> 8) & 0xff) - 64;
      const bool xin = lj < rows && x >= 0 && x < kT2;
      const double kx = ker[r * kRec<2> + li], kr = kx * cx;
      const double* const ky = ker + r * kRec<2> + 16;
      if (real_pair) {
        double* const col = reinterpret_cast<double*>(acc) + ((pk >> 24) & 1);
        for (int j = lj; j < w; j += rows) {
          const int y = ly + j;
          if (xin && y >= 0 && y < kT2) {
            double* const p = col + 2 * (y * kPitch2 + x);
            *p = fma(ky[j], kr, *p);
          }
        }
      } else {
        const double ki = kx * cy;
        for (int j = lj; j < w; j += rows) {
          const int y = ly + j;
          if (xin && y >= 0 && y < kT2) {
            double2* const p = acc + y * kPitch2 + x;
            double2 s = *p;
            s.x = fma(ky[j], kr, s.x);
            s.y = fma(ky[j], ki, s.y);
            *p = s;
          }
        }
      }
      __syncwarp();                       // the next record may touch the same cells
    }
  }
  __syncthreads();
  double2* const out = fine + (keygrid + trans) * a.n_fine + (int64_t)ty * kT2 * a.nf[0] + tx * kT2;
  for (int e = tid; e < kT2 * kT2; e += 256) {
    const int y = e / kT2, x = e % kT2;
    double2 s = make_double2(0.0, 0.0);
    for (int k = 0; k < copies; ++k) {
      const double2 v = sm.acc[k][y * kPitch2 + x];
      s.x += v.x;
      s.y += v.y;
    }
    out[(int64_t)y * a.nf[0] + x] = s;
  }
}

// ----------------------------------------------------------------------------- volumes
// A tile of a static frame holds a handful of records (40,000 atoms on three 320^3 grids: six), so
// the values of a chunk of 16 records are spread over all 256 threads.  A warp owns two z planes and
// covers the cells of a record's footprint inside the tile with consecutive lanes (on average 43
// cells at width 10: two passes); a thread per (x, y) column instead leaves most lanes of a record's
// clipped footprint idle (770 us per launch there, 674 this way; 1257 with a warp per record and atomics).
constexpr int kT3 = 16, kCh3 = 16;       // tile edge, records staged per chunk

struct Volume64Smem {
  EsPairs tab;
  double ker[kCh3 * kRec<3>];
  double2 str[kCh3];
  RecD rec[kCh3];
  double2 acc[kT3 * kT3 * kT3];          // [z][y][x]
};

__global__ void __launch_bounds__(256, 3)
    spread3_f64_kernel(SpreadArgs a, const RecD* __restrict__ recs, const int* __restrict__ idx,
                       const double2* __restrict__ cv, int64_t c_stride,
                       const int* __restrict__ starts, int real_pair, double2* __restrict__ fine,
                       const EsPairs tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Volume64Smem& sm = *reinterpret_cast<Volume64Smem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, w = a.w;
  const int64_t key = blockIdx.x, keygrid = (unsigned)key / (unsigned)a.n_tiles;
  const int tile = (int)(key - keygrid * a.n_tiles);
  const int tx = tile % a.ntile[0], ty = (tile / a.ntile[0]) % a.ntile[1];
  const int tz = tile / (a.ntile[0] * a.ntile[1]);
  const int trans = blockIdx.y;
  const int x = tid & 15, y = tid >> 4;                     // the cell this thread clears and writes
  const int p0 = 2 * warp;                                  // this warp's planes: p0, p0 + 1
  const int r0 = starts[key], r1 = starts[key + 1];
  double2* const out = fine + (keygrid + trans) * a.n_fine +
                       (((int64_t)tz * kT3) * a.nf[1] + ty * kT3 + y) * a.nf[0] + tx * kT3 + x;
  const int64_t plane = (int64_t)a.nf[1] * a.nf[0];
  if (r0 == r1) {                                           // an empty tile
#pragma unroll
    for (int z = 0; z < kT3; ++z) out[z * plane] = make_double2(0.0, 0.0);
    return;
  }
  for (int e = tid; e < (int)(sizeof(EsPairs) / 8); e += 256)
    reinterpret_cast<double*>(&sm.tab)[e] = reinterpret_cast<const double*>(&tab)[e];
  double2* const col = sm.acc + tid;                        // the thread's cell in plane z at col[256 z]
#pragma unroll
  for (int z = 0; z < kT3; ++z) col[256 * z] = make_double2(0.0, 0.0);
  const int np = (w + 1) / 2 - 1;                           // interior pairs
  const double two_over_w = 2.0 / w;
  for (int c0 = r0; c0 < r1; c0 += kCh3) {
    const int nc = min(kCh3, r1 - c0);
    __syncthreads();                                        // the previous chunk has been read
    if (tid < nc) {
      sm.rec[tid] = recs[c0 + tid];
      sm.str[tid] = strength_of(idx, cv, (int64_t)trans * c_stride, c0 + tid);
    }
    __syncthreads();
    // item = (end cell or interior pair of an axis, record): end cells first
    for (int e = tid; e < 3 * (2 + np) * nc; e += 256) {
      const int c = e / nc, r = e - c * nc;
      double* const k3 = sm.ker + r * kRec<3>;
      const int ax = c < 6 ? c >> 1 : (c - 6) / np;
      const double d = ax == 0 ? sm.rec[r].dx : (ax == 1 ? sm.rec[r].dy : sm.rec[r].dz);
      if (c < 6) {
        const int i = (c & 1) ? w - 1 : 0;
        k3[16 * ax + i] = es_end(d, i, two_over_w, a.beta);
      } else {
        eval_pair(sm.tab, c - 6 - ax * np, w, d, k3 + 16 * ax);
      }
    }
    __syncthreads();
    for (int r = 0; r < nc; ++r) {
      const int pk = sm.rec[r].packed;
      const int lz = ((pk >> 16) & 0xff) - 64;
      if (p0 + 1 < lz || p0 >= lz + w) continue;            // warp-uniform: misses our planes
      const bool u0 = p0 >= lz, u1 = p0 + 1 < lz + w;
      const int lx = (pk & 0xff) - 64, ly = ((pk >> 8) & 0xff) - 64;
      const int x0 = max(0, lx), y0 = max(0, ly);
      const int nx = min(kT3, lx + w) - x0, cells = nx * (min(kT3, ly + w) - y0);
      const double* const k3 = sm.ker + r * kRec<3>;
      const double2 c = sm.str[r];
      const double k0 = u0 ? k3[32 + p0 - lz] : 0.0, k1 = u1 ? k3[33 + p0 - lz] : 0.0;
      const unsigned inv = (65536u + nx - 1) / nx;          // i / nx for i < 256
      for (int i = lane; i < cells; i += 32) {
        const int iy = (int)((i * inv) >> 16), ix = i - iy * nx;
        const double v = k3[x0 - lx + ix] * k3[16 + y0 - ly + iy];
        double2* const at = sm.acc + p0 * 256 + (y0 + iy) * 16 + x0 + ix;
        if (real_pair) {
          double* const p = reinterpret_cast<double*>(at) + ((pk >> 24) & 1);
          const double vr = v * c.x;
          const double s0 = p[0], s1 = p[512];
          if (u0) p[0] = fma(vr, k0, s0);
          if (u1) p[512] = fma(vr, k1, s1);
        } else {
          const double vr = v * c.x, vi = v * c.y;
          const double2 s0 = at[0], s1 = at[256];
          if (u0) at[0] = make_double2(fma(vr, k0, s0.x), fma(vi, k0, s0.y));
          if (u1) at[256] = make_double2(fma(vr, k1, s1.x), fma(vi, k1, s1.y));
        }
      }
      __syncwarp();                                         // the next record may touch the same cells
    }
  }
  __syncthreads();
#pragma unroll
  for (int z = 0; z < kT3; ++z) out[z * plane] = col[256 * z];
}

}  // namespace

int launch_spread_f64(const SpreadArgs& a, const RecD* recs, const int* idx, const double2* cv,
                      int64_t c_stride, const int* starts, int nkeys, int ntrans, bool real_pair,
                      double2* fine, cudaStream_t s) {
  const int t = a.dim == 2 ? kT2 : kT3;
  if (a.w < 2 || a.w > 16 || a.tile[0] != t || a.tile[1] != t || (a.dim == 3 && a.tile[2] != t))
    return fail(MPSQ_ERR_ARG, "FP64 spread: width %d or tile not supported", a.w);
  if (nkeys <= 0) return MPSQ_OK;
  if (const int rc = a.dim == 2 ? allow_smem(spread2_f64_kernel, sizeof(Plane64Smem))
                                : allow_smem(spread3_f64_kernel, sizeof(Volume64Smem)))
    return rc;
  const dim3 grid((unsigned)nkeys, (unsigned)ntrans);
  const EsPairs tab = pairs_for(a.w, a.beta);
  const int rp = real_pair ? 1 : 0;
  if (a.dim == 2)
    spread2_f64_kernel<<<grid, 256, sizeof(Plane64Smem), s>>>(a, recs, idx, cv, c_stride, starts, rp,
                                                              fine, tab);
  else
    spread3_f64_kernel<<<grid, 256, sizeof(Volume64Smem), s>>>(a, recs, idx, cv, c_stride, starts, rp,
                                                               fine, tab);
  MPSQ_LAUNCH_CHECK();
  return MPSQ_OK;
}

}  // namespace mpsq
