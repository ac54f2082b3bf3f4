// Tensor-core spreading: packed real species pairs of volumes, and Q planes (FP32 results).
//
// Within one 16^3 tile the spread of the tile's point records onto z-plane p is a small
// matrix product
//     G_p[y, x] = sum_k A_p[y, k] B[k, x],   A_p[y, k] = s_k ky_k[y] kz_k[p],   B[k, x] = kx_k[x]
// over the records k (kx, ky, kz: the ES kernel values of record k along each axis, zero
// outside its w-cell support; s_k its real strength).  A record adds into the real part of the
// grid when it belongs to the first species of the pair and into the imaginary part otherwise
// (the pair is separated after the transform by Hermitian symmetry), so the two components
// are two independent products over disjoint record sets.
//
// The products run on the tensor cores as mma.sync m16n8k16 (f16 operands, FP32
// accumulators).  FP32 accuracy is kept by splitting each operand v into two f16 terms:
// hi = v with its 13 low mantissa bits cleared (exact in f16), lo = v - hi (exact in FP32,
// rounded to f16), and accumulating Ah*Bh + Ah*Bl + Al*Bh; the dropped Al*Bl term and the
// rounding of lo are below 2^-21 of each product.  From width 8 on (tolerances near 1e-7) the
// Al*Bl term is accumulated too (one more MMA per product term set, ~20 % less error at ~1.3 %
// more step time).  A and B carry a factor 2^10 so that the lo
// terms of kernel values down to ~1e-4 stay in the f16 normal range; the tile is scaled by
// 2^-20 when it is written.  Strengths must satisfy |s| <= 8 (the spatial Hann window's
// maximum), which keeps |A| <= 2^13 well inside the f16 range.
//
// A tile's cells are taken as 16 pencils of 4 z x 4 y cells (M = 16) along x (N = 16): a record joins
// the pencils its support touches (2.5 of the 16 on average at width 8 over the tile's halo copies)
// and the A operand of one is one fragment, s ky kz at its 16 (z, y) cells.  Products per plane
// instead (M = 16 y-rows, one fragment for each of the ~9.5 planes that a block of records sorted by
// start z touches) formed 3.7 times as many A operands, which bounded the kernel.  The planes form
// remains for the reproducible order (spread3_ordered_mma_kernel), whose sort by start z it shares.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "mpsq_internal.h"

namespace mpsq {
namespace {

constexpr int kCh = 256;            // staging slots per chunk (ordered kernel)
constexpr int kCap = kCh - 16;      // records per chunk (room for the alignment gap)
constexpr int kKp = kCh + 8;        // float row pitch: conflict-free 64-bit fragment loads
constexpr int kKh = kCh / 2 + 4;    // f16-pair row pitch: conflict-free 32-bit fragment loads

template <int W>
struct MmaSmem {
  static constexpr int kKeys = W + 15;   // start z in [-(W-1), 15]
  float ky[16][kKp];                     // s * ky * 2^10, row y, column slot
  float kz[16][kKp];                     // kz, row z
  uint32_t kxh[16][kKh];                 // hi(kx * 2^10) as f16 pairs (slots 2j, 2j+1), row x
  uint32_t kxl[16][kKh];                 // lo(kx * 2^10)
  int lz[kCh];                           // start z of the record in each slot
  RecF rec[kCh];                         // the record sorted into each slot
  float str[kCh];                        // its real strength
  int member[kCh];                       // the chunk's records grouped by key (chunk order)
  unsigned long long order[kCh];         // their first ordering word (cell offsets, dz bits)
  int count[2 * kKeys];
  int base[2 * kKeys];
  int tcount[2 * kKeys];                 // records per key over the whole tile (large tiles)
  int n0, b1, n1, msel;
};

// The ES kernel value of cell i of a support, phi(z) = exp(beta (sqrt(1 - z^2) - 1)) at
// z = (2 (u + i) - W) / W, u in [0, 1) the point's offset inside its first cell, as a
// polynomial in v = 2u - 1 per cell (Chebyshev interpolation on the host, monomial
// coefficients, Horner on the FMA pipe; no exp/sqrt on the special-function unit).  Degree
// W + 2 up to width 6, 8 at width 7, W from width 8 on: the lowest degrees whose FP32 Horner
// evaluation error (below 1e-7 of the kernel's peak, set by FP32 rounding) is no larger than
// that of W + 2.
template <int W>
struct EsPoly {
  static constexpr int kDeg = W >= 8 ? W : (W == 7 ? 8 : W + 2);
  float c[W][kDeg + 1];   // c[i][k]: coefficient of v^k for cell i
};

template <int W>
__device__ __forceinline__ float es_cell(const EsPoly<W>& p, int i, float v) {
  float r = p.c[i][EsPoly<W>::kDeg];
#pragma unroll
  for (int k = EsPoly<W>::kDeg - 1; k >= 0; --k) r = fmaf(r, v, p.c[i][k]);
  return r;
}

// Chebyshev interpolation of phi on each cell, converted to monomials in v (FP64 on the host).
template <int W>
EsPoly<W> make_es_poly(double beta) {
  constexpr int P = EsPoly<W>::kDeg;
  EsPoly<W> out{};
  for (int i = 0; i < W; ++i) {
    double f[P + 1], a[P + 1];
    for (int j = 0; j <= P; ++j) {
      const double v = std::cos(M_PI * (j + 0.5) / (P + 1));
      const double z = (2.0 * ((v + 1.0) * 0.5 + i) - W) / W;
      f[j] = std::exp(beta * (std::sqrt(std::max(1.0 - z * z, 0.0)) - 1.0));
    }
    for (int k = 0; k <= P; ++k) {
      double s = 0.0;
      for (int j = 0; j <= P; ++j) s += f[j] * std::cos(M_PI * k * (j + 0.5) / (P + 1));
      a[k] = 2.0 * s / (P + 1);
    }
    a[0] *= 0.5;
    // sum_k a_k T_k(v) in monomials: T_0 = 1, T_1 = v, T_{k+1} = 2 v T_k - T_{k-1}
    double t0[P + 1] = {}, t1[P + 1] = {}, m[P + 1] = {};
    t0[0] = 1.0;
    t1[1] = 1.0;
    for (int q = 0; q <= P; ++q) m[q] += a[0] * t0[q];
    if (P >= 1)
      for (int q = 0; q <= P; ++q) m[q] += a[1] * t1[q];
    for (int k = 2; k <= P; ++k) {
      double tk[P + 1] = {};
      for (int q = 0; q <= P; ++q) tk[q] = (q > 0 ? 2.0 * t1[q - 1] : 0.0) - t0[q];
      for (int q = 0; q <= P; ++q) m[q] += a[k] * tk[q];
      for (int q = 0; q <= P; ++q) {
        t0[q] = t1[q];
        t1[q] = tk[q];
      }
    }
    for (int q = 0; q <= P; ++q) out.c[i][q] = (float)m[q];
  }
  return out;
}

__device__ __forceinline__ float clear_low13(float v) {
  return __uint_as_float(__float_as_uint(v) & 0xFFFFE000u);
}

// Two FP32 lanes per instruction (PTX mul/sub .f32x2, IEEE round-to-nearest per lane).
__device__ __forceinline__ float2 mul_f32x2(float2 a, float2 b) {
  unsigned long long pa, pb, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(pa) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(pb) : "f"(b.x), "f"(b.y));
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pa), "l"(pb));
  float2 o;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
  return o;
}
__device__ __forceinline__ float2 sub_f32x2(float2 a, float2 b) {
  unsigned long long pa, pb, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(pa) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(pb) : "f"(b.x), "f"(b.y));
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pa), "l"(pb));
  float2 o;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
  return o;
}

__device__ __forceinline__ uint32_t pack_f16x2(float first, float second) {
  const __half2 h = __floats2half2_rn(first, second);   // first -> low 16 bits
  uint32_t u;
  memcpy(&u, &h, sizeof(u));
  return u;
}

__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 "
               "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same from zero.
__device__ __forceinline__ void mma_16816_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 "
               "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}

// Four 8x8 f16 matrices from shared memory (ldmatrix): lane i gives the address of row i % 8 of
// matrix i / 8 (16 bytes); r[q] receives row lane / 4, columns 2 (lane % 4) .. +1 of matrix q.
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* row_addr) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(row_addr);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

// Split f16 A fragment (hi, lo) of plane p for the K-block starting at slot `first`:
// rows g, g+8 (y) x columns 2t, 2t+1, 2t+8, 2t+9 (records), A = (s ky)[y] * kz[p].
template <int W>
__device__ __forceinline__ void build_a(const MmaSmem<W>& sm, int p, int first, int t,
                                        float2 yA0, float2 yA1, float2 yB0, float2 yB1,
                                        uint32_t (&ah)[4], uint32_t (&al)[4]) {
  const float2 zA = *reinterpret_cast<const float2*>(&sm.kz[p][first + 2 * t]);
  const float2 zB = *reinterpret_cast<const float2*>(&sm.kz[p][first + 2 * t + 8]);
  // products and lo terms two lanes per instruction
  const float2 a[4] = {mul_f32x2(yA0, zA), mul_f32x2(yA1, zA), mul_f32x2(yB0, zB),
                       mul_f32x2(yB1, zB)};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 h = make_float2(clear_low13(a[j].x), clear_low13(a[j].y));
    ah[j] = pack_f16x2(h.x, h.y);
    const float2 l = sub_f32x2(a[j], h);
    al[j] = pack_f16x2(l.x, l.y);
  }
}

// One component's K-blocks [kb0, kb1) of the staged chunk into acc[plane][n-tile][4].
template <int W>
__device__ __forceinline__ void mma_region(const MmaSmem<W>& sm, int kb0, int kb1, int end,
                                           int p0, int g, int t, float (&acc)[2][2][4]) {
  for (int kb = kb0; kb < kb1; ++kb) {
    const int first = kb * 16;
    const int last = min(first + 15, end - 1);
    const int zlo = sm.lz[first], zhi = sm.lz[last] + W - 1;
    const bool use0 = p0 >= zlo && p0 <= zhi;
    const bool use1 = p0 + 1 >= zlo && p0 + 1 <= zhi;
    if (!use0 && !use1) continue;                       // warp-uniform
    // B fragments of both n-tiles (hi and lo) by ldmatrix: matrix q = lane / 8 covers x rows
    // (q / 2) * 8 .. +7 and records (q % 2) * 8 .. +7 of the K-block; the four registers are
    // b0, b1 of n-tile 0 and b0, b1 of n-tile 1
    uint32_t bh4[4], bl4[4];
    {
      const int lane = 4 * g + t, q = lane >> 3, r = lane & 7;
      const int row = (q >> 1) * 8 + r, col = kb * 8 + (q & 1) * 4;   // u32 column (f16 pairs)
      ldmatrix_x4(bh4, &sm.kxh[row][col]);
      ldmatrix_x4(bl4, &sm.kxl[row][col]);
    }
    const uint32_t bh[2][2] = {{bh4[0], bh4[1]}, {bh4[2], bh4[3]}};
    const uint32_t bl[2][2] = {{bl4[0], bl4[1]}, {bl4[2], bl4[3]}};
    const float2 yA0 = *reinterpret_cast<const float2*>(&sm.ky[g][first + 2 * t]);
    const float2 yA1 = *reinterpret_cast<const float2*>(&sm.ky[g + 8][first + 2 * t]);
    const float2 yB0 = *reinterpret_cast<const float2*>(&sm.ky[g][first + 2 * t + 8]);
    const float2 yB1 = *reinterpret_cast<const float2*>(&sm.ky[g + 8][first + 2 * t + 8]);
    // Each product term is issued to every accumulator chain before the next term, so that
    // consecutive MMAs are independent (the smallest terms first).  The tensor cores truncate each
    // sum they return, which along a chain over all K-blocks of a crowded tile adds up to a bias
    // (over 1e-5 of the amplitude for 1,000 coinciding records): a K-block is summed from zero and added rounded to nearest.
    auto add = [&](int plane, const float (&p)[2][4]) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[plane][nt][e] += p[nt][e];
    };
    if (use0 && use1) {   // both planes: four independent accumulator chains
      uint32_t ah0[4], al0[4], ah1[4], al1[4];
      build_a(sm, p0, first, t, yA0, yA1, yB0, yB1, ah0, al0);
      build_a(sm, p0 + 1, first, t, yA0, yA1, yB0, yB1, ah1, al1);
      float s0[2][4], s1[2][4];
      if constexpr (W >= 8) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          mma_16816_first(s0[nt], al0, bl[nt][0], bl[nt][1]);
          mma_16816_first(s1[nt], al1, bl[nt][0], bl[nt][1]);
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          mma_16816(s0[nt], al0, bh[nt][0], bh[nt][1]);
          mma_16816(s1[nt], al1, bh[nt][0], bh[nt][1]);
        }
      } else {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          mma_16816_first(s0[nt], al0, bh[nt][0], bh[nt][1]);
          mma_16816_first(s1[nt], al1, bh[nt][0], bh[nt][1]);
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        mma_16816(s0[nt], ah0, bl[nt][0], bl[nt][1]);
        mma_16816(s1[nt], ah1, bl[nt][0], bl[nt][1]);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        mma_16816(s0[nt], ah0, bh[nt][0], bh[nt][1]);
        mma_16816(s1[nt], ah1, bh[nt][0], bh[nt][1]);
      }
      add(0, s0);
      add(1, s1);
    } else {              // one of them
      auto one = [&](int plane) {
        uint32_t ah[4], al[4];
        build_a(sm, p0 + plane, first, t, yA0, yA1, yB0, yB1, ah, al);
        float s[2][4];
        if constexpr (W >= 8) {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma_16816_first(s[nt], al, bl[nt][0], bl[nt][1]);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma_16816(s[nt], al, bh[nt][0], bh[nt][1]);
        } else {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma_16816_first(s[nt], al, bh[nt][0], bh[nt][1]);
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) mma_16816(s[nt], ah, bl[nt][0], bl[nt][1]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) mma_16816(s[nt], ah, bh[nt][0], bh[nt][1]);
        add(plane, s);
      };
      if (use0) one(0);
      else one(1);
    }
  }
}

template <int W>
__global__ void __launch_bounds__(256, 3)
    spread3_ordered_mma_kernel(SpreadArgs a, const RecF* __restrict__ recs,
                            const float2* __restrict__ cv, const int* __restrict__ starts,
                            float2* __restrict__ fine, const EsPoly<W> poly, int64_t key0,
                            int z0, int64_t gstride) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MmaSmem<W>& sm = *reinterpret_cast<MmaSmem<W>*>(smem_raw);
  constexpr int K1 = MmaSmem<W>::kKeys;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int p0 = 2 * warp;
  const int64_t key = key0 + blockIdx.x;   // < 2^31
  const int keygrid = (int)((unsigned)key / (unsigned)a.n_tiles);
  const int tile = (int)((unsigned)key - (unsigned)keygrid * (unsigned)a.n_tiles);
  const int tx = tile % a.ntile[0];
  const int ty = (tile / a.ntile[0]) % a.ntile[1];
  const int tz = tile / (a.ntile[0] * a.ntile[1]);
  float acc_re[2][2][4], acc_im[2][2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc_re[i][j][k] = acc_im[i][j][k] = 0.0f;
  const int r0 = starts[key], r1 = starts[key + 1];
  // Chunks of at most kCap records: all of the tile's records when they fit one chunk; otherwise whole (component, start z) keys, counted
  // first, packed greedily into chunks (keys in order), so that the partition, like the order
  // inside a chunk, does not depend on the order the records were binned in.  A single key
  // with more than kCap records (an extremely dense tile) takes the binning order.
  auto key_of = [&](const RecF& q) {
    const int lz = ((q.packed >> 16) & 0xff) - 64;
    return ((q.packed >> 24) & 1) * K1 + min(max(lz + W - 1, 0), K1 - 1);
  };
  auto strength = [&](int r) {
    return !cv ? 1.0f : cv[r].x;
  };
  bool by_key = false;
  if (r1 - r0 > kCap) {
    for (int e = tid; e < 2 * K1; e += 256) sm.tcount[e] = 0;
    __syncthreads();
    for (int r = r0 + tid; r < r1; r += 256) atomicAdd(&sm.tcount[key_of(recs[r])], 1);
    __syncthreads();
    by_key = true;
    for (int e = 0; e < 2 * K1; ++e) by_key = by_key && sm.tcount[e] <= kCap;
  }
  int c0 = r0, kb = 0;
  for (;;) {
    int n = 0, kb_hi = kb;
    if (by_key) {
      if (kb >= 2 * K1) break;
      while (kb_hi < 2 * K1 && n + sm.tcount[kb_hi] <= kCap) n += sm.tcount[kb_hi++];
    } else {
      if (c0 >= r1) break;
      n = min(kCap, r1 - c0);
    }
    {  // zero the staging arrays (alignment-gap slots and out-of-support rows must read 0)
      uint4* z4 = reinterpret_cast<uint4*>(&sm.ky[0][0]);
      constexpr int nz = (int)((sizeof(sm.ky) + sizeof(sm.kz) + sizeof(sm.kxh) + sizeof(sm.kxl)) / 16);
      for (int e = tid; e < nz; e += 256) z4[e] = make_uint4(0u, 0u, 0u, 0u);
      for (int e = tid; e < 2 * K1; e += 256) sm.count[e] = 0;
      if (tid == 0) sm.msel = 0;
    }
    __syncthreads();
    // 1. the chunk's records into slots 0..n-1 in any order (by position, or selected by key)
    RecF rec;
    float sv = 0.0f;
    int k = 0, rank = 0;
    if (!by_key) {
      if (tid < n) {
        sm.rec[tid] = recs[c0 + tid];
        sm.str[tid] = strength(c0 + tid);
      }
    } else {
      for (int r = r0 + tid; r < r1; r += 256) {
        const RecF q = recs[r];
        const int k = key_of(q);
        if (k >= kb && k < kb_hi) {
          const int at = atomicAdd(&sm.msel, 1);
          sm.rec[at] = q;
          sm.str[at] = strength(r);
        }
      }
    }
    __syncthreads();
    // 2. group the records by key (component, start z)
    if (tid < n) {
      rec = sm.rec[tid];
      sv = sm.str[tid];
      k = key_of(rec);
      rank = atomicAdd(&sm.count[k], 1);
    }
    __syncthreads();
    // 3. exclusive scan of the key counts (one warp; K1 <= 23 keys per component); the
    //    second component starts on a multiple of 16
    if (warp == 0) {
      const int c0n = lane < K1 ? sm.count[lane] : 0;
      const int c1n = lane < K1 ? sm.count[K1 + lane] : 0;
      int i0 = c0n, i1 = c1n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u0 = __shfl_up_sync(0xffffffffu, i0, o), u1 = __shfl_up_sync(0xffffffffu, i1, o);
        if (lane >= o) {
          i0 += u0;
          i1 += u1;
        }
      }
      const int n0 = __shfl_sync(0xffffffffu, i0, 31), n1 = __shfl_sync(0xffffffffu, i1, 31);
      const int b1 = (n0 + 15) & ~15;
      if (lane < K1) {
        sm.base[lane] = i0 - c0n;
        sm.base[K1 + lane] = b1 + i1 - c1n;
      }
      if (lane == 0) {
        sm.n0 = n0;
        sm.b1 = b1;
        sm.n1 = n1;
      }
    }
    __syncthreads();
    // 4. the slot within the key: the order by content (cell
    //    offsets, then offsets and strength bits), so that the slots, and with them the
    //    accumulation order, follow from the record set alone; records equal in every bit may
    //    take either order
    int pos = rank;
    const uint64_t mine =
        tid < n ? ((uint64_t)(uint32_t)rec.packed << 32) | __float_as_uint(rec.dz) : 0ull;
    if (tid < n) {
      sm.member[sm.base[k] + rank] = tid;
      sm.order[sm.base[k] + rank] = mine;
    }
    __syncthreads();
    if (tid < n) {
      pos = 0;
      const int b = sm.base[k], cnt = sm.count[k];
      for (int q = b; q < b + cnt; ++q) {
        const uint64_t other = sm.order[q];   // one load per member; the record only on a tie
        bool before = other < mine;
        if (other == mine && q != b + rank) {
          const int o = sm.member[q];
          const RecF& u = sm.rec[o];
          const uint32_t a[3] = {__float_as_uint(u.dy), __float_as_uint(u.dx), __float_as_uint(sm.str[o])};
          const uint32_t m[3] = {__float_as_uint(rec.dy), __float_as_uint(rec.dx), __float_as_uint(sv)};
          before = a[0] != m[0] ? a[0] < m[0] : a[1] != m[1] ? a[1] < m[1] : a[2] != m[2] ? a[2] < m[2] : o < tid;
        }
        pos += before ? 1 : 0;
      }
    }
    __syncthreads();
    if (tid < n) {
      const int slot = sm.base[k] + pos;
      sm.rec[slot] = rec;
      sm.str[slot] = sv;
    }
    __syncthreads();
    // 5. thread t evaluates the kernel of the record in slot t and writes its support rows
    //    (consecutive threads write consecutive columns of a row: no bank conflicts)
    {
      const int st = tid;
      const bool live = st < sm.n0 || (st >= sm.b1 && st < sm.b1 + sm.n1);
      if (live) {
        const RecF q = sm.rec[st];
        const float s = sm.str[st] * 1024.0f;
        const int lx = (q.packed & 0xff) - 64;
        const int ly = ((q.packed >> 8) & 0xff) - 64;
        const int lz = ((q.packed >> 16) & 0xff) - 64;
        // offsets d in [-W/2, -W/2 + 1) -> polynomial variable v = 2d + W - 1 in [-1, 1)
        const float vx = fmaf(2.0f, q.dx, (float)(W - 1));
        const float vy = fmaf(2.0f, q.dy, (float)(W - 1));
        const float vz = fmaf(2.0f, q.dz, (float)(W - 1));
        __half* xh = reinterpret_cast<__half*>(&sm.kxh[0][0]);
        __half* xl = reinterpret_cast<__half*>(&sm.kxl[0][0]);
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const int x = lx + i, y = ly + i, z = lz + i;
          if (x >= 0 && x < 16) {
            const float v = es_cell(poly, i, vx) * 1024.0f;
            const float h = clear_low13(v);
            xh[x * 2 * kKh + st] = __float2half_rn(h);
            xl[x * 2 * kKh + st] = __float2half_rn(v - h);
          }
          if (y >= 0 && y < 16) sm.ky[y][st] = es_cell(poly, i, vy) * s;
          if (z >= 0 && z < 16) sm.kz[z][st] = es_cell(poly, i, vz);
        }
        sm.lz[st] = lz;
      }
    }
    __syncthreads();
    const int n0 = sm.n0, b1 = sm.b1, n1 = sm.n1;
    mma_region<W>(sm, 0, (n0 + 15) >> 4, n0, p0, g, t, acc_re);
    mma_region<W>(sm, b1 >> 4, (b1 + n1 + 15) >> 4, b1 + n1, p0, g, t, acc_im);
    c0 += kCap;
    kb = kb_hi;
    __syncthreads();   // another chunk reuses the staging arrays
  }
  float2* out = fine + (int64_t)keygrid * gstride;
  const int64_t nf0 = a.nf[0], nf1 = a.nf[1];
  const float sc = 1.0f / 1048576.0f;
#pragma unroll
  for (int pi = 0; pi < 2; ++pi) {
    const int64_t zrow = ((int64_t)tz * 16 - z0 + p0 + pi) * nf1 + (int64_t)ty * 16;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const int64_t xcol = (int64_t)tx * 16 + nt * 8 + 2 * t;
#pragma unroll
      for (int hv = 0; hv < 2; ++hv) {
        const int y = g + 8 * hv;
        const float4 v = make_float4(acc_re[pi][nt][2 * hv] * sc, acc_im[pi][nt][2 * hv] * sc,
                                     acc_re[pi][nt][2 * hv + 1] * sc, acc_im[pi][nt][2 * hv + 1] * sc);
        *reinterpret_cast<float4*>(out + (zrow + y) * nf0 + xcol) = v;
      }
    }
  }
}

// The polynomial for one kernel width and beta, kept per width (a process uses one beta each).
template <int W>
EsPoly<W> es_poly_for(double beta) {
  static std::mutex mu;
  static double cached_beta = -1.0;
  static EsPoly<W> poly;
  std::lock_guard<std::mutex> lock(mu);
  if (cached_beta != beta) {
    poly = make_es_poly<W>(beta);
    cached_beta = beta;
  }
  return poly;
}

// ------------------------------------------------------------------------- Q planes
// One 32 x 32 tile of a plane is G[y, x] = sum_k (s_k ky_k[y]) kx_k[x] over its records: one
// matrix product with K = the records, for the real and the imaginary part of the strength
// (packed pairs: the part of the record's component, 0 for the other).  Both operands are split
// into two f16 terms as above and all four products are accumulated in FP32 registers, so the
// sum needs no atomics and does not care how many records coincide (the atoms of a crystal
// column project onto one cell, where shared-memory atomics serialise).
//
// One CTA of 8 warps per tile, chunks of 128 records.  Two threads per record evaluate its x and y
// values into the record's own rows ([record][cell], f16 pairs), which ldmatrix.trans turns into
// fragments; before the next chunk each thread clears the words it wrote, so nothing is zero-filled
// but the first time.  Warp w takes the K-blocks w >> 1 and (w >> 1) + 4 of a chunk (16 records
// each) for the x half w & 1 of the tile: 10 ldmatrix per 32 MMAs, 32 accumulator registers.  A
// K-block without records of a component skips that component.  Bound by shared-memory bandwidth:
// 11 frames of 163,840 atoms (three 320^2 grids each, width 7) took 166 us per launch with a warp per
// 16 x 16 cells over [cell][record] arrays zero-filled per chunk, 116 us in this form; the
// shared-memory atomics of one record per warp took 1.48 ms.
constexpr int kPCh = 128;          // records per chunk
constexpr int kPP = 40;            // row pitch in f16 (80 B): conflict-free ldmatrix rows
constexpr int kPT = 32;            // tile edge

struct PlaneSmem {
  __half a[2][2][kPCh][kPP];       // [component][hi, lo][record][y]: s ky 2^10
  __half b[2][kPCh][kPP];          // [hi, lo][record][x]: kx 2^10
  int used[2][kPCh / 16];          // components present in each K-block (bits), by chunk parity
};

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], unsigned a) {   // shared address
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* row_addr) {
  ldmatrix_x4_trans(r, (unsigned)__cvta_generic_to_shared(row_addr));
}

// The f16 hi and lo terms of v[0..W) into the rows at cells l .. l+W-1, those inside the tile, as
// 32-bit words of two cells (cells of a word outside the support are zero): packed in pairs from the
// support's start, and moved up by one cell where that is odd.
template <int W, int CELLS>
__device__ __forceinline__ void put_row(__half* hi, __half* lo, int l, const float (&v)[W]) {
  const int sh = (l & 1) * 16, w0 = l >> 1;
  uint32_t ph = 0u, pl = 0u;         // the pair before
#pragma unroll
  for (int j = 0; j <= W / 2; ++j) {
    uint32_t h = 0u, q = 0u;
    if (2 * j < W) {
      const float a = v[2 * j], b = 2 * j + 1 < W ? v[2 * j + 1 < W ? 2 * j + 1 : 0] : 0.0f;
      const float ah = clear_low13(a), bh = clear_low13(b);
      h = pack_f16x2(ah, bh);
      q = pack_f16x2(a - ah, b - bh);
    }
    if ((unsigned)(w0 + j) < (unsigned)(CELLS / 2)) {
      reinterpret_cast<uint32_t*>(hi)[w0 + j] = __funnelshift_l(ph, h, sh);
      reinterpret_cast<uint32_t*>(lo)[w0 + j] = __funnelshift_l(pl, q, sh);
    }
    ph = h;
    pl = q;
  }
}
// The same with both alignments packed and one selected (fewer registers live across the words: the
// plane kernel spills with the form above, 122 us per launch of the job below instead of 116).
template <int W, int CELLS>
__device__ __forceinline__ void put_row_select(__half* hi, __half* lo, int l, const float (&v)[W]) {
  const bool odd = l & 1;
  const int w0 = l >> 1;
  float h[W];
#pragma unroll
  for (int i = 0; i < W; ++i) h[i] = clear_low13(v[i]);
#pragma unroll
  for (int j = 0; j <= W / 2; ++j) {
    // even start: cells 2j, 2j + 1; odd start: cells 2j - 1, 2j
    const int a = 2 * j < W ? 2 * j : 0, b = 2 * j + 1 < W ? 2 * j + 1 : 0, o = j > 0 ? 2 * j - 1 : 0;
    const float e0 = 2 * j < W ? h[a] : 0.0f, e1 = 2 * j + 1 < W ? h[b] : 0.0f, o0 = j > 0 ? h[o] : 0.0f;
    const float f0 = 2 * j < W ? v[a] - e0 : 0.0f, f1 = 2 * j + 1 < W ? v[b] - e1 : 0.0f;
    const float g0 = j > 0 ? v[o] - o0 : 0.0f;
    if ((unsigned)(w0 + j) < (unsigned)(CELLS / 2)) {
      reinterpret_cast<uint32_t*>(hi)[w0 + j] = odd ? pack_f16x2(o0, e0) : pack_f16x2(e0, e1);
      reinterpret_cast<uint32_t*>(lo)[w0 + j] = odd ? pack_f16x2(g0, f0) : pack_f16x2(f0, f1);
    }
  }
}
template <int W, int CELLS>
__device__ __forceinline__ void clear_row(__half* hi, __half* lo, int l) {
#pragma unroll
  for (int j = 0; j <= W / 2; ++j)
    if ((unsigned)((l >> 1) + j) < (unsigned)(CELLS / 2)) {
      reinterpret_cast<uint32_t*>(hi)[(l >> 1) + j] = 0u;
      reinterpret_cast<uint32_t*>(lo)[(l >> 1) + j] = 0u;
    }
}

template <int W>
__global__ void __launch_bounds__(256, 3)
    spread2_mma_kernel(SpreadArgs a, const RecF* __restrict__ recs, const float2* __restrict__ cv,
                       const int* __restrict__ starts, int real_pair, float2* __restrict__ fine,
                       const EsPoly<W> poly) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PlaneSmem& sm = *reinterpret_cast<PlaneSmem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned key = blockIdx.x;
  const unsigned keygrid = key / (unsigned)a.n_tiles, tile = key - keygrid * (unsigned)a.n_tiles;
  const unsigned ty = tile / (unsigned)a.ntile[0], tx = tile - ty * (unsigned)a.ntile[0];
  const int mx = warp & 1, kw = warp >> 1;       // x half, first K-block
  float acc[2][2][2][4] = {};                    // [component][y half][x eighth][fragment]
  const int r0 = starts[key], r1 = starts[key + 1];
  // rows that some chunk uses (a multiple of 16)
  const int rows = min(kPCh, (r1 - r0 + 15) & ~15);
  for (int e = tid; e < 6 * rows * (kPP / 8); e += 256) {
    const int p = e / (rows * (kPP / 8)), c = e - p * (rows * (kPP / 8));
    reinterpret_cast<uint4*>(&sm.a[0][0][0][0] + p * (kPCh * kPP))[c] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (tid < 2 * (kPCh / 16)) sm.used[0][tid] = real_pair ? 0 : 3;
  const int k = tid & (kPCh - 1);                // this thread's record of the chunk
  const bool yaxis = tid >= kPCh;
  int l = 0, p0 = 0, par = 0;
  bool wrote = false;
  RecF q;
  float2 c = make_float2(1.0f, 0.0f);
  auto fetch = [&](int r) {                      // the thread's next record, ahead of its use
    if (r < r1) {
      q = recs[r];
      if (cv && yaxis) c = cv[r];
    }
  };
  fetch(r0 + k);
  __syncthreads();
  for (int c0 = r0; c0 < r1; c0 += kPCh, par ^= 1) {
    const int n = min(kPCh, r1 - c0);
    const int nb = (n + 15) >> 4;               // K-blocks of 16 records
    if (wrote) {
      if (yaxis) {
        clear_row<W, kPT>(sm.a[p0][0][k], sm.a[p0][1][k], l);
        if (!real_pair) clear_row<W, kPT>(sm.a[1][0][k], sm.a[1][1][k], l);
      } else {
        clear_row<W, kPT>(sm.b[0][k], sm.b[1][k], l);
      }
    }
    wrote = k < n;
    if (wrote) {
      l = (yaxis ? (q.packed >> 8) & 0xff : q.packed & 0xff) - 64;
      const float v = fmaf(2.0f, yaxis ? q.dy : q.dx, (float)(W - 1));   // [-1, 1)
      float f[W];
#pragma unroll
      for (int i = 0; i < W; ++i) f[i] = es_cell(poly, i, v);
      const float s0 = (yaxis ? c.x : 1.0f) * 1024.0f;
      float fs[W];
#pragma unroll
      for (int i = 0; i < W; ++i) fs[i] = f[i] * s0;
      if (yaxis) {
        p0 = real_pair ? (q.packed >> 24) & 1 : 0;
        if (real_pair) atomicOr(&sm.used[par][k >> 4], 1 << p0);
        put_row_select<W, kPT>(sm.a[p0][0][k], sm.a[p0][1][k], l, fs);
        if (!real_pair) {
#pragma unroll
          for (int i = 0; i < W; ++i) fs[i] = f[i] * (c.y * 1024.0f);
          put_row_select<W, kPT>(sm.a[1][0][k], sm.a[1][1][k], l, fs);
        }
      } else {
        put_row_select<W, kPT>(sm.b[0][k], sm.b[1][k], l, fs);
      }
    }
    fetch(c0 + kPCh + k);
    __syncthreads();
    if (real_pair && tid < kPCh / 16) sm.used[par ^ 1][tid] = 0;   // for the next chunk
    for (int kb = kw; kb < nb; kb += 4) {
      // ldmatrix.trans rows are records: A matrices (y 0-7, k 0-7), (y 8-15, k 0-7), (y 0-7,
      // k 8-15), (y 8-15, k 8-15); B matrices (x 0-7, k 0-7), (x 0-7, k 8-15), then x 8-15
      const int m = lane >> 3, r = 16 * kb + (lane & 7);
      const int ar = r + (m >> 1) * 8, ac = (m & 1) * 8;
      const int br = r + (m & 1) * 8, bc = 16 * mx + (m >> 1) * 8;
      uint32_t bh[4], bl[4];
      ldmatrix_x4_trans(bh, &sm.b[0][br][bc]);
      ldmatrix_x4_trans(bl, &sm.b[1][br][bc]);
      const int used = sm.used[par][kb];
#pragma unroll
      for (int comp = 0; comp < 2; ++comp) {
        if (!((used >> comp) & 1)) continue;       // warp-uniform
#pragma unroll
        for (int my = 0; my < 2; ++my) {
          uint32_t ah[4], al[4];
          ldmatrix_x4_trans(ah, &sm.a[comp][0][ar][16 * my + ac]);
          ldmatrix_x4_trans(al, &sm.a[comp][1][ar][16 * my + ac]);
          // The tensor core truncates its running sum: the bias of a chain over all records of a
          // cell grows with their number (1.7e-5 for 1,024 coinciding atoms), so each K-block is
          // summed on its own and added rounded to nearest.
          float p[2][4] = {};
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma_16816(p[nt], al, bl[2 * nt], bl[2 * nt + 1]);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma_16816(p[nt], al, bh[2 * nt], bh[2 * nt + 1]);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma_16816(p[nt], ah, bl[2 * nt], bl[2 * nt + 1]);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) mma_16816(p[nt], ah, bh[2 * nt], bh[2 * nt + 1]);
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[comp][my][nt][e] += p[nt][e];
        }
      }
    }
    __syncthreads();                            // the next chunk rewrites the rows
  }
  // sum of the four partial tiles over the staging memory, as complex [y][x]
  float* const part = reinterpret_cast<float*>(smem_raw) + kw * (2 * kPT * kPT);
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int my = 0; my < 2; ++my)
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int hv = 0; hv < 2; ++hv) {
        const int y = 16 * my + g + 8 * hv, x = 16 * mx + 8 * nt + 2 * t;
        *reinterpret_cast<float4*>(part + 2 * (y * kPT + x)) =
            make_float4(acc[0][my][nt][2 * hv], acc[1][my][nt][2 * hv],
                        acc[0][my][nt][2 * hv + 1], acc[1][my][nt][2 * hv + 1]);
      }
  __syncthreads();
  const float sc = 1.0f / 1048576.0f;
  const float4* const sum = reinterpret_cast<const float4*>(smem_raw);
  float2* const out = fine + (int64_t)keygrid * a.n_fine + (int64_t)ty * kPT * a.nf[0] + tx * kPT;
  for (int e = tid; e < kPT * kPT / 2; e += 256) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float4 u = sum[p * (kPT * kPT / 2) + e];
      v = make_float4(v.x + u.x, v.y + u.y, v.z + u.z, v.w + u.w);
    }
    const int y = e / (kPT / 2), x = 2 * (e % (kPT / 2));
    *reinterpret_cast<float4*>(out + (int64_t)y * a.nf[0] + x) =
        make_float4(v.x * sc, v.y * sc, v.z * sc, v.w * sc);
  }
}

template <int W>
int launch_plane_w(const SpreadArgs& a, const RecF* recs, const float2* cv, const int* starts,
                   int nkeys, int real_pair, float2* fine, cudaStream_t s) {
  if (const int rc = allow_smem(spread2_mma_kernel<W>, sizeof(PlaneSmem))) return rc;
  spread2_mma_kernel<W><<<(unsigned)nkeys, 256, sizeof(PlaneSmem), s>>>(
      a, recs, cv, starts, real_pair, fine, es_poly_for<W>(a.beta));
  MPSQ_LAUNCH_CHECK();
  return MPSQ_OK;
}

// --------------------------------------------------------------- volumes, packed real pairs
// One CTA of 8 warps per tile.  Per chunk of 224 records: (1) the records' rows are cleared; (2) one
// thread per (record, axis) evaluates the kernel into the record's row (x as f16 hi and lo, s ky and
// kz as FP32) and the y threads note which pencils the record touches; (3) warp w takes the pencils 2w
// and 2w + 1: it collects their records by ballots (first-species ones from the front of its list,
// second-species ones from the back), then per K-block of 16 entries the B fragments come by
// ldmatrix.trans from the records' rows, the A fragment from eight products, and the MMAs of the
// components present follow (a block that holds both masks A once for each).  Cost follows the
// records: a nearly empty tile costs its 32 KB of output and two barriers.  Per launch, planes form and
// this one: three 512^3 grids with 42 records per tile (width 7) 1.30 ms and 0.95, three 1152^3 grids
// (width 6) 14.4 ms and 10.6, one 320^3 grid with 10 records per tile 108 us and 76; one 384^3 grid with
// 215 records per tile (width 8) 302 us and 293.  50 KB of shared memory
// keep the SM's split at 164 KB with three CTAs: with 68 KB each (256 records, padded rows) it went to
// 228 KB, which left the passes of a second frame lane without L1 (5.31 ms for eight frames on one
// lane, 5.78 on two).
constexpr int kNCh = 224;            // records per chunk

__device__ __forceinline__ float lds_f32(unsigned a) {        // shared address
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float2 lds_f32x2(unsigned a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}

struct PencilRow {                   // 208 B: eight rows' 16-byte pieces fall on different banks
  __half xh[16], xl[16];             // hi and lo of kx 2^10
  float ky[16];                      // s ky 2^10
  float kz[16];
  uint32_t pad[4];
};
struct PencilSmem {
  PencilRow row[kNCh + 1];           // the last one stays zero (list padding)
  uint32_t mask[kNCh];               // pencils touched (bit 4 zq + yq), component in bit 16
  unsigned char list[16][kNCh];      // records of a pencil
};
static_assert(sizeof(PencilRow) == 208, "row pitch");

template <int W>
__global__ void __launch_bounds__(256, 3)
    spread3_pencil_mma_kernel(SpreadArgs a, const RecF* __restrict__ recs,
                              const float2* __restrict__ cv, const int* __restrict__ starts,
                              float2* __restrict__ fine, const EsPoly<W> poly, int64_t key0, int z0,
                              int64_t gstride) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PencilSmem& sm = *reinterpret_cast<PencilSmem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  // (32-bit index arithmetic: a 64-bit division per warp was a fifth of a sparse tile's instructions)
  const unsigned key = (unsigned)key0 + blockIdx.x;
  const unsigned keygrid = key / (unsigned)a.n_tiles, tile = key - keygrid * (unsigned)a.n_tiles;
  const unsigned tyz = tile / (unsigned)a.ntile[0], tx = tile - tyz * (unsigned)a.ntile[0];
  const unsigned tz = tyz / (unsigned)a.ntile[1], ty = tyz - tz * (unsigned)a.ntile[1];
  float acc[2][2][2][4] = {};        // [pencil][component][x half][fragment]
  const int r0 = starts[key], r1 = starts[key + 1];
  if (tid < 13) reinterpret_cast<uint4*>(&sm.row[kNCh])[tid] = make_uint4(0u, 0u, 0u, 0u);
  for (int c0 = r0; c0 < r1; c0 += kNCh) {
    const int n = min(kNCh, r1 - c0);
    if (c0 > r0) __syncthreads();    // the previous chunk has been read
    for (int e = tid; e < 13 * n; e += 256) reinterpret_cast<uint4*>(sm.row)[e] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (int e = tid; e < 3 * n; e += 256) {
      const int ax = (e >= n ? 1 : 0) + (e >= 2 * n ? 1 : 0), r = e - ax * n;
      const RecF q = recs[c0 + r];
      PencilRow& row = sm.row[r];
      const int l = ((q.packed >> (8 * ax)) & 0xff) - 64;
      const float d = ax == 0 ? q.dx : (ax == 1 ? q.dy : q.dz);
      const float v = fmaf(2.0f, d, (float)(W - 1));       // [-1, 1)
      const float s = ax == 2 ? 1.0f : (ax == 1 && cv ? cv[c0 + r].x * 1024.0f : 1024.0f);
      float f[W];
#pragma unroll
      for (int i = 0; i < W; ++i) f[i] = es_cell(poly, i, v) * s;
      if (ax == 0) {
        put_row<W, 16>(row.xh, row.xl, l, f);
      } else {
        float* const k = (ax == 1 ? row.ky : row.kz) + l;
#pragma unroll
        for (int i = 0; i < W; ++i)
          if ((unsigned)(l + i) < 16u) k[i] = f[i];
        if (ax == 1) {
          const int lz = ((q.packed >> 16) & 0xff) - 64;
          const int yb = max(l, 0) >> 2, ye = min(l + W - 1, 15) >> 2;
          const int zb = max(lz, 0) >> 2, ze = min(lz + W - 1, 15) >> 2;
          const uint32_t ym = (2u << ye) - (1u << yb);
          const uint32_t zs = 0x1111u & (0xffffu << (4 * zb)) & (0xffffu >> (4 * (3 - ze)));
          sm.mask[r] = ym * zs | (((uint32_t)q.packed >> 24) & 1u) << 16;
        }
      }
    }
    __syncthreads();
    // this warp's lists
    int n0[2] = {0, 0}, n1[2] = {0, 0};
    const unsigned below = (1u << lane) - 1u;
    unsigned char* const list = sm.list[2 * warp];
    for (int b = 0; b < n; b += 32) {
      const uint32_t m = b + lane < n ? sm.mask[b + lane] >> (2 * warp) : 0u;
      const bool second = (m >> (16 - 2 * warp)) & 1u;
      const unsigned sec = __ballot_sync(0xffffffffu, second), mine = second ? sec : ~sec;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const bool in = (m >> s) & 1u;
        const unsigned all = __ballot_sync(0xffffffffu, in);
        const int k = __popc(all & mine & below);
        const int at = second ? kNCh - 1 - n1[s] - k : n0[s] + k;
        if (in) list[s * kNCh + at] = (unsigned char)(b + lane);
        const int c = __popc(all & sec);
        n1[s] += c;
        n0[s] += __popc(all) - c;
      }
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int p = 2 * warp + s, tot = n0[s] + n1[s];
      // A rows g and g + 8: cells (z, y) and (z + 1, y)
      const int yc = 4 * (p & 3) + (g & 3), zc = 4 * (p >> 2) + 2 * (g >> 2);
      // shared addresses of this lane's pieces of row 0
      const unsigned row0 = (unsigned)__cvta_generic_to_shared(&sm.row[0]);
      const unsigned xrow = row0 + (unsigned)offsetof(PencilRow, xh) + (lane >> 4) * 16;
      const unsigned yrow = row0 + (unsigned)offsetof(PencilRow, ky) + 4 * yc;
      const unsigned zrow = row0 + (unsigned)offsetof(PencilRow, kz) + 4 * zc;
      for (int b = 0; b < tot; b += 16) {
        // list entry of this lane (lanes 0-15: entries 0-15 of the block, 16-31 the same again)
        const int at = b + (lane & 15);
        int rr = kNCh;
        if (at < tot) rr = list[s * kNCh + (at < n0[s] ? at : kNCh - 1 + n0[s] - at)];
        const unsigned ro = (unsigned)rr * (unsigned)sizeof(PencilRow);   // row offset
        uint32_t bh[4], bl[4];
        ldmatrix_x4_trans(bh, xrow + ro);
        ldmatrix_x4_trans(bl, xrow + ro + (unsigned)offsetof(PencilRow, xl));
        uint32_t ah[4], al[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {          // entries 2t, 2t + 1, then + 8
          const unsigned oa = __shfl_sync(0xffffffffu, ro, 2 * t + 8 * h);
          const unsigned ob = __shfl_sync(0xffffffffu, ro, 2 * t + 1 + 8 * h);
          const float ya = lds_f32(yrow + oa), yb = lds_f32(yrow + ob);
          const float2 va = mul_f32x2(make_float2(ya, ya), lds_f32x2(zrow + oa));
          const float2 vb = mul_f32x2(make_float2(yb, yb), lds_f32x2(zrow + ob));
          const float2 ha = make_float2(clear_low13(va.x), clear_low13(va.y));
          const float2 hb = make_float2(clear_low13(vb.x), clear_low13(vb.y));
          const float2 la = sub_f32x2(va, ha), lb = sub_f32x2(vb, hb);
          ah[2 * h] = pack_f16x2(ha.x, hb.x);
          ah[2 * h + 1] = pack_f16x2(ha.y, hb.y);
          al[2 * h] = pack_f16x2(la.x, lb.x);
          al[2 * h + 1] = pack_f16x2(la.y, lb.y);
        }
        auto products = [&](float (&c)[2][4], const uint32_t (&fh)[4], const uint32_t (&fl)[4]) {
          // (smallest terms first; the two x halves are independent chains).  The tensor cores
          // truncate each sum they return, which over a crowded tile's steps adds up to a bias (4e-6
          // for 225 coinciding records): a step starts from zero and is added rounded to nearest.
          float p[2][4];
          if constexpr (W >= 8) {
            mma_16816_first(p[0], fl, bl[0], bl[1]);
            mma_16816_first(p[1], fl, bl[2], bl[3]);
            mma_16816(p[0], fl, bh[0], bh[1]);
            mma_16816(p[1], fl, bh[2], bh[3]);
          } else {
            mma_16816_first(p[0], fl, bh[0], bh[1]);
            mma_16816_first(p[1], fl, bh[2], bh[3]);
          }
          mma_16816(p[0], fh, bl[0], bl[1]);
          mma_16816(p[1], fh, bl[2], bl[3]);
          mma_16816(p[0], fh, bh[0], bh[1]);
          mma_16816(p[1], fh, bh[2], bh[3]);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            c[0][q] += p[0][q];
            c[1][q] += p[1][q];
          }
        };
        if (b + 16 <= n0[s] || n1[s] == 0) {   // (warp-uniform)
          products(acc[s][0], ah, al);
        } else if (b >= n0[s]) {
          products(acc[s][1], ah, al);
        } else {                               // both: columns before entry n0 - b are the first's
          uint32_t fh[4], fl[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int e = n0[s] - b - (2 * t + 8 * (q >> 1));   // entries of this pair that are the first's
            const uint32_t m = e >= 2 ? 0xffffffffu : (e == 1 ? 0x0000ffffu : 0u);
            fh[q] = ah[q] & m;
            fl[q] = al[q] & m;
            ah[q] &= ~m;
            al[q] &= ~m;
          }
          products(acc[s][0], fh, fl);
          products(acc[s][1], ah, al);
        }
      }
    }
  }
  float2* const out = fine + (int64_t)keygrid * gstride;
  const int64_t nf0 = a.nf[0], nf1 = a.nf[1];
  const float sc = 1.0f / 1048576.0f;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int p = 2 * warp + s;
#pragma unroll
    for (int hv = 0; hv < 2; ++hv) {
      const int y = 4 * (p & 3) + (g & 3), z = 4 * (p >> 2) + 2 * (g >> 2) + hv;
      const int64_t row = ((int64_t)tz * 16 - z0 + z) * nf1 + (int64_t)ty * 16 + y;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
        *reinterpret_cast<float4*>(out + row * nf0 + (int64_t)tx * 16 + nt * 8 + 2 * t) =
            make_float4(acc[s][0][nt][2 * hv] * sc, acc[s][1][nt][2 * hv] * sc,
                        acc[s][0][nt][2 * hv + 1] * sc, acc[s][1][nt][2 * hv + 1] * sc);
    }
  }
}

template <int W>
int launch_w(const SpreadArgs& a, const RecF* recs, const float2* cv, const int* starts, int nkeys,
             float2* fine, cudaStream_t s, int64_t key0, int z0, int64_t gstride, bool repro) {
  if (const int rc = repro ? allow_smem(spread3_ordered_mma_kernel<W>, sizeof(MmaSmem<W>))
                           : allow_smem(spread3_pencil_mma_kernel<W>, sizeof(PencilSmem)))
    return rc;
  const EsPoly<W> p = es_poly_for<W>(a.beta);
  if (repro)
    spread3_ordered_mma_kernel<W><<<(unsigned)nkeys, 256, sizeof(MmaSmem<W>), s>>>(
        a, recs, cv, starts, fine, p, key0, z0, gstride);
  else
    spread3_pencil_mma_kernel<W><<<(unsigned)nkeys, 256, sizeof(PencilSmem), s>>>(
        a, recs, cv, starts, fine, p, key0, z0, gstride);
  MPSQ_LAUNCH_CHECK();
  return MPSQ_OK;
}

}  // namespace

bool spread_pair_mma_enabled() {
  static const bool on = [] {
    const char* e = getenv("MPSQ_SPREAD");
    return !(e && strcmp(e, "fma") == 0);
  }();
  return on;
}

int launch_spread_pair_mma(const SpreadArgs& a, const RecF* recs, const float2* cv, const int* starts,
                           int nkeys, float2* fine, cudaStream_t s, int64_t key0, int z0,
                           int64_t gstride, bool repro) {
  if (a.dim != 3 || a.tile[0] != 16 || a.tile[1] != 16 || a.tile[2] != 16)
    return fail(MPSQ_ERR_ARG, "spread mma: 16^3 tiles only");
  if ((reinterpret_cast<uintptr_t>(fine) & 15) != 0 || (a.nf[0] & 1) != 0)
    return fail(MPSQ_ERR_ARG, "spread mma: grid must be 16-byte aligned with even rows");
  if (gstride <= 0) {
    key0 = 0;
    z0 = 0;
    gstride = a.n_fine;
  }
  if (nkeys <= 0) return MPSQ_OK;
#define MPSQ_W(W) launch_w<W>(a, recs, cv, starts, nkeys, fine, s, key0, z0, gstride, repro)
  switch (a.w) {
    case 3: return MPSQ_W(3);
    case 4: return MPSQ_W(4);
    case 5: return MPSQ_W(5);
    case 6: return MPSQ_W(6);
    case 7: return MPSQ_W(7);
    case 8: return MPSQ_W(8);
#undef MPSQ_W
    default: return fail(MPSQ_ERR_ARG, "spread mma: kernel width %d not compiled", a.w);
  }
}

int launch_spread_plane_mma(const SpreadArgs& a, const RecF* recs, const float2* cv,
                            const int* starts, int nkeys, bool real_pair, float2* fine,
                            cudaStream_t s) {
  if (a.dim != 2 || a.tile[0] != kPT || a.tile[1] != kPT || (reinterpret_cast<uintptr_t>(fine) & 15) != 0)
    return fail(MPSQ_ERR_ARG, "plane spread: 32^2 tiles of a 16-byte aligned grid only");
  if (nkeys <= 0) return MPSQ_OK;
  const int rp = real_pair ? 1 : 0;
  switch (a.w) {
    case 3: return launch_plane_w<3>(a, recs, cv, starts, nkeys, rp, fine, s);
    case 4: return launch_plane_w<4>(a, recs, cv, starts, nkeys, rp, fine, s);
    case 5: return launch_plane_w<5>(a, recs, cv, starts, nkeys, rp, fine, s);
    case 6: return launch_plane_w<6>(a, recs, cv, starts, nkeys, rp, fine, s);
    case 7: return launch_plane_w<7>(a, recs, cv, starts, nkeys, rp, fine, s);
    case 8: return launch_plane_w<8>(a, recs, cv, starts, nkeys, rp, fine, s);
    default: return fail(MPSQ_ERR_ARG, "plane spread: kernel width %d not compiled", a.w);
  }
}

}  // namespace mpsq
