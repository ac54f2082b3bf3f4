// S(Q,omega) job pipeline: the frame loop of mp_sqom (code/src/mp_sqom56.f90:965-1165) on the
// GPU.  Per frame, one kernel selects atoms, computes their NUFFT phases and strengths and
// bins them (mp_sqom56.f90:1100-1143 fused into the binning), one kernel spreads all species
// grids, pruned line passes transform them, and the last of them (FP32) or one kernel more (FP64)
// deconvolves, separates packed species pairs, applies the species weights (:1338-1377, weight tables :901-936) and stores the weighted
// amplitude cs(t,Q) of the frame.
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "passes.h"

namespace mpsq {

// Parameters of the per-point preparation, passed by value.
struct PrepArgs {
  int dim;
  int n_species;
  int64_t species_offset[MPSQ_MAX_SPECIES + 1];
  int group_of[MPSQ_MAX_SPECIES];  // -1: species not transformed (mask 0)
  int comp_of[MPSQ_MAX_SPECIES];   // 0 real / 1 imaginary component in a packed pair
  int input_method;
  int phase_rounding;
  int use_range;
  int bulk_nsuper1;
  int n_row[3];
  double axis[3][3];
  float axis_f[3][3];
  double tpe[3];
  float tpe_f[3];
  double centre[3];
  float centre_f[3];
  double pos_min[3], pos_max[3];
  float pos_min_f[3], pos_max_f[3];
  float tol_f;
  int has_qc;
  double q_center[3];
  float tpq_f[3];  // 2 pi q_center in FP32 (reference rounding)
  int window;
  int pack;
  int64_t n_atoms_frame;
  // FP32 path: fine-grid coordinate g_k = sum_b A_kb r_b + B_k as hi+lo float pairs, and the
  // strength phase in turns q_center . r likewise
  float ahi[3][3], alo[3][3], bhi[3], blo[3];
  float qhi[3], qlo[3];
  float inv_nf[3];
  int nf[3];
  int diag;   // 1: A is diagonal (axis-aligned grid), g_k needs only r_k
};

}  // namespace mpsq

using namespace mpsq;

struct mpsq_job {
  mpsq_job_desc d{};
  cudaStream_t s = nullptr;
  EsKernel es{};
  GridGeom g{};
  SpreadArgs sa{};
  PrepArgs pa{};
  WeightArgs wa{};
  int ngroups = 0;
  float4* traj = nullptr;
  int4* at_ind = nullptr;
  void* fine = nullptr;
  int* counts = nullptr;
  int* starts = nullptr;
  // locality order of the atoms (rebuilt from the first frame of each multi-frame transform)
  int* perm = nullptr;
  int* perm_counts = nullptr;
  int* perm_starts = nullptr;
  bool perm_built = false;
  void* recs = nullptr;
  void* str = nullptr;
  int64_t cap = 0;
  void* corr[3] = {nullptr, nullptr, nullptr};   // within corr_mem
  void* corr_mem = nullptr;
  void* cs = nullptr;
  void* cs_species = nullptr;
  cufftHandle fft = 0;
  bool have_fft = false;
  // volumes on cuFFT: x transforms over every row, then (z, y) transforms of the kept x columns
  cufftHandle xfft[3] = {0, 0, 0};   // x rows; (z, y) of columns [0, h0]; of [n0 - h0, n0)
  int xfft_h0 = 0;
  bool have_xfft = false;
  // FP64 grids whose lengths have plans: pruned line transforms (x-pass output, plan tables)
  bool have_lines = false;
  GridLines lines;
  void* line_tables = nullptr;
  void* line_tmp = nullptr;
  int* err = nullptr;
  bool profile = false;
  cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  double stage_ms[4] = {0, 0, 0, 0};
  int64_t stage_frames = 0;
  // pruned fine-grid transform (FP32, 3D)
  bool pruned = false;
  float2* tw[3] = {nullptr, nullptr, nullptr};   // within tw_mem
  void* tw_mem = nullptr;
  float2* b1 = nullptr;
  int h[3] = {0, 0, 0}, K[3] = {1, 1, 1};
  // second frame lane (pruned FP32 path): its own stream and per-frame scratch, so that two
  // frames are in flight at once and their latency-bound kernels overlap
  bool lane2 = false;
  cudaStream_t s2 = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  void* fine2 = nullptr;
  int* counts2 = nullptr;
  int* starts2 = nullptr;
  void* recs2 = nullptr;
  void* str2 = nullptr;
  // per-atom preparation of the FP32 split path (counting pass -> scatter pass), per lane
  void* prep = nullptr;
  void* prep2 = nullptr;
  float2* b1_2 = nullptr;
  // frame batch (own-pass FP32 jobs whose frames are too small to fill the chip): one allocation
  // with the per-frame scratch of `batch` frames (1: none), whose frames run through every kernel
  // of the pipeline in one launch as further grids
  int batch = 1;
  void* batch_mem = nullptr;
  // one-phonon mode: displacement fields (n_species x 2 x n_row2 x n_row1, job precision)
  void* oneph_u = nullptr;
  float* oneph_base = nullptr;
  cufftHandle oneph_fft = 0;
  bool have_oneph_fft = false;
  std::mutex map_mu;                             // of the kept arrays of the map calls (MapMem)
  void* scratch[kScratchCount] = {};
  size_t scratch_bytes[kScratchCount] = {};
  void* main_mem = nullptr;   // traj .. err of every job, but for the large ones among them:
  std::vector<void*> large_mem;
  void* lane_mem = nullptr;   // the second lane's scratch
  int n_alloc = 0;  // device allocations made so far (fault injection below)
  // run-time choices (mpsq_job_set_option / mpsq_job_autotune)
  int opt_graph = 0;        // replay the frame loop of a transform call as a captured graph
  int opt_spread = 0;       // 0: tensor-core spreading of real pairs, 1: CUDA-core kernel
  int opt_xrows = 8;        // rows per CTA of the pruned X pass (4 or 8)
  int opt_zslab = 0;        // fine-grid planes per slab of the spread/X/Y pipeline (0: whole)
  int opt_repro = 0;        // 1: tensor-core spreading orders each tile's records by content
  int opt_lanes = 2;        // frame lanes used when a second lane exists (1 or 2)
  struct Graph {
    int32_t first, count;
    cudaGraphExec_t exec;
    int64_t launches;
  };
  std::vector<Graph> graphs;  // captured frame loops, by (first, count)
  // Q slab (q_slab > 0): the store holds kz planes [slab_z0, slab_z0 + slab_planes())
  int64_t slab_nz = 0;
  int64_t slab_z0 = 0;
  int64_t slab_planes() const { return slab_nz ? std::min(slab_nz, g.m[2] - slab_z0) : g.m[2]; }
  int64_t store_modes() const { return g.m[0] * g.m[1] * slab_planes(); }
};

// Device memory of a job: stream-ordered (from the device's memory pool, on the job's stream)
// when the job was created with stream_ordered != 0, plain otherwise.
// Host-side fault injection for tests of the error paths: with MPSQ_FAIL_ALLOC=k in the
// environment the k-th device allocation of every job reports cudaErrorMemoryAllocation
// without calling the allocator.
static bool injected_alloc_failure(mpsq_job* j) {
  const char* e = getenv("MPSQ_FAIL_ALLOC");
  return e && ++j->n_alloc == atoi(e);
}

// The library's own pool of a device (stream_ordered = 2): one-call jobs leave at most this much in it
// for the next call.  mpsq_release_memory gives it back, as does an allocation that would fail otherwise.
constexpr uint64_t kPoolKeeps = uint64_t(512) << 20;
constexpr int kPoolDevices = 64;
static std::mutex g_pool_mu;
static cudaMemPool_t g_pool[kPoolDevices] = {};
static cudaMemPool_t own_pool() {          // null where there is none to be had
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= kPoolDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_pool_mu);
  if (!g_pool[dev]) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    uint64_t keep = kPoolKeeps;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    g_pool[dev] = pool;
  }
  return g_pool[dev];
}
static bool release_pools() {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  bool any = false;
  for (cudaMemPool_t pool : g_pool)
    if (pool) any = cudaMemPoolTrimTo(pool, 0) == cudaSuccess || any;
  return any;
}
extern "C" int mpsq_release_memory(void) {
  release_pools();
  cudaGetLastError();
  return MPSQ_OK;
}

static cudaError_t job_alloc_once(const mpsq_job* j, void** ptr, size_t bytes) {
  if (!j->d.stream_ordered) return cudaMalloc(ptr, bytes);
  cudaMemPool_t pool = j->d.stream_ordered == 2 ? own_pool() : nullptr;
  return pool ? cudaMallocFromPoolAsync(ptr, bytes, pool, j->s) : cudaMallocAsync(ptr, bytes, j->s);
}
static cudaError_t job_alloc(mpsq_job* j, void** ptr, size_t bytes) {
  if (injected_alloc_failure(j)) {
    *ptr = nullptr;
    return cudaErrorMemoryAllocation;
  }
  bytes = std::max<size_t>(bytes, 16);
  cudaError_t e = job_alloc_once(j, ptr, bytes);
  if (e == cudaErrorMemoryAllocation && release_pools()) {
    cudaGetLastError();
    e = job_alloc_once(j, ptr, bytes);
  }
  return e;
}
static void job_release(mpsq_job* j, void* ptr) {
  if (!ptr) return;
  if (j->d.stream_ordered)
    cudaFreeAsync(ptr, j->s);
  else
    cudaFree(ptr);
}
// No kernel writes the per-species amplitudes of masked species: the store is cleared, on the job's
// stream, where it holds any (at creation, and when a slab of another height moves its rows).
static cudaError_t clear_masked_species(mpsq_job* j) {
  if (!j->cs_species) return cudaSuccess;
  bool masked = false;
  for (int s = 0; s < j->d.n_species; ++s) masked = masked || !j->d.mask[s];
  if (!masked) return cudaSuccess;
  const size_t value = j->d.precision == MPSQ_FP64 ? sizeof(double2) : sizeof(float2);
  return cudaMemsetAsync(j->cs_species, 0,
                         (size_t)j->d.n_frames * j->d.n_species * j->store_modes() * value, j->s);
}
// What the pool of a stream-ordered job holds but nothing uses: free for the job, though not by
// cudaMemGetInfo, which would let the jobs that ran before decide how this one runs.
static size_t idle_pool_bytes(const mpsq_job* j) {
  cudaMemPool_t pool = j->d.stream_ordered == 2 ? own_pool() : nullptr;
  int dev = 0;
  uint64_t reserved = 0, used = 0;
  if (!j->d.stream_ordered || cudaGetDevice(&dev) != cudaSuccess ||
      (!pool && cudaDeviceGetDefaultMemPool(&pool, dev) != cudaSuccess) ||
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
    return 0;
  return reserved > used ? (size_t)(reserved - used) : 0;
}
static cudaError_t job_upload(mpsq_job* j, void* dst, const void* src, size_t bytes) {
  // pageable source: the copy is staged before the call returns
  return j->d.stream_ordered ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, j->s)
                             : cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
}

namespace mpsq {

// Selection, phases and strengths of one atom of one frame (mp_sqom56.f90:1104-1142): false
// for an atom that is not transformed; otherwise its grid, pair component and strength and
// either its first support cell and offset (FP32 split path) or its folded fine-grid
// coordinate (FP64 and phase-rounding paths).
template <typename T>
struct PointPrep {
  int grid, comp;
  bool split;
  int sc[3];
  float dc[3];
  double g[3];
  typename Cplx<T>::type c;
};

template <typename T>
__device__ __forceinline__ bool prep_point(const float4* __restrict__ frame,
                                           const int4* __restrict__ at_ind, const PrepArgs& p,
                                           const SpreadArgs& a, int64_t j, PointPrep<T>& o) {
  int s = 0;
  while (s + 1 < p.n_species && j >= p.species_offset[s + 1]) ++s;
  if (j < p.species_offset[0] || j >= p.species_offset[p.n_species]) return false;
  const int grid = p.group_of[s];
  if (grid < 0) return false;
  const float4 r = frame[j];
  if (p.input_method == MPSQ_CELL) {
    if (r.x == 0.0f && r.y == 0.0f && r.z == 0.0f) return false;  // vacancy (:1107)
    if (p.use_range && at_ind) {
      const int4 ci = at_ind[j];
      const int c3[3] = {ci.x, ci.y, ci.z};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int c = c3[k] - p.n_row[k] / 2 - 1;
        if ((float)c < p.pos_min_f[k] || (float)c > p.pos_max_f[k]) return false;  // (:1109-1111)
      }
    }
  } else {
    const float rr[3] = {r.x, r.y, r.z};
#pragma unroll
    for (int k = 0; k < 3; ++k)  // (:1121-1128)
      if (!(rr[k] >= p.pos_min_f[k] - p.tol_f && rr[k] < p.pos_max_f[k] + p.tol_f)) return false;
  }
  if constexpr (sizeof(T) == 4) {
    if (!p.phase_rounding) {
      // FP32 split precision: exact phase reduction in two-float arithmetic (no FP64 pipe)
      const float rf[3] = {r.x, r.y, r.z};
      int* const sc = o.sc;
      float* const dc = o.dc;
      for (int k = 0; k < 3; ++k) {
        sc[k] = 0;
        dc[k] = 0.0f;
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {  // unrolled: sc, dc stay in registers
        if (k < p.dim) {
          // (the zero off-diagonal terms of an axis-aligned grid add exactly nothing)
          const F2 gk = p.diag ? affine1_f2(rf[k], p.ahi[k][k], p.alo[k][k], p.bhi[k], p.blo[k])
                               : affine_f2(rf, p.ahi[k], p.alo[k], p.bhi[k], p.blo[k]);
          split_cell_f2(gk, p.nf[k], p.inv_nf[k], a.w, &sc[k], &dc[k]);
        }
      }
      float2 c = make_float2(1.0f, 0.0f);
      if (p.has_qc) {
        const F2 t = affine_f2(rf, p.qhi, p.qlo, 0.0f, 0.0f);
        const float fl = floorf(t.hi);
        const float fr = __fadd_rn(__fsub_rn(t.hi, fl), t.lo);
        float sn, cn;
        sincospif(2.0f * fr, &sn, &cn);
        c = make_float2(cn, -sn);
      }
      if (p.window) {  // spatial Hann window (1+cos x)(1+cos y) (:1118)
        const int nw = p.dim == 2 ? 2 : 3;
        float f = 1.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (k >= nw) break;
          float pr = 0.0f;
#pragma unroll
          for (int b = 0; b < 3; ++b) pr = fmaf(p.axis_f[k][b], rf[b] - p.centre_f[b], pr);
          f *= 1.0f + cosf(pr * p.tpe_f[k]);
        }
        c.x *= f;
        c.y *= f;
      }
      o.comp = p.pack ? p.comp_of[s] : 0;
      if (p.pack && c.x == 0.0f) return false;
      o.grid = grid;
      o.split = true;
      o.c.x = (T)c.x;
      o.c.y = (T)c.y;
      return true;
    }
  }
  double x[3] = {0.0, 0.0, 0.0};
  double g[3] = {0.0, 0.0, 0.0};
  const double rd[3] = {(double)r.x, (double)r.y, (double)r.z};
  const float rf[3] = {r.x, r.y, r.z};
  for (int k = 0; k < p.dim; ++k) {
    if (p.phase_rounding) {
      // FP32 dot product and FP32 scale as the reference computes xf, yf (:1115-1116)
      float pr = 0.0f;
      for (int b = 0; b < 3; ++b) pr = __fadd_rn(pr, __fmul_rn(p.axis_f[k][b], __fsub_rn(rf[b], p.centre_f[b])));
      x[k] = (double)__fmul_rn(pr, p.tpe_f[k]);
    } else {
      double pr = 0.0;
      for (int b = 0; b < 3; ++b) pr += p.axis[k][b] * (rd[b] - p.centre[b]);
      x[k] = pr * p.tpe[k];
    }
    g[k] = fold_grid(x[k] * a.gscale[k], (double)a.nf[k], a.ginv[k]);
  }
  typename Cplx<T>::type c;
  if (p.has_qc) {
    if (p.phase_rounding) {
      float arg = 0.0f;
      for (int b = 0; b < 3; ++b) arg = __fadd_rn(arg, __fmul_rn(p.tpq_f[b], rf[b]));
      // the argument carries the reference's FP32 rounding; the exponential itself is
      // evaluated in the job's precision
      if (sizeof(T) == 8) {
        double sn, cn;
        sincos((double)arg, &sn, &cn);
        c.x = (T)cn;
        c.y = (T)(-sn);
      } else {
        float sn, cn;
        sincosf(arg, &sn, &cn);
        c.x = (T)cn;
        c.y = (T)(-sn);
      }
    } else {
      double turns = 0.0;
      for (int b = 0; b < 3; ++b) turns += p.q_center[b] * rd[b];
      turns -= floor(turns);
      if (sizeof(T) == 8) {
        double sn, cn;
        sincospi(2.0 * turns, &sn, &cn);
        c.x = (T)cn;
        c.y = (T)(-sn);
      } else {
        float sn, cn;
        sincospif((float)(2.0 * turns), &sn, &cn);
        c.x = (T)cn;
        c.y = (T)(-sn);
      }
    }
  } else {
    c.x = (T)1;
    c.y = (T)0;
  }
  if (p.window) {  // spatial Hann window (1+cos x)(1+cos y) (:1118)
    const int nw = p.dim == 2 ? 2 : 3;
    T f = (T)1;
    for (int k = 0; k < nw; ++k) f *= (T)1 + (T)cos(x[k]);
    c.x *= f;
    c.y *= f;
  }
  o.comp = p.pack ? p.comp_of[s] : 0;
  if (p.pack && c.x == (T)0) return false;  // zero strength contributes nothing
  o.grid = grid;
  o.split = false;
  o.c = c;
  for (int k = 0; k < 3; ++k) o.g[k] = g[k];
  return true;
}

// Binning of one frame.  Pass 0 (kScatter false) counts, pass 1 scatters; str == nullptr:
// unit strengths (no centre phase, no window), which are not stored.  Thread i takes atom
// perm[i] (a locality order, so that a warp's atoms share tiles and its cursor atomics
// combine) or atom i without a permutation.  blockIdx.y is the frame of a batch: consecutive
// frames of the trajectory, each binned under a set of a.ngrid grids of its own.
template <typename T, bool kScatter>
__global__ void job_bin_kernel(const float4* __restrict__ frame, const int4* __restrict__ at_ind,
                               const int* __restrict__ perm, PrepArgs p, SpreadArgs a,
                               int* cursor, const int* __restrict__ starts,
                               typename RecOf<T>::type* recs, typename Cplx<T>::type* str,
                               int64_t cap, int* err) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n_atoms_frame) return;
  const int64_t j = perm ? perm[i] : i;
  frame += (int64_t)blockIdx.y * p.n_atoms_frame;
  PointPrep<T> q;
  if (!prep_point<T>(frame, at_ind, p, a, j, q)) return;
  q.grid += (int)blockIdx.y * a.ngrid;
  if constexpr (sizeof(T) == 4) {
    if (q.split) {
      const float2 c = make_float2(q.c.x, q.c.y);
      emit_cells<float>(a, q.sc, q.dc, q.grid, q.comp, kScatter, cursor, starts, (RecF*)recs,
                        (float2*)str, c, nullptr, 0, cap, err);
      return;
    }
  }
  emit_records<T>(a, q.g, q.grid, q.comp, kScatter, cursor, starts, recs, str, q.c, nullptr, 0,
                  cap, err);
}

// FP32 split path in two passes that prepare each atom once.  Pass 0 runs the selection, the
// exact two-float cell split and the strength, keeps the result per atom (in locality order:
// coalesced) and counts the atom's records per tile; pass 1 reads it back and writes the
// records.  Per atom: int4 {s0 | s1 << 16, s2 | grid << 16 | comp << 24, d0, d1} (y = -1: not
// transformed), d2, and the strength when strengths are not all 1.
struct PrepCache {
  int4* cell;
  float* d2;
  float2* c;   // null: unit strengths
};

__device__ __forceinline__ int low16_signed(int v) { return (v & 0xffff) - ((v & 0x8000) << 1); }

__global__ void job_bin_count_split_kernel(const float4* __restrict__ frame,
                                           const int4* __restrict__ at_ind,
                                           const int* __restrict__ perm, PrepArgs p, SpreadArgs a,
                                           int* cursor, PrepCache pc, int* err) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n_atoms_frame) return;
  const int64_t j = perm ? perm[i] : i;
  const int64_t fr = blockIdx.y, e = fr * p.n_atoms_frame + i;   // frame of the batch, cache slot
  PointPrep<float> q;
  if (!prep_point<float>(frame + fr * p.n_atoms_frame, at_ind, p, a, j, q) || !q.split) {
    pc.cell[e] = make_int4(0, -1, 0, 0);
    return;
  }
  pc.cell[e] = make_int4((int)(((unsigned)q.sc[0] & 0xffffu) | ((unsigned)q.sc[1] << 16)),
                         (int)(((unsigned)q.sc[2] & 0xffffu) | ((unsigned)q.grid << 16) |
                               ((unsigned)q.comp << 24)),
                         __float_as_int(q.dc[0]), __float_as_int(q.dc[1]));
  pc.d2[e] = q.dc[2];
  if (pc.c) pc.c[e] = make_float2(q.c.x, q.c.y);
  emit_cells<float>(a, q.sc, q.dc, q.grid + (int)fr * a.ngrid, q.comp, false, cursor, nullptr, nullptr, nullptr,
                    make_float2(0.f, 0.f), nullptr, 0, 0, err);
}

__global__ void job_bin_scatter_split_kernel(int64_t n, PrepCache pc, SpreadArgs a, int* cursor,
                                             const int* __restrict__ starts,
                                             RecF* __restrict__ recs, float2* __restrict__ str,
                                             int64_t cap, int* err) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t fr = blockIdx.y, e = fr * n + i;
  const int4 r = __ldcs(pc.cell + e);
  if (r.y == -1) return;
  const int sc[3] = {low16_signed(r.x), r.x >> 16, low16_signed(r.y)};
  const float dc[3] = {__int_as_float(r.z), __int_as_float(r.w), __ldcs(pc.d2 + e)};
  const float2 c = pc.c ? __ldcs(pc.c + e) : make_float2(1.f, 0.f);
  emit_cells<float>(a, sc, dc, ((r.y >> 16) & 0xff) + (int)fr * a.ngrid, (r.y >> 24) & 0x7f, true, cursor, starts,
                    recs, str, c, nullptr, 0, cap, err);
}

// Locality order of the atoms of one frame: a counting sort by the tile of each atom's first
// support cell (atoms that are not transformed go to a last bucket, key nkeys).  Pass 0
// counts, pass 1 writes perm[starts[key] + slot] = atom.
template <typename T, bool kScatter>
__global__ void job_perm_kernel(const float4* __restrict__ frame, const int4* __restrict__ at_ind,
                                PrepArgs p, SpreadArgs a, int64_t nkeys, int* cursor,
                                const int* __restrict__ starts, int* __restrict__ perm) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= p.n_atoms_frame) return;
  PointPrep<T> q;
  int64_t key = nkeys;
  if (prep_point<T>(frame, at_ind, p, a, j, q)) {
    int t[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (k < a.dim) {
        const int c = q.split ? q.sc[k] : (int)ceil(q.g[k] - 0.5 * a.w);
        int tk = c >> a.tshift[k];
        tk = tk < 0 ? tk + a.ntile[k] : (tk >= a.ntile[k] ? tk - a.ntile[k] : tk);
        t[k] = tk;
      }
    }
    key = (int64_t)q.grid * a.n_tiles + ((int64_t)t[2] * a.ntile[1] + t[1]) * a.ntile[0] + t[0];
  }
  // one atomic per key of a warp (a crystal's atoms come in site order, so a warp's 32 atoms
  // share a few keys; on a plane of 300 tiles one atomic per atom took 60 us per pass)
  const unsigned peers = __match_any_sync(__activemask(), (int)key);
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(&cursor[key], __popc(peers));
  if constexpr (kScatter) {
    base = __shfl_sync(peers, base, leader);
    perm[starts[key] + base + __popc(peers & ((1u << lane) - 1u))] = (int)j;
  }
}

// Deconvolution, pair separation, species weighting; writes cs(t, Q) for one frame.
// Grid: x over the m0 modes of a row, y over the m1 rows, z over the nz planes z0.. of the
// store's Q slab (the whole grid: z0 = 0, nz = m2; 32-bit index math) of each frame of a batch.
// kept: `fine` holds the kept frequencies of the line transforms (K2, K1, K0 per grid) instead of
// the whole transformed grids; grid `real` of a frame keeps x frequencies [0, h] only (K0 = h + 1).
struct KeptLayout {
  int on, K0, K1, h[3], real;
};
template <typename T>
__global__ void job_deconv_kernel(SpreadArgs a, KeptLayout kept, int m0, int m1, int m2, int z0, int nz,
                                  const typename Cplx<T>::type* __restrict__ fine,
                                  const T* __restrict__ c0, const T* __restrict__ c1,
                                  const T* __restrict__ c2, WeightArgs w,
                                  typename Cplx<T>::type* __restrict__ cs_frame,
                                  typename Cplx<T>::type* __restrict__ cs_species_frame) {
  using C = typename Cplx<T>::type;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m0) return;
  const int fr = (int)blockIdx.z / nz, lz = (int)blockIdx.z - fr * nz;   // frame, plane of the slab
  const int j = blockIdx.y, l = z0 + lz;
  const int row = lz * m1 + j;                            // row of the store
  const int64_t nm = (int64_t)m0 * m1 * nz;
  fine += (int64_t)fr * w.ngroups * a.n_fine;
  cs_frame += fr * nm;
  cs_species_frame += fr * (nm * w.n_species);            // (null unless species are stored)
  const int64_t q = (int64_t)row * m0 + i;
  const int kx = i - m0 / 2, ky = j - m1 / 2, kz = l - m2 / 2;
  const int nf0 = (int)a.nf[0], nf1 = (int)a.nf[1], nf2 = (int)a.nf[2];
  // fine-grid positions of mode k and of -k (periodic)
  const int sx = kx < 0 ? kx + nf0 : kx, sy = ky < 0 ? ky + nf1 : ky, sz = kz < 0 ? kz + nf2 : kz;
  const int mx = kx > 0 ? nf0 - kx : -kx, my = ky > 0 ? nf1 - ky : -ky, mz = kz > 0 ? nf2 - kz : -kz;
  const int64_t src = kept.on ? ((int64_t)(kz + kept.h[2]) * kept.K1 + ky + kept.h[1]) * kept.K0 + kx + kept.h[0]
                              : ((int64_t)sz * nf1 + sy) * nf0 + sx;
  const int64_t srcm = kept.on ? ((int64_t)(kept.h[2] - kz) * kept.K1 + kept.h[1] - ky) * kept.K0 + kept.h[0] - kx
                               : ((int64_t)mz * nf1 + my) * nf0 + mx;
  const T corr = c0[i] * c1[j] * c2[l];
  T s2 = 0;
  if (w.weight_mode == MPSQ_WEIGHT_XRAY) {
    T qv[3];
    for (int b = 0; b < 3; ++b)
      qv[b] = WP<T>::q0(w, b) + (T)kx * WP<T>::qs(w, 0, b) + (T)ky * WP<T>::qs(w, 1, b) +
              (T)kz * WP<T>::qs(w, 2, b);
    s2 = WP<T>::kappa(w) * (qv[0] * qv[0] + qv[1] * qv[1] + qv[2] * qv[2] + WP<T>::extra(w));
  }
  T accr = 0, acci = 0;
  for (int gi = 0; gi < w.ngroups; ++gi) {
    C G = fine[gi * a.n_fine + src];
    if (w.pair[gi]) {
      const C Gm = fine[gi * a.n_fine + srcm];
      const int sa = w.sp_a[gi], sb = w.sp_b[gi];
      const T wa = (T)0.5 * species_weight<T>(w, sa, s2), wb = (T)0.5 * species_weight<T>(w, sb, s2);
      // (the deconvolution factor is common to all grids and multiplies their weighted sum below)
      accr += wa * (G.x + Gm.x) + wb * (G.y + Gm.y);
      acci += wa * (G.y - Gm.y) - wb * (G.x - Gm.x);
      if (w.store_species) {
        const T ar = (T)0.5 * (G.x + Gm.x) * corr, ai = (T)0.5 * (G.y - Gm.y) * corr;
        const T br = (T)0.5 * (G.y + Gm.y) * corr, bi = (T)(-0.5) * (G.x - Gm.x) * corr;
        C va, vb;
        va.x = ar * WP<T>::wnorm(w);
        va.y = ai * WP<T>::wnorm(w);
        vb.x = br * WP<T>::wnorm(w);
        vb.y = bi * WP<T>::wnorm(w);
        cs_species_frame[(int64_t)sa * nm + q] = va;
        cs_species_frame[(int64_t)sb * nm + q] = vb;
      }
    } else {
      const int sa = w.sp_a[gi];
      const T wa = species_weight<T>(w, sa, s2);
      if (kept.on && gi == kept.real) {
        const int sg = kx < 0 ? -1 : 1;      // the conjugate of the mirror frequency for kx < 0
        G = fine[gi * a.n_fine + ((int64_t)(kept.h[2] + sg * kz) * kept.K1 + kept.h[1] + sg * ky) * (kept.h[0] + 1) + sg * kx];
        if (kx < 0) G.y = -G.y;
      }
      accr += wa * G.x;
      acci += wa * G.y;
      if (w.store_species) {
        C va;
        va.x = G.x * corr * WP<T>::wnorm(w);
        va.y = G.y * corr * WP<T>::wnorm(w);
        cs_species_frame[(int64_t)sa * nm + q] = va;
      }
    }
  }
  const T f = corr * WP<T>::wnorm(w);
  C out;
  out.x = accr * f;
  out.y = acci * f;
  cs_frame[q] = out;
}

// -------------------------------------------------------------------- one-phonon mode
// mp_sqom's j_oneph = 1 branch (code/src/mp_sqom56.f90:1037-1098): per species, the in-plane
// displacements of the atoms are summed over the cell columns of the plane into two real
// fields u_x(k, l), u_y(k, l) on the n_row x n_row cell grid, Fourier transformed (forward,
// exp(-i), unscaled) and divided by n_row, and every Q pixel of the n_bz x n_bz zones takes
// A_j(Q) = exp(-2 pi i q . b_j) (q_x u_qx + q_y u_qy) at the zone-folded cell frequency.
// Plane 1 is (hk0): k, l = cell indices 1, 2, d = r - b - cell + n_row/2.  Plane 2 is (hhl):
// k = mod(c1 - 1 + c2 - 1, n_row) + 1, l = c3, d_x = (d1 + d2 + 2)/sqrt 2, d_y = d3 + 1
// (the reference's "+1" on this plane kept).  Displacements in FP32 in the reference's order.

// u: [n_species][2][n2][n1] complex, zeroed; atoms at exactly (0,0,0) are vacancies (:1049).
template <typename T>
__global__ void oneph_scatter_kernel(const float4* __restrict__ frame, const int4* __restrict__ at_ind,
                                     PrepArgs p, int plane, const float* __restrict__ base,
                                     int n1, int n2, typename Cplx<T>::type* __restrict__ u) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= p.n_atoms_frame) return;
  if (j < p.species_offset[0] || j >= p.species_offset[p.n_species]) return;
  int s = 0;
  while (s + 1 < p.n_species && j >= p.species_offset[s + 1]) ++s;
  if (p.group_of[s] < 0) return;  // masked species are not transformed
  const float4 r = frame[j];
  if (r.x == 0.0f && r.y == 0.0f && r.z == 0.0f) return;
  const int4 c = at_ind[j];
  const float b0 = base[3 * s], b1 = base[3 * s + 1], b2 = base[3 * s + 2];
  int k, l;
  float dx, dy;
  if (plane == 1) {
    k = c.x;
    l = c.y;
    dx = __fadd_rn(__fsub_rn(__fsub_rn(r.x, b0), (float)c.x), (float)(p.n_row[0] / 2));
    dy = __fadd_rn(__fsub_rn(__fsub_rn(r.y, b1), (float)c.y), (float)(p.n_row[1] / 2));
  } else {
    const int per = (p.n_row[0] + p.n_row[1]) / 2;
    k = ((c.x - 1 + c.y - 1) % per + per) % per + 1;
    l = c.z;
    float t = __fadd_rn(__fadd_rn(__fsub_rn(__fsub_rn(r.x, b0), (float)c.x), (float)(p.n_row[0] / 2)), 1.0f);
    t = __fadd_rn(__fadd_rn(__fsub_rn(__fsub_rn(__fadd_rn(t, r.y), b1), (float)c.y), (float)(p.n_row[1] / 2)), 1.0f);
    dx = __fdiv_rn(t, sqrtf(2.0f));
    dy = __fadd_rn(__fadd_rn(__fsub_rn(__fsub_rn(r.z, b2), (float)c.z), (float)(p.n_row[2] / 2)), 1.0f);
  }
  if (k < 1 || k > n1 || l < 1 || l > n2) return;  // outside the cell grid
  const int64_t cell = (int64_t)(l - 1) * n1 + (k - 1);
  const int64_t plane_sz = (int64_t)n1 * n2;
  atomicAdd(&u[(2 * (int64_t)s) * plane_sz + cell].x, (T)dx);
  atomicAdd(&u[(2 * (int64_t)s + 1) * plane_sz + cell].x, (T)dy);
}

// One thread per Q pixel (i, j) of the m0 x m1 plane; pixels beyond the n_bz zones (which the
// reference never writes) are zero.  Species weights, mask and window norm as the NUFFT path.
template <typename T>
__global__ void oneph_expand_kernel(const typename Cplx<T>::type* __restrict__ u, PrepArgs p,
                                    int plane, const float* __restrict__ base, int n1, int n2,
                                    int m0, int m1, int n_bz, float qx_min, float qy_min,
                                    int nqx_min, int nqy_min, WeightArgs w,
                                    typename Cplx<T>::type* __restrict__ cs_frame,
                                    typename Cplx<T>::type* __restrict__ cs_species_frame) {
  using C = typename Cplx<T>::type;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int jq = blockIdx.y;
  if (i >= m0) return;
  const int64_t q = (int64_t)jq * m0 + i;
  const int64_t nm = (int64_t)m0 * m1;
  const int ii = i / n1, jj = jq / n2;
  const bool inside = ii < n_bz && jj < n_bz;
  const int k = i - ii * n1 + 1, l = jq - jj * n2 + 1;
  // q_x = qx_min + (ii - 1) + (k - 1) / n_row in FP32 (1-based ii there)
  const float qx = __fadd_rn(__fadd_rn(qx_min, (float)ii), __fdiv_rn((float)(k - 1), (float)n1));
  const float qy = __fadd_rn(__fadd_rn(qy_min, (float)jj), __fdiv_rn((float)(l - 1), (float)n2));
  int kk = (nqx_min + k) % n1, ll = (nqy_min + l) % n2;
  if (kk == 0) kk = n1;
  if (ll == 0) ll = n2;
  const int64_t cell = (int64_t)(ll - 1) * n1 + (kk - 1);
  const int64_t plane_sz = (int64_t)n1 * n2;
  T s2 = 0;
  if (w.weight_mode == MPSQ_WEIGHT_XRAY) {
    const int kx = i - m0 / 2, ky = jq - m1 / 2;
    T qv[3];
    for (int b = 0; b < 3; ++b)
      qv[b] = WP<T>::q0(w, b) + (T)kx * WP<T>::qs(w, 0, b) + (T)ky * WP<T>::qs(w, 1, b);
    s2 = WP<T>::kappa(w) * (qv[0] * qv[0] + qv[1] * qv[1] + qv[2] * qv[2] + WP<T>::extra(w));
  }
  const float tpi = 6.28318530717958647692f;
  T accr = 0, acci = 0;
  for (int s = 0; s < p.n_species; ++s) {
    if (p.group_of[s] < 0) continue;
    C a;
    a.x = (T)0;
    a.y = (T)0;
    if (inside) {
      const C ux = u[(2 * (int64_t)s) * plane_sz + cell];
      const C uy = u[(2 * (int64_t)s + 1) * plane_sz + cell];
      const T fx = (T)qx / (T)n1, fy = (T)qy / (T)n2;
      const T vr = fx * ux.x + fy * uy.x, vi = fx * ux.y + fy * uy.y;
      const float b0 = base[3 * s], b1 = base[3 * s + 1], b2 = base[3 * s + 2];
      const float dot = plane == 1 ? __fadd_rn(__fmul_rn(qx, b0), __fmul_rn(qy, b1))
                                   : __fadd_rn(__fmul_rn(qx, __fadd_rn(b0, b1)), __fmul_rn(qy, b2));
      const float arg = __fmul_rn(tpi, dot);
      T sn, cn;
      if constexpr (sizeof(T) == 8) {
        sincos((double)arg, &sn, &cn);
      } else {
        sincosf(arg, &sn, &cn);
      }
      a.x = cn * vr + sn * vi;      // (cos - i sin)(vr + i vi)
      a.y = cn * vi - sn * vr;
    }
    const T ws = species_weight<T>(w, s, s2);
    accr += ws * a.x;
    acci += ws * a.y;
    if (w.store_species) {
      C v;
      v.x = a.x * WP<T>::wnorm(w);
      v.y = a.y * WP<T>::wnorm(w);
      cs_species_frame[(int64_t)s * nm + q] = v;
    }
  }
  C out;
  out.x = accr * WP<T>::wnorm(w);
  out.y = acci * WP<T>::wnorm(w);
  cs_frame[q] = out;
}

static size_t csize(int prec) { return prec == MPSQ_FP64 ? sizeof(double2) : sizeof(float2); }
static size_t rsize(int prec) { return prec == MPSQ_FP64 ? sizeof(RecD) : sizeof(RecF); }

static int job_layout(const mpsq_job_desc* d, EsKernel* es, GridGeom* g, int* ngroups,
                      int group_of[], int comp_of[], int pair[], int sp_a[], int sp_b[],
                      int* pack) {
  if (d->ndim != 2 && d->ndim != 3) return fail(MPSQ_ERR_ARG, "job: ndim must be 2 or 3");
  if (d->precision != MPSQ_FP32 && d->precision != MPSQ_FP64)
    return fail(MPSQ_ERR_ARG, "job: bad precision");
  if (d->n_species < 1 || d->n_species > MPSQ_MAX_SPECIES)
    return fail(MPSQ_ERR_ARG, "job: n_species must be in 1..%d", MPSQ_MAX_SPECIES);
  if (d->n_frames < 1) return fail(MPSQ_ERR_ARG, "job: n_frames must be >= 1");
  if (d->n_atoms_frame < 1) return fail(MPSQ_ERR_ARG, "job: n_atoms_frame must be >= 1");
  if (d->species_offset[0] < 0 || d->species_offset[d->n_species] > d->n_atoms_frame)
    return fail(MPSQ_ERR_ARG, "job: species offsets outside the frame");
  for (int s = 0; s < d->n_species; ++s)
    if (d->species_offset[s + 1] < d->species_offset[s])
      return fail(MPSQ_ERR_ARG, "job: species offsets not increasing");
  if (d->weight_mode < 1 || d->weight_mode > 3) return fail(MPSQ_ERR_ARG, "job: bad weight_mode");
  if (d->q_slab < 0 || (d->q_slab > 0 && d->ndim != 3))
    return fail(MPSQ_ERR_ARG, "job: q_slab must be 0, or > 0 for a 3D job");
  *es = es_params(d->eps, d->precision);
  int rc = make_geom(d->ndim, d->n_modes, es->w, g);
  if (rc) return rc;
  if (d->precision == MPSQ_FP32 && !d->no_pruned_fft) {
    // FP32 volumes: fine lengths from the compiled pruned transforms (the smallest at or above
    // the 2,3,5-smooth length; an upsampling above 2 only lowers the kernel's error), so that
    // every grid up to 1600 points per axis takes the pruned passes instead of cuFFT.  Planes keep
    // their lengths: the plane passes are compiled for every one of them up to 1600.
    for (int k = 0; k < 3 && d->ndim == 3; ++k) {
      const int64_t n = compiled_fft_size_at_least(g->nf[k]);
      if (n > 0) {
        g->nf[k] = n;
        g->ntile[k] = (int)(n / g->tile[k]);
      }
    }
    g->n_tiles = (int64_t)g->ntile[0] * g->ntile[1] * g->ntile[2];
    g->n_fine = g->nf[0] * g->nf[1] * g->nf[2];
  }
  const bool qc0 = d->q_center[0] == 0.0 && d->q_center[1] == 0.0 && d->q_center[2] == 0.0;
  *pack = (qc0 && !d->no_pack) ? 1 : 0;
  int n = 0;
  int open = -1;  // group with a free imaginary slot
  for (int s = 0; s < d->n_species; ++s) {
    group_of[s] = -1;
    comp_of[s] = 0;
    if (!d->mask[s]) continue;
    if (*pack && open >= 0) {
      group_of[s] = open;
      comp_of[s] = 1;
      pair[open] = 1;
      sp_b[open] = s;
      open = -1;
    } else {
      group_of[s] = n;
      pair[n] = 0;
      sp_a[n] = s;
      sp_b[n] = s;
      if (*pack) open = n;
      ++n;
    }
  }
  *ngroups = n;
  return MPSQ_OK;
}

}  // namespace mpsq

// ================================================================================ C ABI
static void job_free(mpsq_job* j) {
  if (!j) return;
  if (j->have_fft) cufftDestroy(j->fft);
  if (j->have_xfft)
    for (auto h : j->xfft)
      if (h) cufftDestroy(h);
  job_release(j, j->main_mem);
  for (void* p : j->large_mem) job_release(j, p);
  job_release(j, j->at_ind);
  job_release(j, j->corr_mem);
  for (void* p : j->scratch) job_release(j, p);
  job_release(j, j->b1);
  job_release(j, j->tw_mem);
  job_release(j, j->lane_mem);
  job_release(j, j->batch_mem);
  job_release(j, j->line_tables);
  job_release(j, j->line_tmp);
  if (j->have_oneph_fft) cufftDestroy(j->oneph_fft);
  job_release(j, j->oneph_u);
  job_release(j, j->oneph_base);
  for (auto& gr : j->graphs) cudaGraphExecDestroy(gr.exec);
  if (j->fork) cudaEventDestroy(j->fork);
  if (j->join) cudaEventDestroy(j->join);
  if (j->s2) cudaStreamDestroy(j->s2);
  for (auto& e : j->ev)
    if (e) cudaEventDestroy(e);
  delete j;
}

// Bytes of the per-atom preparation cache of the FP32 split path (0: not used): cell words
// (16 B) and d2 (4 B) per atom, plus the strength (8 B, at offset 24 n) unless all are 1.
static size_t prep_cache_bytes(int precision, int phase_rounding, bool unit_str, int64_t n) {
  if (precision != MPSQ_FP32 || phase_rounding || n <= 0) return 0;
  return (size_t)n * (unit_str ? 20 : 32);
}
static size_t prep_cache_bytes(const mpsq_job* j) {
  return prep_cache_bytes(j->d.precision, j->pa.phase_rounding, !j->pa.has_qc && !j->pa.window,
                          j->d.n_atoms_frame);
}

// Whether the fine grids are transformed by the pruned passes (FP32, compiled lengths).
static bool takes_pruned_passes(const mpsq_job_desc* d, const GridGeom& g) {
  bool pruned = d->precision == MPSQ_FP32 && !d->no_pruned_fft;
  for (int k = 0; k < d->ndim && pruned; ++k)
    pruned = fft_size_compiled((int)g.nf[k]) || (d->ndim == 2 && fft_plane_size_compiled((int)g.nf[k]));
  return pruned;
}

// Whether FP64 grids take the pruned line transforms (no_pruned_fft keeps cuFFT).
static bool takes_lines(const mpsq_job_desc* d, const GridGeom& g) {
  return d->precision == MPSQ_FP64 && !d->no_pruned_fft && grid_lines_ok(g, d->precision);
}

// The largest array that a plain job's map calls keep in a slot: a map of its store and a 1/|Q| table of
// up to 64 MB (and of 1 MB at least, for cuts), small windows, paths.
static size_t scratch_cap(const mpsq_job_desc& d, const GridGeom& g, JobScratch slot) {
  if (slot == kScratchWindow) return size_t(64) << 10;
  if (slot == kScratchPath) return size_t(1) << 20;
  const int64_t planes = d.q_slab > 0 ? std::min<int64_t>(d.q_slab, g.m[2]) : g.m[2];
  return (size_t)std::min<int64_t>(std::max<int64_t>(g.m[0] * g.m[1] * planes * 4, 1 << 20), 64 << 20);
}

// Record slots of a frame: every selected atom's halo copies.
static int64_t records_cap(const mpsq_job_desc* d) {
  return std::max<int64_t>(1, (d->species_offset[d->n_species] - d->species_offset[0]) * (d->ndim == 3 ? 8 : 4));
}

// Scratch of a frame batch, carved from one allocation: every array holds `frames` frames, laid
// out as if each frame had a set of grids of its own.
struct BatchScratch {
  void* fine;
  void* b1;       // x-pass output
  int* counts;
  int* starts;
  void* recs;
  void* str;
  void* prep;
  size_t bytes;
};
static BatchScratch carve_batch(const mpsq_job_desc* d, const GridGeom& g, int ngrid, bool unit_str, int frames,
                                void* mem) {
  const int64_t ng = (int64_t)ngrid * frames, nkeys = ng * g.n_tiles, cap = records_cap(d);
  BatchScratch b{};
  char* const base = static_cast<char*>(mem);
  auto take = [&](size_t bytes) {
    void* p = base ? base + b.bytes : nullptr;
    b.bytes += (bytes + 255) & ~size_t(255);
    return p;
  };
  const size_t cs = csize(d->precision);
  b.fine = take((size_t)ng * g.n_fine * cs);
  b.b1 = take((size_t)ng * g.nf[2] * g.nf[1] * (2 * (g.m[0] / 2) + 1) * cs);   // kept x frequencies
  b.counts = (int*)take(sizeof(int) * (nkeys + 1));
  b.starts = (int*)take(sizeof(int) * (nkeys + 1));
  b.recs = take((size_t)frames * cap * rsize(d->precision));
  b.str = take(unit_str ? 0 : (size_t)frames * cap * cs);
  b.prep = take((size_t)frames * prep_cache_bytes(d->precision, d->phase_rounding, unit_str, d->n_atoms_frame));
  return b;
}
static BatchScratch carve_batch(const mpsq_job* j, int frames, void* mem) {
  return carve_batch(&j->d, j->g, j->sa.ngrid, !j->pa.has_qc && !j->pa.window, frames, mem);
}

// Frames per batch, at most (1: no batches).  A frame of a Q plane or of a small volume gives each kernel
// a few hundred CTAs or fewer, so a launch costs its latency and not its work; frames are batched while
// their scratch stays within 192 MB together, up to 32.  Measured with the tensor-core plane spreading, 32
// frames of 163,840 atoms onto 160^2 modes: 5.09 -> 0.71 ms (230 launches -> 24).  From 48 MB per frame on
// (fewer than four frames) a frame fills the chip and two lanes overlap what is left.
static int most_batch_frames(const mpsq_job_desc* d, const GridGeom& g, int ngrid, bool unit_str) {
  if (d->no_frame_batch || d->n_frames < 2 || !(takes_pruned_passes(d, g) || takes_lines(d, g))) return 1;
  const size_t n = (size_t(192) << 20) / carve_batch(d, g, ngrid, unit_str, 1, nullptr).bytes;
  return n < 4 ? 1 : (int)std::min<int64_t>({(int64_t)n, 32, (int64_t)INT32_MAX / records_cap(d)});
}

// The batch of a job, in parts as equal as its frames allow.  mpsq_job_estimate_bytes counts it; on a
// device that is nearly full all the same (below 16 times the batch free, the job's pool included) the
// frames run one at a time.
static void make_batch(mpsq_job* j) {
  const int frames = j->d.n_frames;
  int n = most_batch_frames(&j->d, j->g, j->sa.ngrid, !j->pa.has_qc && !j->pa.window);
  if (n < 2) return;
  const int parts = (frames + n - 1) / n;
  n = (frames + parts - 1) / parts;
  const size_t bytes = carve_batch(j, n, nullptr).bytes;
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || bytes * 16 > free_b + idle_pool_bytes(j)) return;
  if (job_alloc_once(j, &j->batch_mem, bytes) != cudaSuccess) {   // frame by frame
    cudaGetLastError();
    j->batch_mem = nullptr;
    return;
  }
  j->batch = n;
}

extern "C" int mpsq_job_estimate_bytes(const mpsq_job_desc* d, int64_t* bytes) {
  if (!d || !bytes) return fail(MPSQ_ERR_ARG, "estimate: null pointer");
  EsKernel es;
  GridGeom g;
  int ng, gof[MPSQ_MAX_SPECIES], cof[MPSQ_MAX_SPECIES], pr[MPSQ_MAX_SPECIES],
      sa[MPSQ_MAX_SPECIES], sb[MPSQ_MAX_SPECIES], pack;
  int rc = job_layout(d, &es, &g, &ng, gof, cof, pr, sa, sb, &pack);
  if (rc) return rc;
  const int64_t per = d->ndim == 3 ? 8 : 4;
  int64_t b = 0;
  b += (int64_t)d->n_frames * d->n_atoms_frame * 16;                  // trajectory
  b += (int64_t)std::max(1, ng) * g.n_fine * (int64_t)csize(d->precision);  // fine grids
  b += d->n_atoms_frame * per * (int64_t)(rsize(d->precision) + csize(d->precision));
  b += (int64_t)(std::max(1, ng) * g.n_tiles + 1) * 8;
  b += d->n_atoms_frame * 4 + (int64_t)(std::max(1, ng) * g.n_tiles + 2) * 8;  // locality order
  const int64_t prep = (int64_t)prep_cache_bytes(d->precision, d->phase_rounding, false,
                                                 d->n_atoms_frame);  // per-atom preparation
  b += prep;
  const int64_t store = d->q_slab > 0 ? g.m[0] * g.m[1] * std::min<int64_t>(d->q_slab, g.m[2])
                                      : g.n_modes;                      // modes per frame kept
  b += (int64_t)d->n_frames * store * (int64_t)csize(d->precision);     // cs(t,Q)
  if (d->store_species)
    b += (int64_t)d->n_frames * d->n_species * store * (int64_t)csize(d->precision);
  const bool pruned = takes_pruned_passes(d, g);
  if (takes_lines(d, g)) {       // x-pass output and tables of the line transforms
    GridLines gl;
    gl.dim = g.dim;
    for (int k = 0; k < g.dim; ++k) {
      gl.n[k] = g.nf[k];
      gl.K[k] = 2 * (int)(g.m[k] / 2) + 1;
      b += g.nf[k] * 20 + 256;
    }
    b += gl.tmp_elems(std::max(1, ng)) * (int64_t)sizeof(double2);
  } else if (pruned && d->ndim == 2) {  // X-pass output
    b += (int64_t)std::max(1, ng) * g.nf[1] * (2 * (g.m[0] / 2) + 1) * 8;
  } else if (pruned) {  // X-pass output, plus a second frame lane (fine grid, bins, records, X output)
    const int64_t b1 = (int64_t)std::max(1, ng) * g.nf[2] * g.nf[1] * (2 * (g.m[0] / 2) + 1) * 8;
    b += b1;
    b += (int64_t)std::max(1, ng) * g.n_fine * 8 + (int64_t)(std::max(1, ng) * g.n_tiles + 1) * 8 +
         d->n_atoms_frame * per * (int64_t)(rsize(d->precision) + csize(d->precision)) + b1 + prep;
  } else {
    // cuFFT work areas (estimate): the strided (z, y) plans of the kept x columns of a 3D grid
    // hold up to their own data each, about a quarter of the grid per plan
    b += g.n_fine * (int64_t)csize(d->precision) / (d->ndim == 3 ? 2 : 4);
  }
  // frame batch: as of a long run, whatever the number of frames (admission may compare runs by it)
  const bool unit_str = !d->spatial_window && (pack || (d->q_center[0] == 0.0 && d->q_center[1] == 0.0 && d->q_center[2] == 0.0));
  const int batch = most_batch_frames(d, g, std::max(1, ng), unit_str);
  if (batch > 1) b += (int64_t)carve_batch(d, g, std::max(1, ng), unit_str, batch, nullptr).bytes;
  if (!d->stream_ordered)
    for (int s = 0; s < kScratchCount; ++s) b += (int64_t)scratch_cap(*d, g, (JobScratch)s);
  // deconvolution factors, twiddles, rounding of every part up to the allocators' 256 and 512 bytes
  for (int k = 0; k < 3; ++k) b += g.m[k] * 8 + g.nf[k] * 16;
  b += 32 * 512;
  *bytes = b;
  return MPSQ_OK;
}

// Volumes on cuFFT (FP64, and FP32 fine grids off the compiled length ladder) transform only
// what the deconvolution reads: one batch of x transforms over every row, then batched 2D
// (z, y) transforms over the x columns whose frequencies are kept, [0, h0] and [n0 - h0, n0)
// with h0 = m0 / 2 (the modes and their mirrors), strided by n0 within each grid.  About half
// the columns take the (z, y) part, so the transform does ~2/3 of a full 3D one.
static int make_xpruned_fft(mpsq_job* j) {
  const GridGeom& g = j->g;
  const cufftType type = j->d.precision == MPSQ_FP64 ? CUFFT_Z2Z : CUFFT_C2C;
  const long long n0 = g.nf[0], n1 = g.nf[1], n2 = g.nf[2];
  const int h0 = (int)(g.m[0] / 2);
  long long nx[1] = {n0};
  long long nzy[2] = {n2, n1};
  const long long batch[3] = {(long long)j->sa.ngrid * n1 * n2, h0 + 1, h0};
  for (int k = 0; k < 3; ++k) {
    if (batch[k] == 0) continue;
    MPSQ_CUFFT_TRY(cufftCreate(&j->xfft[k]));
    j->have_xfft = true;
    size_t ws = 0;
    cufftResult r = k == 0 ? cufftMakePlanMany64(j->xfft[k], 1, nx, nullptr, 1, n0, nullptr, 1, n0,
                                                 type, batch[k], &ws)
                           : cufftMakePlanMany64(j->xfft[k], 2, nzy, nzy, n0, 1, nzy, n0, 1, type,
                                                 batch[k], &ws);
    if (r == CUFFT_SUCCESS) r = cufftSetStream(j->xfft[k], j->s);
    if (r != CUFFT_SUCCESS)
      return fail(MPSQ_ERR_CUFFT, "cufftMakePlanMany (%s part, %lld x %lld x %lld) status %d",
                  k == 0 ? "x" : "z-y", n0, n1, n2, (int)r);
  }
  j->xfft_h0 = h0;
  return MPSQ_OK;
}

static int exec_xpruned_fft(mpsq_job* j) {
  const int prec = j->d.precision;
  const size_t cs = prec == MPSQ_FP64 ? sizeof(double2) : sizeof(float2);
  char* base = static_cast<char*>(j->fine);
  int rc = exec_fft(j->xfft[0], prec, base, CUFFT_FORWARD);
  if (rc) return rc;
  const int64_t n0 = j->g.nf[0];
  for (int gi = 0; gi < j->sa.ngrid; ++gi) {
    char* grid = base + (size_t)gi * j->g.n_fine * cs;
    rc = exec_fft(j->xfft[1], prec, grid, CUFFT_FORWARD);
    if (!rc && j->xfft[2])
      rc = exec_fft(j->xfft[2], prec, grid + (size_t)(n0 - j->xfft_h0) * cs, CUFFT_FORWARD);
    if (rc) return rc;
  }
  return MPSQ_OK;
}

extern "C" int mpsq_job_create(const mpsq_job_desc* d, void* stream, mpsq_job** out) {
  if (!d || !out) return fail(MPSQ_ERR_ARG, "job_create: null pointer");
  *out = nullptr;
  auto* j = new mpsq_job();
  j->d = *d;
  j->s = (cudaStream_t)stream;
  if (d->stream_ordered == 1) {
    // keep memory that jobs give back in the pool for the next job (process-local setting)
    static std::once_flag once;
    std::call_once(once, [] {
      int dev = 0;
      cudaMemPool_t pool;
      if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
        uint64_t keep = ~0ull;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
      }
      cudaGetLastError();
    });
  }
  int gof[MPSQ_MAX_SPECIES], cof[MPSQ_MAX_SPECIES], pr[MPSQ_MAX_SPECIES] = {0},
      sa[MPSQ_MAX_SPECIES] = {0}, sb[MPSQ_MAX_SPECIES] = {0}, pack = 0;
  int rc = job_layout(d, &j->es, &j->g, &j->ngroups, gof, cof, pr, sa, sb, &pack);
  if (rc) {
    delete j;
    return rc;
  }
  const int prec = d->precision;
  // spread geometry
  SpreadArgs& a = j->sa;
  a.dim = d->ndim;
  a.w = j->es.w;
  a.beta = j->es.beta;
  for (int k = 0; k < 3; ++k) {
    a.nf[k] = j->g.nf[k];
    a.tile[k] = j->g.tile[k];
    a.ntile[k] = j->g.ntile[k];
  }
  a.n_tiles = j->g.n_tiles;
  a.n_fine = j->g.n_fine;
  a.ngrid = std::max(1, j->ngroups);
  finish_spread_args(a);
  // preparation parameters
  PrepArgs& p = j->pa;
  p.dim = d->ndim;
  p.n_species = d->n_species;
  for (int s = 0; s <= d->n_species; ++s) p.species_offset[s] = d->species_offset[s];
  for (int s = 0; s < d->n_species; ++s) {
    p.group_of[s] = gof[s];
    p.comp_of[s] = cof[s];
  }
  p.input_method = d->input_method;
  p.phase_rounding = d->phase_rounding;
  p.use_range = d->use_range;
  p.bulk_nsuper1 = d->bulk_nsuper1;
  for (int k = 0; k < 3; ++k) {
    p.n_row[k] = d->n_row[k];
    for (int b = 0; b < 3; ++b) {
      p.axis[k][b] = d->axis[k][b];
      p.axis_f[k][b] = (float)d->axis[k][b];
    }
    p.tpe[k] = d->tpe[k];
    p.tpe_f[k] = (float)d->tpe[k];
    p.centre[k] = d->centre[k];
    p.centre_f[k] = (float)d->centre[k];
    p.pos_min[k] = d->pos_min[k];
    p.pos_max[k] = d->pos_max[k];
    p.pos_min_f[k] = (float)d->pos_min[k];
    p.pos_max_f[k] = (float)d->pos_max[k];
    p.q_center[k] = d->q_center[k];
    p.tpq_f[k] = (float)(2.0 * M_PI) * (float)d->q_center[k];
  }
  p.tol_f = d->bulk_nsuper1 ? (float)d->eps_x : 1.0f;
  p.has_qc = pack ? 0 : !(d->q_center[0] == 0.0 && d->q_center[1] == 0.0 && d->q_center[2] == 0.0);
  p.window = d->spatial_window;
  p.pack = pack;
  p.n_atoms_frame = d->n_atoms_frame;
  p.diag = 1;
  for (int k = 0; k < 3; ++k) {
    const double sc = d->tpe[k] * a.gscale[k];  // radians -> fine-grid units along axis k
    double bk = 0.0;
    for (int b = 0; b < 3; ++b) {
      const double A = d->axis[k][b] * sc;
      p.ahi[k][b] = (float)A;
      p.alo[k][b] = (float)(A - (double)p.ahi[k][b]);
      bk -= A * d->centre[b];
    }
    p.bhi[k] = (float)bk;
    p.blo[k] = (float)(bk - (double)p.bhi[k]);
    p.qhi[k] = (float)d->q_center[k];
    p.qlo[k] = (float)(d->q_center[k] - (double)p.qhi[k]);
    p.nf[k] = (int)j->g.nf[k];
    for (int b = 0; b < 3; ++b)
      if (b != k && (p.ahi[k][b] != 0.0f || p.alo[k][b] != 0.0f)) p.diag = 0;
    p.inv_nf[k] = (float)(1.0 / (double)j->g.nf[k]);
  }
  // weighting parameters
  WeightArgs& w = j->wa;
  w.ngroups = j->ngroups;
  for (int gi = 0; gi < j->ngroups; ++gi) {
    w.pair[gi] = pr[gi];
    w.sp_a[gi] = sa[gi];
    w.sp_b[gi] = sb[gi];
  }
  w.weight_mode = d->weight_mode;
  for (int s = 0; s < d->n_species; ++s) {
    w.b_coh[s] = d->b_coh[s];
    for (int i = 0; i < 9; ++i) w.xff[s][i] = d->xff[s][i];
  }
  w.kappa = d->ff_convention == MPSQ_FF_STANDARD ? 1.0 / (16.0 * M_PI * M_PI) : 1.0 / 16.0;
  for (int b = 0; b < 3; ++b) {
    w.q0[b] = d->qphys_origin[b];
    for (int k = 0; k < 3; ++k) w.qs[k][b] = d->qphys_step[k][b];
  }
  w.extra_sq = d->qphys_extra_sq;
  w.wnorm = d->spatial_window ? (d->ndim == 2 ? 0.25 : 0.125) : 1.0;
  for (int s = 0; s < d->n_species; ++s) {
    w.b_coh_f[s] = (float)w.b_coh[s];
    for (int i = 0; i < 9; ++i) w.xff_f[s][i] = (float)w.xff[s][i];
    for (int i = 0; i < 4; ++i) w.xb2_f[s][i] = (float)(w.xff[s][2 * i + 1] * M_LOG2E);
  }
  w.kappa_f = (float)w.kappa;
  for (int b = 0; b < 3; ++b) {
    w.q0_f[b] = (float)w.q0[b];
    for (int k = 0; k < 3; ++k) w.qs_f[k][b] = (float)w.qs[k][b];
  }
  // a Q origin below the FP32 rounding of the largest |Q| leaves |Q(-k)| = |Q(k)|
  double q_max = 0.0, q_org = 0.0;
  for (int b = 0; b < 3; ++b) {
    double e = 0.0;
    for (int k = 0; k < d->ndim; ++k) e += std::fabs(w.qs[k][b]) * (double)(d->n_modes[k] / 2);
    q_max = std::max(q_max, e);
    q_org = std::max(q_org, std::fabs(w.q0[b]));
  }
  w.even = q_org <= 6e-8 * q_max ? 1 : 0;
  w.extra_f = (float)w.extra_sq;
  w.wnorm_f = (float)w.wnorm;
  w.store_species = d->store_species;
  w.n_species = d->n_species;

  // device memory
  j->cap = records_cap(d);
  if (j->cap > (int64_t)INT32_MAX) {
    job_free(j);
    return fail(MPSQ_ERR_ARG, "job: too many atoms per frame for int32 bins");
  }
  const size_t cs = csize(prec);
  const int64_t nkeys = (int64_t)a.ngrid * j->g.n_tiles;
  cudaError_t e = cudaSuccess;
  // One allocation for what every job has, carved: a request server creates jobs on many streams, and an
  // allocation from the stream-ordered pool costs more there (eight jobs in flight: ~30 us each) than
  // everything else a small job's creation does.  Arrays from 32 MB get their own: one block of 41 GB takes
  // the driver longer to find again after a job has been closed (a job of three 1152^3 grids: 8.3 ms in one
  // block, 4.2 this way, 5.1 with every array on its own).
  std::vector<std::pair<void**, size_t>> parts;
  auto A = [&](void** ptr, size_t bytes) { parts.push_back({ptr, (std::max<size_t>(bytes, 16) + 255) & ~size_t(255)}); };
  auto allocate = [&](void** mem) {
    constexpr size_t apart = size_t(32) << 20;
    size_t total = 0;
    for (const auto& p : parts) total += p.second < apart ? p.second : 0;
    if (e == cudaSuccess) e = job_alloc(j, mem, total);
    char* at = static_cast<char*>(*mem);
    for (const auto& p : parts) {
      if (p.second >= apart) {
        if (e == cudaSuccess) e = job_alloc(j, p.first, p.second);
        if (e == cudaSuccess) j->large_mem.push_back(*p.first);
        continue;
      }
      *p.first = e == cudaSuccess ? at : nullptr;
      at += e == cudaSuccess ? p.second : 0;
    }
    parts.clear();
  };
  A((void**)&j->traj, (size_t)d->n_frames * d->n_atoms_frame * sizeof(float4));
  A(&j->fine, (size_t)a.ngrid * j->g.n_fine * cs);
  A((void**)&j->counts, sizeof(int) * (nkeys + 1));
  A((void**)&j->starts, sizeof(int) * (nkeys + 1));
  A((void**)&j->perm, sizeof(int) * std::max<int64_t>(d->n_atoms_frame, 1));
  A((void**)&j->perm_counts, sizeof(int) * (nkeys + 2));
  A((void**)&j->perm_starts, sizeof(int) * (nkeys + 2));
  A(&j->recs, (size_t)j->cap * rsize(prec));
  A(&j->str, (size_t)j->cap * cs);
  const size_t prep_b = prep_cache_bytes(j);
  if (prep_b) A(&j->prep, prep_b);
  j->slab_nz = d->q_slab > 0 ? std::min<int64_t>(d->q_slab, j->g.m[2]) : 0;
  const int64_t store = j->store_modes();
  A(&j->cs, (size_t)d->n_frames * store * cs);
  if (d->store_species) A(&j->cs_species, (size_t)d->n_frames * d->n_species * store * cs);
  A((void**)&j->err, sizeof(int));
  allocate(&j->main_mem);
  // deconvolution factors of the three axes in one block (an axis like an earlier one copies it), with the
  // pruned passes' gains taken back
  const bool pruned = takes_pruned_passes(d, j->g);
  std::vector<float2> axis_tw[3];          // the passes' twiddles, empty for an axis like an earlier one
  {
    std::vector<double> c[3];
    size_t off[3], bytes = 0;
    const size_t esz = prec == MPSQ_FP64 ? 8 : 4;
    for (int k = 0; k < 3; ++k) {
      c[k].assign(j->g.m[k], 1.0);
      int like = -1;
      for (int q = 0; q < k && k < d->ndim; ++q)
        if (j->g.m[q] == j->g.m[k] && j->g.nf[q] == j->g.nf[k]) like = q;
      if (like >= 0)
        c[k] = c[like];
      else if (k < d->ndim) {
        es_correction(j->es, j->g.nf[k], j->g.m[k], c[k].data());
        if (pruned) {
          std::vector<double> gain;
          axis_tw[k] = pass_twiddles((int)j->g.nf[k], &gain);
          const int64_t half = j->g.m[k] / 2;                  // mode i is frequency i - half
          for (int64_t i = 0; i < j->g.m[k]; ++i) c[k][i] /= gain[std::abs(i - half)];
        }
      }
      off[k] = bytes;
      bytes += (c[k].size() * esz + 255) & ~size_t(255);
    }
    std::vector<char> host(bytes);
    for (int k = 0; k < 3; ++k)
      for (size_t i = 0; i < c[k].size(); ++i) {
        if (prec == MPSQ_FP64)
          memcpy(&host[off[k] + 8 * i], &c[k][i], 8);
        else {
          const float v = (float)c[k][i];
          memcpy(&host[off[k] + 4 * i], &v, 4);
        }
      }
    if (e == cudaSuccess) e = job_alloc(j, &j->corr_mem, bytes);
    if (e == cudaSuccess) e = job_upload(j, j->corr_mem, host.data(), bytes);
    for (int k = 0; k < 3; ++k) j->corr[k] = static_cast<char*>(j->corr_mem) + off[k];
  }
  if (e == cudaSuccess)
    e = j->d.stream_ordered ? cudaMemsetAsync(j->err, 0, sizeof(int), j->s) : cudaMemset(j->err, 0, sizeof(int));
  if (e == cudaSuccess) e = clear_masked_species(j);
  if (e != cudaSuccess) {
    job_free(j);
    return fail(e == cudaErrorMemoryAllocation ? MPSQ_ERR_ALLOC : MPSQ_ERR_CUDA, "job_create: %s",
                cudaGetErrorString(e));
  }
  // Pruned fine-grid transform for FP32 grids of compiled lengths.
  if (pruned) {
    for (int k = 0; k < 3; ++k) {
      j->h[k] = (int)(j->g.m[k] / 2);
      j->K[k] = 2 * j->h[k] + 1;
    }
    const int64_t n1 = j->g.nf[1], n2 = j->g.nf[2];
    e = job_alloc(j, (void**)&j->b1, sizeof(float2) * (size_t)a.ngrid * n2 * n1 * j->K[0]);
    std::vector<float2> tw;               // the tables of the different lengths, one after another
    size_t off[3];
    for (int k = 0; k < d->ndim; ++k) {
      off[k] = tw.size();
      for (int q = 0; q < k; ++q)
        if (j->g.nf[q] == j->g.nf[k]) off[k] = off[q];
      if (off[k] == tw.size()) {
        tw.insert(tw.end(), axis_tw[k].begin(), axis_tw[k].end());
        tw.resize((tw.size() + 31) & ~size_t(31));
      }
    }
    if (e == cudaSuccess) e = job_alloc(j, &j->tw_mem, sizeof(float2) * tw.size());
    if (e == cudaSuccess) e = job_upload(j, j->tw_mem, tw.data(), sizeof(float2) * tw.size());
    for (int k = 0; k < d->ndim; ++k) j->tw[k] = static_cast<float2*>(j->tw_mem) + off[k];
    if (e != cudaSuccess) {
      job_free(j);
      return fail(e == cudaErrorMemoryAllocation ? MPSQ_ERR_ALLOC : MPSQ_ERR_CUDA,
                  "job_create (pruned transform): %s", cudaGetErrorString(e));
    }
    j->pruned = true;
    // second lane (frames alternate between two streams) for multi-frame jobs when its scratch
    // is small next to the free device memory
    const char* lanes = getenv("MPSQ_LANES");
    const size_t extra = (size_t)a.ngrid * j->g.n_fine * cs + 2 * sizeof(int) * (nkeys + 1) +
                         (size_t)j->cap * (rsize(prec) + cs) +
                         sizeof(float2) * (size_t)a.ngrid * n2 * n1 * j->K[0] + prep_b;
    size_t free_b = 0, total_b = 0;
    if (d->ndim == 3 && !d->stream_ordered && d->n_frames > 1 && !(lanes && strcmp(lanes, "1") == 0) &&
        cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && extra * 4 < free_b) {
      cudaError_t e2 = cudaStreamCreateWithFlags(&j->s2, cudaStreamNonBlocking);
      if (e2 == cudaSuccess) e2 = cudaEventCreateWithFlags(&j->fork, cudaEventDisableTiming);
      if (e2 == cudaSuccess) e2 = cudaEventCreateWithFlags(&j->join, cudaEventDisableTiming);
      A(&j->fine2, (size_t)a.ngrid * j->g.n_fine * cs);
      A((void**)&j->counts2, sizeof(int) * (nkeys + 1));
      A((void**)&j->starts2, sizeof(int) * (nkeys + 1));
      A(&j->recs2, (size_t)j->cap * rsize(prec));
      A(&j->str2, (size_t)j->cap * cs);
      A((void**)&j->b1_2, sizeof(float2) * (size_t)a.ngrid * n2 * n1 * j->K[0]);
      if (prep_b) A(&j->prep2, prep_b);
      size_t total = 0;
      for (const auto& p : parts) total += p.second;
      if (e2 == cudaSuccess) e2 = cudaMalloc(&j->lane_mem, total);
      if (e2 == cudaSuccess) {
        char* at = static_cast<char*>(j->lane_mem);
        for (const auto& p : parts) {
          *p.first = at;
          at += p.second;
        }
        j->lane2 = true;
      } else {  // run with one lane
        cudaGetLastError();
        j->lane_mem = nullptr;
      }
      parts.clear();
    }
    make_batch(j);
  } else if (takes_lines(d, j->g)) {
    std::vector<char> tables;
    grid_lines_plan(j->g, MPSQ_FP64, (int64_t)a.ngrid * (d->n_frames > 1 ? 8 : 1), &j->lines, &tables);
    e = job_alloc(j, &j->line_tables, tables.size());
    if (e == cudaSuccess) e = job_alloc(j, &j->line_tmp, sizeof(double2) * j->lines.tmp_elems(a.ngrid));
    if (e == cudaSuccess) e = job_upload(j, j->line_tables, tables.data(), tables.size());
    if (e != cudaSuccess) {
      job_free(j);
      return fail(e == cudaErrorMemoryAllocation ? MPSQ_ERR_ALLOC : MPSQ_ERR_CUDA,
                  "job_create (line transforms): %s", cudaGetErrorString(e));
    }
    grid_lines_bind(&j->lines, j->line_tables);
    j->have_lines = true;
    make_batch(j);
  } else {
    if (d->ndim == 3) {
      rc = make_xpruned_fft(j);
      if (rc) {
        job_free(j);
        return rc;
      }
    } else {
      rc = make_fft_plan(j->g, a.ngrid, prec, j->s, &j->fft);
      if (rc) {
        job_free(j);
        return rc;
      }
      j->have_fft = true;
    }
  }
  *out = j;
  return MPSQ_OK;
}

extern "C" int mpsq_job_destroy(mpsq_job* j) {
  if (j && !j->d.stream_ordered) {
    if (j->s2) cudaStreamSynchronize(j->s2);
    if (j->s) cudaStreamSynchronize(j->s);
  }
  job_free(j);   // stream-ordered: the frees follow the job's queued work on its stream
  return MPSQ_OK;
}

extern "C" int mpsq_job_set_frames_on(mpsq_job* j, const float* pos, int32_t first,
                                      int32_t count, int host, void* stream) {
  if (!j || !pos) return fail(MPSQ_ERR_ARG, "set_frames: null pointer");
  if (first < 0 || count < 0 || first + count > j->d.n_frames)
    return fail(MPSQ_ERR_ARG, "set_frames: frames [%d, %d) outside [0, %d)", first, first + count,
                j->d.n_frames);
  const size_t bytes = (size_t)count * j->d.n_atoms_frame * sizeof(float4);
  float4* dst = j->traj + (size_t)first * j->d.n_atoms_frame;
  MPSQ_CUDA_TRY(cudaMemcpyAsync(dst, pos, bytes, host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice,
                                (cudaStream_t)stream));
  return MPSQ_OK;
}

extern "C" int mpsq_job_set_frames(mpsq_job* j, const float* pos, int32_t first, int32_t count,
                                   int host) {
  if (!j) return fail(MPSQ_ERR_ARG, "set_frames: null job");
  return mpsq_job_set_frames_on(j, pos, first, count, host, j->s);
}

extern "C" int mpsq_job_set_cell_index(mpsq_job* j, const int32_t* at_ind, int host) {
  if (!j || !at_ind) return fail(MPSQ_ERR_ARG, "set_cell_index: null pointer");
  if (!j->at_ind) MPSQ_CUDA_TRY(job_alloc(j, (void**)&j->at_ind, (size_t)j->d.n_atoms_frame * sizeof(int4)));
  MPSQ_CUDA_TRY(cudaMemcpyAsync(j->at_ind, at_ind, (size_t)j->d.n_atoms_frame * sizeof(int4),
                                host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, j->s));
  return MPSQ_OK;
}

// Planes per slab of the z-slab pipeline for this job (0: whole-grid passes).  It applies to
// FP32 volumes on the pruned transform whose packed pairs spread on the tensor cores, with a
// slab that leaves room for the Y output at the start of the fine buffer.
static int zslab_planes(const mpsq_job* j) {
  const int zs = j->opt_zslab;
  if (zs <= 0 || !j->pruned || j->d.precision != MPSQ_FP32 || j->d.ndim != 3) return 0;
  const SpreadArgs& a = j->sa;
  if (!j->pa.pack || j->opt_spread != 0 || !spread_pair_mma_enabled() || a.w < 3 || a.w > 8 ||
      a.tile[0] != 16 || a.tile[1] != 16 || a.tile[2] != 16)
    return 0;
  const int64_t n0 = j->g.nf[0], n1 = j->g.nf[1], n2 = j->g.nf[2];
  if (zs >= n2 || n2 % 16 != 0) return 0;
  if (n2 * j->K[1] * j->K[0] + zs * n1 * n0 > a.n_fine) return 0;
  return zs;
}

template <typename T>
static int job_transform_body(mpsq_job* j, int32_t first, int32_t count) {
  using C = typename Cplx<T>::type;
  using R = typename RecOf<T>::type;
  cudaStream_t s = j->s;  // the stream of the current frame's lane
  const SpreadArgs& a = j->sa;
  const int64_t nkeys = (int64_t)a.ngrid * a.n_tiles;
  const int bt = 256;
  const unsigned nb = (unsigned)((j->d.n_atoms_frame + bt - 1) / bt);
  const int64_t nm = j->store_modes();
  const bool prof = j->profile;
  auto mark = [&](int k) -> int {
    if (prof) MPSQ_CUDA_TRY(cudaEventRecord(j->ev[k], s));
    return MPSQ_OK;
  };
  // two lanes: even frames of the call on the job's stream, odd ones on the second lane,
  // which first waits for everything queued on the job's stream (uploads included); the
  // job's stream waits for the second lane at the end
  // small frames run in batches instead (sizes as equal as they go)
  const int zs = prof ? 0 : zslab_planes(j);
  // (two frames of a small volume: two lanes, 84 us, are ahead of a batch of two, 89 us)
  const int n_batch = j->batch > 1 && !prof && zs == 0 && count > (j->lane2 ? 2 : 1)
                          ? (count + j->batch - 1) / j->batch : 0;
  const int per_batch = n_batch ? (count + n_batch - 1) / n_batch : 1;
  BatchScratch bs{};
  if (n_batch) bs = carve_batch(j, j->batch, j->batch_mem);
  const bool two = j->lane2 && j->opt_lanes == 2 && !prof && count > 1 && !n_batch;
  cudaStream_t const main_s = j->s;
  // locality order from the first frame (atoms move little between frames; any order gives the
  // same records, a spatial one lets a warp's cursor atomics combine)
  if (count > 1 && j->ngroups > 0) {
    const float4* f0 = j->traj + (size_t)first * j->d.n_atoms_frame;
    MPSQ_CUDA_TRY(cudaMemsetAsync(j->perm_counts, 0, sizeof(int) * (nkeys + 2), main_s));
    job_perm_kernel<T, false><<<nb, bt, 0, main_s>>>(f0, j->at_ind, j->pa, a, nkeys,
                                                      j->perm_counts, j->perm_starts, j->perm);
    MPSQ_LAUNCH_CHECK();
    int rc = launch_scan<T>(j->perm_counts, j->perm_starts, nkeys + 1, main_s);
    if (rc) return rc;
    MPSQ_CUDA_TRY(cudaMemsetAsync(j->perm_counts, 0, sizeof(int) * (nkeys + 2), main_s));
    job_perm_kernel<T, true><<<nb, bt, 0, main_s>>>(f0, j->at_ind, j->pa, a, nkeys,
                                                     j->perm_counts, j->perm_starts, j->perm);
    MPSQ_LAUNCH_CHECK();
    j->perm_built = true;
  }
  const int* const perm = j->perm_built ? j->perm : nullptr;
  const bool plane = j->d.ndim == 2;
  WeightArgs plane_weights = j->wa;     // pass Z runs on the y axis of a plane
  for (int b = 0; b < 3; ++b) {
    plane_weights.qs_f[2][b] = j->wa.qs_f[1][b];
    plane_weights.qs_f[1][b] = 0.0f;
  }
  // unit strengths (no centre phase, no spatial window) are implied, not stored
  const bool unit_str = !j->pa.has_qc && !j->pa.window;
  if (two) {
    MPSQ_CUDA_TRY(cudaEventRecord(j->fork, main_s));
    MPSQ_CUDA_TRY(cudaStreamWaitEvent(j->s2, j->fork, 0));
  }
  for (int32_t t = first; t < first + count; t += per_batch) {
    const int nf = std::min<int32_t>(per_batch, first + count - t);   // frames of this batch
    const bool odd = two && ((t - first) & 1);
    s = odd ? j->s2 : main_s;
    int* const counts = n_batch ? bs.counts : odd ? j->counts2 : j->counts;
    int* const starts = n_batch ? bs.starts : odd ? j->starts2 : j->starts;
    void* const recs = n_batch ? bs.recs : odd ? j->recs2 : j->recs;
    void* const str = unit_str ? nullptr : n_batch ? bs.str : (odd ? j->str2 : j->str);
    void* const fine = n_batch ? bs.fine : odd ? j->fine2 : j->fine;
    float2* const b1 = n_batch ? (float2*)bs.b1 : odd ? j->b1_2 : j->b1;
    const int64_t bkeys = nkeys * nf, bcap = j->cap * nf;
    const dim3 bgrid(nb, (unsigned)nf);
    SpreadArgs ab = a;          // the grids of all frames of the batch
    ab.ngrid = a.ngrid * nf;
    const float4* frame = j->traj + (size_t)t * j->d.n_atoms_frame;
    // FP32 split path: atoms prepared once, by the counting pass
    const bool cached = sizeof(T) == 4 && j->prep != nullptr;
    PrepCache pc{};
    if (cached) {
      char* base = static_cast<char*>(n_batch ? bs.prep : odd ? j->prep2 : j->prep);
      const size_t n = (size_t)j->d.n_atoms_frame * nf;
      pc.cell = reinterpret_cast<int4*>(base);
      pc.d2 = reinterpret_cast<float*>(base + 16 * n);
      pc.c = unit_str ? nullptr : reinterpret_cast<float2*>(base + 24 * n);
    }
    if (mark(0)) return MPSQ_ERR_CUDA;
    PhaseRange bin_range("mpsq:sort");
    MPSQ_CUDA_TRY(cudaMemsetAsync(counts, 0, sizeof(int) * (bkeys + 1), s));
    if (j->ngroups > 0) {
      if (cached)
        job_bin_count_split_kernel<<<bgrid, bt, 0, s>>>(frame, j->at_ind, perm, j->pa, a, counts,
                                                        pc, j->err);
      else
        job_bin_kernel<T, false><<<bgrid, bt, 0, s>>>(frame, j->at_ind, perm, j->pa, a, counts,
                                                      starts, (R*)recs, (C*)str, bcap, j->err);
      MPSQ_LAUNCH_CHECK();
    }
    int rc = launch_scan<T>(counts, starts, bkeys, s);
    if (rc) return rc;
    MPSQ_CUDA_TRY(cudaMemsetAsync(counts, 0, sizeof(int) * (bkeys + 1), s));
    if (j->ngroups > 0) {
      if (cached)
        job_bin_scatter_split_kernel<<<bgrid, bt, 0, s>>>(j->d.n_atoms_frame, pc, a, counts, starts,
                                                          (RecF*)recs, (float2*)str, bcap, j->err);
      else
        job_bin_kernel<T, true><<<bgrid, bt, 0, s>>>(frame, j->at_ind, perm, j->pa, a, counts,
                                                     starts, (R*)recs, (C*)str, bcap, j->err);
      MPSQ_LAUNCH_CHECK();
    }
    if (mark(1)) return MPSQ_ERR_CUDA;
    nvtxRangePop();                       // end of mpsq:sort
    nvtxRangePushA("mpsq:spread");
    if (zs == 0) {   // otherwise spread slab by slab with the X and Y passes, below
      rc = launch_spread<T>(ab, (const R*)recs, (const C*)str, starts, j->pa.pack != 0, (C*)fine,
                            s, j->opt_spread == 0, j->opt_repro != 0);
      if (rc) return rc;
    }
    if (mark(2)) return MPSQ_ERR_CUDA;
    nvtxRangePop();                       // end of mpsq:spread
    nvtxRangePushA("mpsq:fft+deconv");    // popped by bin_range at the end of the frame
    C* csf = (C*)j->cs + (size_t)t * nm;
    C* css = j->cs_species ? (C*)j->cs_species + (size_t)t * j->d.n_species * nm : nullptr;
    bool done = false;
    if constexpr (sizeof(T) == 4) {
      if (j->pruned) {
        PruneLaunch pl;
        pl.fine = (const float2*)fine;
        pl.n_fine = a.n_fine;
        pl.b1 = b1;
        pl.b2 = (float2*)fine;  // the fine grids are dead after pass X
        // a plane takes pass X, then pass Z on its y axis over one row (no pass Y)
        const int axis[3] = {0, plane ? 2 : 1, plane ? 1 : 2};
        for (int i = 0; i < 3; ++i) {
          const int k = axis[i];
          pl.n[i] = (int)j->g.nf[k];
          pl.m[i] = (int)j->g.m[k];
          pl.h[i] = j->h[k];
          pl.K[i] = j->K[k];
          pl.tw[i] = j->tw[k];
          pl.c[i] = (const float*)j->corr[k];
        }
        pl.ngrid = ab.ngrid;
        pl.frames = nf;
        pl.ngroups = j->ngroups;
        pl.xrows = j->opt_xrows;
        pl.z0 = (int)j->slab_z0;
        pl.nz = plane ? pl.m[2] : (int)j->slab_planes();
        pl.fz0 = 0;
        pl.fnz = pl.n[2];
        pl.s = s;
        if (zs > 0) {
          // z-slab pipeline: the tiles of zs fine-grid planes are spread into a slab-sized
          // region at the end of the fine buffer (beyond the Y output at its start), and the
          // X and Y passes of those planes follow at once, so the slab and its X output
          // (reused for every slab) are read back from L2
          const int64_t n0 = j->g.nf[0], n1 = j->g.nf[1], n2 = j->g.nf[2];
          const int64_t nl = (int64_t)a.ntile[0] * a.ntile[1];
          float2* fslab = (float2*)fine + (int64_t)a.ngrid * (a.n_fine - zs * n1 * n0);
          for (int64_t z0 = 0; z0 < n2; z0 += zs) {
            const int nzp = (int)std::min<int64_t>(zs, n2 - z0);
            const int64_t gstride = nzp * n1 * n0;
            for (int g = 0; g < a.ngrid; ++g) {
              rc = launch_spread_pair_mma(a, (const RecF*)recs, (const float2*)str, starts,
                                          (int)((nzp / 16) * nl), fslab, s,
                                          (int64_t)g * a.n_tiles + (z0 / 16) * nl, (int)z0,
                                          gstride, j->opt_repro != 0);
              if (rc) return rc;
            }
            pl.fine = fslab;
            pl.n_fine = gstride;
            pl.fz0 = (int)z0;
            pl.fnz = nzp;
            rc = run_pruned_xy(pl);
            if (rc) return rc;
          }
        } else {
          rc = plane ? run_pruned_x(pl) : run_pruned_xy(pl);
          if (rc) return rc;
          if (plane) pl.b2 = b1;
        }
        if (prof) MPSQ_CUDA_TRY(cudaEventRecord(j->ev[3], s));
        rc = run_pruned_z(pl, plane ? plane_weights : j->wa, (float2*)csf, (float2*)css);
        if (rc) return rc;
        done = true;
      }
    }
    if (!done) {
      KeptLayout kept{};
      const C* spec = (const C*)fine;
      if (j->have_lines) {
        // the last grid of a frame is real when its species has no partner (pairs are packed in order)
        const bool real = j->pa.pack && j->ngroups > 0 && !j->wa.pair[j->ngroups - 1];
        rc = run_grid_lines(j->lines, ab.ngrid, a.ngrid, real, fine, n_batch ? bs.b1 : j->line_tmp, false, s);
        kept = {1, j->lines.K[0], j->lines.K[1], {j->lines.h[0], j->lines.h[1], j->lines.h[2]},
                real ? j->ngroups - 1 : -1};
        spec += j->lines.kept();
      } else {
        rc = j->have_xfft ? exec_xpruned_fft(j) : exec_fft(j->fft, j->d.precision, j->fine,
                                                            CUFFT_FORWARD);
      }
      if (rc) return rc;
      if (mark(3)) return MPSQ_ERR_CUDA;
      const dim3 dgrid((unsigned)((j->g.m[0] + 127) / 128), (unsigned)j->g.m[1],
                       (unsigned)(j->slab_planes() * nf));
      job_deconv_kernel<T><<<dgrid, 128, 0, s>>>(
          a, kept, (int)j->g.m[0], (int)j->g.m[1], (int)j->g.m[2], (int)j->slab_z0,
          (int)j->slab_planes(), spec, (const T*)j->corr[0],
          (const T*)j->corr[1], (const T*)j->corr[2], j->wa, csf, css);
      MPSQ_LAUNCH_CHECK();
    }
    if (prof) {
      if (mark(4)) return MPSQ_ERR_CUDA;
      MPSQ_CUDA_TRY(cudaEventSynchronize(j->ev[4]));
      for (int k = 0; k < 4; ++k) {
        float ms = 0.0f;
        MPSQ_CUDA_TRY(cudaEventElapsedTime(&ms, j->ev[k], j->ev[k + 1]));
        j->stage_ms[k] += ms;
      }
      j->stage_frames += 1;
    }
  }
  if (two) {
    MPSQ_CUDA_TRY(cudaEventRecord(j->join, j->s2));
    MPSQ_CUDA_TRY(cudaStreamWaitEvent(main_s, j->join, 0));
  }
  return MPSQ_OK;
}

static int job_transform_direct(mpsq_job* j, int32_t first, int32_t count) {
  return j->d.precision == MPSQ_FP64 ? job_transform_body<double>(j, first, count)
                                     : job_transform_body<float>(j, first, count);
}

// The frame loop of one transform call captured once as a CUDA graph (per (first, count)) and
// replayed: the same kernels and copies, issued by one graph launch instead of ~7 launches per
// frame.  Capture runs on a private stream (the job's stream may be the legacy default stream,
// which cannot be captured); the graph is launched on the job's stream.
static int job_transform_graph(mpsq_job* j, int32_t first, int32_t count) {
  for (const auto& gr : j->graphs) {
    if (gr.first == first && gr.count == count) {
      MPSQ_CUDA_TRY(cudaGraphLaunch(gr.exec, j->s));
      count_launch((int)gr.launches);
      return MPSQ_OK;
    }
  }
  cudaStream_t cap = nullptr;
  MPSQ_CUDA_TRY(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
  cudaStream_t const user = j->s;
  const int64_t n0 = g_launches.load();
  cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
  int rc = MPSQ_OK;
  if (e == cudaSuccess) {
    j->s = cap;
    rc = job_transform_direct(j, first, count);
    j->s = user;
  }
  cudaGraph_t graph = nullptr;
  if (e == cudaSuccess) {
    const cudaError_t e2 = cudaStreamEndCapture(cap, &graph);
    if (rc == MPSQ_OK) e = e2;
  }
  const int64_t launches = g_launches.load() - n0;
  count_launch(-(int)launches);      // captured, not run
  cudaGraphExec_t exec = nullptr;
  if (e == cudaSuccess && rc == MPSQ_OK) e = cudaGraphInstantiate(&exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  cudaStreamDestroy(cap);
  if (rc) return rc;
  if (e != cudaSuccess) return fail(MPSQ_ERR_CUDA, "transform graph: %s", cudaGetErrorString(e));
  if (j->graphs.size() >= 16) {      // bounded cache: drop the oldest
    cudaGraphExecDestroy(j->graphs.front().exec);
    j->graphs.erase(j->graphs.begin());
  }
  j->graphs.push_back({first, count, exec, launches});
  MPSQ_CUDA_TRY(cudaGraphLaunch(exec, j->s));
  count_launch((int)launches);
  return MPSQ_OK;
}

extern "C" int mpsq_job_transform(mpsq_job* j, int32_t first, int32_t count) {
  if (!j) return fail(MPSQ_ERR_ARG, "transform: null job");
  if (first < 0 || count < 0 || first + count > j->d.n_frames)
    return fail(MPSQ_ERR_ARG, "transform: frames outside the trajectory");
  if (j->opt_graph && !j->profile && count > 0) return job_transform_graph(j, first, count);
  return job_transform_direct(j, first, count);
}

static void drop_graphs(mpsq_job* j) {
  for (auto& gr : j->graphs) cudaGraphExecDestroy(gr.exec);
  j->graphs.clear();
}

extern "C" int mpsq_job_set_option(mpsq_job* j, int option, int value) {
  if (!j) return fail(MPSQ_ERR_ARG, "set_option: null job");
  switch (option) {
    case MPSQ_OPT_GRAPH:
      if (value != 0 && value != 1) return fail(MPSQ_ERR_ARG, "set_option: graph must be 0 or 1");
      j->opt_graph = value;
      break;
    case MPSQ_OPT_SPREAD:
      if (value != 0 && value != 1) return fail(MPSQ_ERR_ARG, "set_option: spread must be 0 or 1");
      j->opt_spread = value;
      break;
    case MPSQ_OPT_XROWS:
      if (value != 4 && value != 8) return fail(MPSQ_ERR_ARG, "set_option: X rows must be 4 or 8");
      j->opt_xrows = value;
      break;
    case MPSQ_OPT_LANES:
      if (value != 1 && value != 2) return fail(MPSQ_ERR_ARG, "set_option: lanes must be 1 or 2");
      j->opt_lanes = value;
      break;
    case MPSQ_OPT_ZSLAB:
      if (value < 0 || value % 16 != 0 || value > 4096)
        return fail(MPSQ_ERR_ARG, "set_option: z-slab planes must be 0 or a multiple of 16");
      j->opt_zslab = value;
      break;
    case MPSQ_OPT_REPRODUCIBLE:
      if (value != 0 && value != 1)
        return fail(MPSQ_ERR_ARG, "set_option: reproducible must be 0 or 1");
      j->opt_repro = value;
      break;
    default:
      return fail(MPSQ_ERR_ARG, "set_option: unknown option %d", option);
  }
  drop_graphs(j);   // captured graphs hold the previous choice
  return MPSQ_OK;
}

// Autotuner: times the transform of frames [first, first + count) under every combination of
// the run-time choices that applies to this job (spreading kernel, X-pass rows, frame lanes,
// graph replay, z-slab pipeline), keeps the fastest and, given a cache file, records it there
// under a key of the job's shape and the device's SM count, so that later jobs of the same
// shape take the choice without timing.
// Cache lines: "<key> <graph> <spread> <xrows> <lanes> <zslab> <ms>".
static std::string tune_key(const mpsq_job* j) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  char buf[256];
  snprintf(buf, sizeof(buf), "mpsq-tune-2:p%d:d%d:n%lldx%lldx%lld:w%d:g%d:pk%d:pr%d:l%d:b%d:sm%d",
           j->d.precision, j->d.ndim, (long long)j->g.nf[0], (long long)j->g.nf[1],
           (long long)j->g.nf[2], j->es.w, j->sa.ngrid, j->pa.pack, j->pruned ? 1 : 0,
           j->lane2 ? 1 : 0, j->batch, sms);
  return buf;
}

extern "C" int mpsq_job_autotune(mpsq_job* j, int32_t first, int32_t count, const char* cache_path,
                                 int* choice, double* best_ms) {
  if (!j) return fail(MPSQ_ERR_ARG, "autotune: null job");
  if (first < 0 || count < 1 || first + count > j->d.n_frames)
    return fail(MPSQ_ERR_ARG, "autotune: frames outside the trajectory");
  const std::string key = tune_key(j);
  int best[5] = {j->opt_graph, j->opt_spread, j->opt_xrows, j->opt_lanes, j->opt_zslab};
  double best_t = -1.0;
  if (cache_path && *cache_path) {
    if (FILE* f = fopen(cache_path, "r")) {
      char line[512], k[256];
      while (fgets(line, sizeof(line), f)) {
        int g, sp, xr, ln, zs;
        double ms;
        if (sscanf(line, "%255s %d %d %d %d %d %lf", k, &g, &sp, &xr, &ln, &zs, &ms) == 7 &&
            key == k) {
          best[0] = g;
          best[1] = sp;
          best[2] = xr;
          best[3] = ln;
          best[4] = zs;
          best_t = ms;
        }
      }
      fclose(f);
    }
  }
  const bool cached = best_t >= 0.0;
  if (!cached) {
    const bool fma_ok = j->d.precision == MPSQ_FP32 && j->d.ndim == 3 && j->pa.pack != 0;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    MPSQ_CUDA_TRY(cudaEventCreate(&e0));
    MPSQ_CUDA_TRY(cudaEventCreate(&e1));
    int rc = MPSQ_OK;
    // candidate settings {graph, spread, xrows, lanes, zslab}; the z-slab pipeline is tried at
    // 64 planes where it applies (tensor-core spreading of pairs on the pruned transform)
    const int zs_saved = j->opt_zslab, sp_saved = j->opt_spread;
    j->opt_spread = 0;
    j->opt_zslab = 64;
    const bool zs_ok = zslab_planes(j) > 0;
    j->opt_zslab = zs_saved;
    j->opt_spread = sp_saved;
    std::vector<std::array<int, 5>> cand;
    for (int g = 0; g <= 1; ++g)
      for (int sp = 0; sp <= (fma_ok ? 1 : 0); ++sp)
        for (int xr : {8, 4})
          for (int ln = 2; ln >= 1; --ln)
            for (int zs : {0, 64})
              if ((j->pruned || xr == 8) && (j->lane2 || ln == 1) && (!zs || (zs_ok && sp == 0)))
                cand.push_back({g, sp, xr, ln, zs});
    for (size_t c = 0; c < cand.size() && !rc; ++c) {
      const std::array<int, 5>& o = cand[c];
      j->opt_graph = o[0];
      j->opt_spread = o[1];
      j->opt_xrows = o[2];
      j->opt_lanes = o[3];
      j->opt_zslab = o[4];
      drop_graphs(j);
      rc = mpsq_job_transform(j, first, count);           // warm-up (and capture)
      if (!rc && cudaEventRecord(e0, j->s) != cudaSuccess) rc = MPSQ_ERR_CUDA;
      for (int r = 0; r < 2 && !rc; ++r) rc = mpsq_job_transform(j, first, count);
      if (!rc && cudaEventRecord(e1, j->s) != cudaSuccess) rc = MPSQ_ERR_CUDA;
      if (!rc && cudaEventSynchronize(e1) != cudaSuccess) rc = MPSQ_ERR_CUDA;
      float ms = 0.0f;
      if (!rc && cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) rc = MPSQ_ERR_CUDA;
      ms *= 0.5f;
      if (!rc && (best_t < 0.0 || ms < best_t)) {
        best_t = ms;
        for (int i = 0; i < 5; ++i) best[i] = o[i];
      }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) {
      if (rc == MPSQ_ERR_CUDA) fail(MPSQ_ERR_CUDA, "autotune: %s", cudaGetErrorString(cudaGetLastError()));
      return rc;
    }
  }
  j->opt_graph = best[0];
  j->opt_spread = best[1];
  j->opt_xrows = best[2];
  j->opt_lanes = best[3];
  j->opt_zslab = best[4];
  drop_graphs(j);
  if (!cached && cache_path && *cache_path) {
    if (FILE* f = fopen(cache_path, "a")) {
      fprintf(f, "%s %d %d %d %d %d %.4f\n", key.c_str(), best[0], best[1], best[2], best[3],
              best[4], best_t);
      fclose(f);
    }
  }
  if (choice) {
    choice[0] = best[0];
    choice[1] = best[1];
    choice[2] = best[2];
    choice[3] = best[3];
  }
  if (best_ms) *best_ms = best_t;
  return MPSQ_OK;
}

extern "C" int mpsq_job_get_option(const mpsq_job* j, int option, int* value) {
  if (!j || !value) return fail(MPSQ_ERR_ARG, "get_option: null pointer");
  switch (option) {
    case MPSQ_OPT_GRAPH: *value = j->opt_graph; break;
    case MPSQ_OPT_SPREAD: *value = j->opt_spread; break;
    case MPSQ_OPT_XROWS: *value = j->opt_xrows; break;
    case MPSQ_OPT_LANES: *value = j->opt_lanes; break;
    case MPSQ_OPT_ZSLAB: *value = j->opt_zslab; break;
    case MPSQ_OPT_REPRODUCIBLE: *value = j->opt_repro; break;
    default: return fail(MPSQ_ERR_ARG, "get_option: unknown option %d", option);
  }
  return MPSQ_OK;
}

template <typename T>
static int job_onephonon_t(mpsq_job* j, int32_t first, int32_t count, int32_t plane, int32_t n_bz,
                           float qx_min, float qy_min) {
  using C = typename Cplx<T>::type;
  const int n1 = j->d.n_row[0], n2 = j->d.n_row[1];
  const int m0 = (int)j->d.n_modes[0], m1 = (int)j->d.n_modes[1];
  const int ns = j->d.n_species;
  const size_t usz = (size_t)ns * 2 * n1 * n2 * sizeof(C);
  if (!j->oneph_u) MPSQ_CUDA_TRY(job_alloc(j, &j->oneph_u, usz));
  if (!j->have_oneph_fft) {
    int n[2] = {n2, n1};
    MPSQ_CUFFT_TRY(cufftPlanMany(&j->oneph_fft, 2, n, nullptr, 1, n1 * n2, nullptr, 1, n1 * n2,
                                 sizeof(T) == 8 ? CUFFT_Z2Z : CUFFT_C2C, 2 * ns));
    j->have_oneph_fft = true;
  }
  MPSQ_CUFFT_TRY(cufftSetStream(j->oneph_fft, j->s));
  // nqx_min = n_row * (qx_min - floor(qx_min)), FP32, truncated (:1039-1040)
  const int nqx_min = (int)(float)((float)n1 * (qx_min - std::floor(qx_min)));
  const int nqy_min = (int)(float)((float)n2 * (qy_min - std::floor(qy_min)));
  const int bt = 256;
  const unsigned nb = (unsigned)((j->d.n_atoms_frame + bt - 1) / bt);
  const int64_t nm = j->g.n_modes;
  for (int32_t t = first; t < first + count; ++t) {
    MPSQ_CUDA_TRY(cudaMemsetAsync(j->oneph_u, 0, usz, j->s));
    oneph_scatter_kernel<T><<<nb, bt, 0, j->s>>>(j->traj + (size_t)t * j->d.n_atoms_frame,
                                                  j->at_ind, j->pa, plane, j->oneph_base, n1, n2,
                                                  (C*)j->oneph_u);
    MPSQ_LAUNCH_CHECK();
    if constexpr (sizeof(T) == 8) {
      MPSQ_CUFFT_TRY(cufftExecZ2Z(j->oneph_fft, (cufftDoubleComplex*)j->oneph_u,
                                  (cufftDoubleComplex*)j->oneph_u, CUFFT_FORWARD));
    } else {
      MPSQ_CUFFT_TRY(cufftExecC2C(j->oneph_fft, (cufftComplex*)j->oneph_u,
                                  (cufftComplex*)j->oneph_u, CUFFT_FORWARD));
    }
    C* csf = (C*)j->cs + (size_t)t * nm;
    C* css = j->cs_species ? (C*)j->cs_species + (size_t)t * ns * nm : nullptr;
    oneph_expand_kernel<T><<<dim3((unsigned)((m0 + 127) / 128), (unsigned)m1), 128, 0, j->s>>>(
        (const C*)j->oneph_u, j->pa, plane, j->oneph_base, n1, n2, m0, m1, n_bz, qx_min, qy_min,
        nqx_min, nqy_min, j->wa, csf, css);
    MPSQ_LAUNCH_CHECK();
  }
  return MPSQ_OK;
}

extern "C" int mpsq_job_transform_onephonon(mpsq_job* j, int32_t first, int32_t count,
                                            int32_t plane, int32_t n_bz, float qx_min,
                                            float qy_min, const float* at_base) {
  if (!j || !at_base) return fail(MPSQ_ERR_ARG, "transform_onephonon: null pointer");
  if (first < 0 || count < 0 || first + count > j->d.n_frames)
    return fail(MPSQ_ERR_ARG, "transform_onephonon: frames outside the trajectory");
  if (j->d.input_method != MPSQ_CELL || j->d.ndim != 2)
    return fail(MPSQ_ERR_ARG, "transform_onephonon: CELL input on a Q plane only (the reference "
                "turns the mode off for BULK input)");
  if (plane != 1 && plane != 2)
    return fail(MPSQ_ERR_ARG, "transform_onephonon: plane must be 1 (hk0) or 2 (hhl), got %d", plane);
  const int* nr = j->d.n_row;
  if (nr[0] != nr[1] || (plane == 2 && nr[2] != nr[0]))
    return fail(MPSQ_ERR_ARG, "transform_onephonon: needs n_row(1) = n_row(2) (= n_row(3) on "
                "(hhl)); the reference's index ranges mix the axes otherwise");
  if (n_bz < 1 || (int64_t)n_bz * nr[0] > j->d.n_modes[0] || (int64_t)n_bz * nr[1] > j->d.n_modes[1])
    return fail(MPSQ_ERR_ARG, "transform_onephonon: %d zones of %d cells exceed the %lld x %lld plane",
                n_bz, nr[0], (long long)j->d.n_modes[0], (long long)j->d.n_modes[1]);
  if (!j->at_ind) return fail(MPSQ_ERR_STATE, "transform_onephonon: set the cell indices first");
  if (!j->oneph_base) MPSQ_CUDA_TRY(job_alloc(j, (void**)&j->oneph_base, sizeof(float) * 3 * MPSQ_MAX_SPECIES));
  MPSQ_CUDA_TRY(cudaMemcpyAsync(j->oneph_base, at_base, sizeof(float) * 3 * j->d.n_species,
                                cudaMemcpyHostToDevice, j->s));
  // (a host-to-device copy from pageable memory has left the caller's buffer on return)
  return j->d.precision == MPSQ_FP64
             ? job_onephonon_t<double>(j, first, count, plane, n_bz, qx_min, qy_min)
             : job_onephonon_t<float>(j, first, count, plane, n_bz, qx_min, qy_min);
}

extern "C" int mpsq_job_profile(mpsq_job* j, int enable) {
  if (!j) return fail(MPSQ_ERR_ARG, "profile: null job");
  if (enable)
    for (auto& e : j->ev)
      if (!e) MPSQ_CUDA_TRY(cudaEventCreate(&e));
  j->profile = enable != 0;
  return MPSQ_OK;
}

extern "C" int mpsq_job_stage_ms(mpsq_job* j, double* ms4, int64_t* frames, int reset) {
  if (!j) return fail(MPSQ_ERR_ARG, "stage_ms: null job");
  if (ms4)
    for (int k = 0; k < 4; ++k) ms4[k] = j->stage_ms[k];
  if (frames) *frames = j->stage_frames;
  if (reset) {
    for (double& v : j->stage_ms) v = 0.0;
    j->stage_frames = 0;
  }
  return MPSQ_OK;
}

extern "C" int mpsq_job_amplitudes(mpsq_job* j, void** cs_dev) {
  if (!j || !cs_dev) return fail(MPSQ_ERR_ARG, "amplitudes: null pointer");
  *cs_dev = j->cs;
  return MPSQ_OK;
}

extern "C" int mpsq_job_info(const mpsq_job* j, int* width, int64_t* fine_grid, int* n_grids,
                             int* pruned, int* lanes) {
  if (!j) return fail(MPSQ_ERR_ARG, "job_info: null job");
  if (width) *width = j->es.w;
  if (fine_grid)
    for (int k = 0; k < 3; ++k) fine_grid[k] = j->g.nf[k];
  if (n_grids) *n_grids = j->sa.ngrid;
  if (pruned) *pruned = j->pruned ? 1 : 0;
  if (lanes) *lanes = j->lane2 ? 2 : 1;
  return MPSQ_OK;
}

extern "C" int mpsq_job_set_q_slab(mpsq_job* j, int64_t z0) {
  if (!j) return fail(MPSQ_ERR_ARG, "set_q_slab: null job");
  if (j->slab_nz == 0) return fail(MPSQ_ERR_STATE, "set_q_slab: job created without q_slab");
  if (z0 < 0 || z0 >= j->g.m[2])
    return fail(MPSQ_ERR_ARG, "set_q_slab: z0 = %lld outside [0, %lld)", (long long)z0,
                (long long)j->g.m[2]);
  const int64_t planes = j->slab_planes();
  j->slab_z0 = z0;
  if (j->slab_planes() != planes) MPSQ_CUDA_TRY(clear_masked_species(j));
  drop_graphs(j);   // captured graphs hold the previous slab
  return MPSQ_OK;
}

extern "C" int mpsq_job_sync(mpsq_job* j) {
  if (!j) return fail(MPSQ_ERR_ARG, "sync: null job");
  MPSQ_CUDA_TRY(cudaStreamSynchronize(j->s));
  return check_dev_error(j->err, j->s);
}

// ---- accessors used by the time-axis unit
namespace mpsq {
MapMem::MapMem(mpsq_job* j) : job(j), kept(j->map_mu, std::defer_lock) {
  if (!j->d.stream_ordered) (void)kept.try_lock();
}
MapMem::~MapMem() {
  for (void* p : own) cudaFreeAsync(p, job->s);
}
int MapMem::take(JobScratch slot, size_t bytes, void** p) {
  bytes = std::max<size_t>(bytes, 16);
  cudaError_t e = cudaSuccess;
  if (kept.owns_lock() && bytes <= scratch_cap(job->d, job->g, slot)) {
    if (bytes > job->scratch_bytes[slot]) {
      job_release(job, job->scratch[slot]);   // (cudaFree waits for kernels that still use it)
      job->scratch[slot] = nullptr;
      job->scratch_bytes[slot] = 0;
      e = job_alloc(job, &job->scratch[slot], bytes);
      if (e == cudaSuccess) job->scratch_bytes[slot] = bytes;
    }
    *p = job->scratch[slot];
  } else {
    e = job->d.stream_ordered ? job_alloc_once(job, p, bytes) : cudaMallocAsync(p, bytes, job->s);
    if (e == cudaSuccess) own.push_back(*p);
  }
  if (e == cudaSuccess) return MPSQ_OK;
  cudaGetLastError();
  *p = nullptr;
  return fail(e == cudaErrorMemoryAllocation ? MPSQ_ERR_ALLOC : MPSQ_ERR_CUDA, "map memory: %s",
              cudaGetErrorString(e));
}
JobView job_view(mpsq_job* j) {
  JobView v;
  v.precision = j->d.precision;
  v.s = j->s;
  v.cs = j->cs;
  v.cs_species = j->cs_species;
  v.n_q = j->store_modes();
  v.slab = j->slab_nz > 0;
  v.n_frames = j->d.n_frames;
  v.n_species = j->d.n_species;
  for (int k = 0; k < 3; ++k) v.m[k] = j->g.m[k];
  v.store_species = j->d.store_species;
  return v;
}
}  // namespace mpsq
