// Pruned fine-grid transform of FP32 grids (passes.cu): host interface.
#pragma once

#include <vector>

#include "weights.cuh"

namespace mpsq {

// Only the 2h+1 central frequencies f in [-h, h] (h = m/2) of each dimension are needed
// (modes -m/2..(m-1)/2 plus the mirror +m/2 that packed-pair separation reads), so the 3D
// FFT runs as three passes that each keep 2h+1 of n outputs:
//   X: fine (n2, n1, n0)   -> b1 (n2, n1, K0)
//   Y: b1                  -> b2 (n2, K1, K0)
//   Z: b2 column tiles and their mirror tiles -> deconvolution, pair separation, species
//      weights, cs(t, Q)
// K = 2h+1; frequency f is stored at index f + h.  A Q plane takes X, then Z on its y axis.
struct PruneLaunch {
  const float2* fine;
  int64_t n_fine;
  float2* b1;
  float2* b2;
  int n[3], m[3], h[3], K[3];
  int ngrid, ngroups;
  int frames = 1;            // frames of the batch (ngrid counts the grids of all of them)
  int xrows = 8;             // rows per CTA of the X pass (4 or 8)
  int z0 = 0, nz = 0;        // kz planes of the store's Q slab
  int fz0 = 0, fnz = 0;      // fine-grid planes [fz0, fz0 + fnz) of the X and Y passes
  const float2* tw[3];       // pass_twiddles of each axis, in device memory
  const float* c[3];
  cudaStream_t s;
};

// Fine-grid lengths of volumes: a ladder with steps of at most 1.5 that covers fine grids up to 1600
// points per axis (the largest a pass's shared-memory tile holds); each is exercised on the GPU by a
// parity test against the FP64 direct sum.
#define MPSQ_FFT_SIZES(X)                                                                    \
  X(64) X(96) X(128) X(160) X(192) X(256) X(320) X(384) X(512) X(640) X(768) X(960) X(1024)   \
  X(1152) X(1280) X(1536) X(1600)
// Further lengths that only planes take (multiples of the 32-cell tile with factors 2, 3, 5, up to
// 1600): a plane's grid keeps its length instead of moving up the ladder.
#define MPSQ_FFT_PLANE_SIZES(X) X(32) X(288) X(480) X(576) X(800) X(864) X(1440)

bool fft_size_compiled(int n);
bool fft_plane_size_compiled(int n);               // of the further lengths
int64_t compiled_fft_size_at_least(int64_t n);     // of the ladder; 0 above the largest
// The twiddles of the passes over lines of length n.  gains: what the FP32 rounding of all constants and
// twiddles makes of frequencies f and -f on average, |f| <= n / 4, for the deconvolution factors to take
// back.  It does not average out over a line: up to 4e-8 for some frequencies (0 for f = 0), and the power
// of all modes of a 512^3 grid together would be 1.9e-7 short.
std::vector<float2> pass_twiddles(int n, std::vector<double>* gains = nullptr);

// Pass X, and X and Y, over the fine-grid planes [fz0, fz0 + fnz).
int run_pruned_x(const PruneLaunch& p);
int run_pruned_xy(const PruneLaunch& p);
// Pass Z with the deconvolution and weights, over the whole of b2.
int run_pruned_z(const PruneLaunch& p, const WeightArgs& w, float2* csf, float2* css);

}  // namespace mpsq
