// Interface between simple.cu (drivers, element-wise kernels, float64 / SIMT paths) and
// simple_pairs.cu (the float32 tensor-core path of the simple lattices on the fp16-pair engine).
#pragma once
#include <algorithm>

#include "common.cuh"

namespace frnnt {

// extra state of the tensor-core path: `saved_bytes` follow the regular saved area (kept
// from forward to backward), `scratch_bytes` follow the regular scratch area
struct SimplePairsLayout {
  int Cp, Tq;  // row pitches (halves) of the planes with C resp. T entries per row
  int Sp;      // row pitch (floats) of am_sym [B][T][Sp] = am[b][t][symbols[b][s]]
  size_t lp_hi, lp_lo, ap_hi, ap_lo, lm_blk, lm_sym, lnorm, am_blk, am_sym, am_sum, weak, saved_bytes;
  size_t rw_hi, rw_lo, parts, inv_scale, scratch_bytes;
  SimplePairsLayout(int B, int S, int T, int C);
};

// Cells and frames that the planes cannot serve.  A plane pair of e^{x - max} is off by up to 2^-39,
// however small the value, and a normalizer z = sum_c A[t][c] L[s][c] by up to
// 2^-39 (sum_c A + sum_c L).  That counts where z is small because the two rows peak at
// different symbols (confident models).  Cells with z below 2^-19 of those two sums, for
// which the bound is 1e-6 of z, are computed in float32 from lm and am on the FMA pipe:
// the forward after its product, the backward beside it.  Without them the weights g / z of
// an utterance stay within 2^18 of each other, so that planes under one scale hold them, too.
constexpr float kWeak = 1.f / 524288.f;  // 2^-19
__host__ __device__ inline float weak_bound(float lm_sum, float am_sum) { return kWeak * (lm_sum + am_sum); }
// the same for the am-only normalizer sum_c A[t][c] u[c], sum_c u = 1
__device__ __forceinline__ bool am_only_weak(float ammax, float amonly) { return ammax - amonly > 13.1698f; }  // 19 log 2

// offset, inside the pairs saved area, of sum_c e^{am - ammax} per frame (B*T floats)
size_t simple_pairs_amsum_offset(int B, int S, int T, int C);

// offset, inside the pairs scratch, of the per-row maxima of |rw| that the caller fills in
// (B*(S+1) floats) before launch_simple_grads_pairs
size_t simple_pairs_rowmax_offset(int B, int S, int T, int C);

bool simple_pairs_supported(const void *lm, const void *am, int S1, int T, int C, int rnnt_type);

// whether a call gets the more accurate form of the products
bool simple_pairs_exact(const void *lm, const void *am, int C, int input_dtype);

// stage 0: row maxima / sums, exp planes, per-row scalars, the -inf column of px;
// stage 1: normalizer product + lattices (needs amonly / loguni when the am-only branch is on;
// a positive delay_penalty is added to px as the reference's loss functions do)
// lm / am: float32, or 16-bit values when input_dtype is FRNNT_F16 / FRNNT_BF16
int launch_simple_forward_pairs(const void *lm, const void *am, const int64_t *symbols,
                                const int64_t *boundary, int blank, int rnnt_type, int smoothed,
                                int am_only_off, float both, float ls, float as, float *px, float *py,
                                float *norm, float *lmmax, float *lmsum, float *ammax,
                                const float *amonly, const float *loguni, void *pairs_saved, int B, int S,
                                int T, int C, int stage, cudaStream_t st, double delay_penalty,
                                int input_dtype);

// the weak cells of the normalizer, px and py again in float32 (simple.cu)
struct SimpleLattice {  // what the cells of the lattices are made of
  float *norm, *px, *py;
  const float *am_sym;  // [B][T][Sp]
  const int64_t *symbols, *boundary;
  const float *lmmax, *ammax, *lm_blk, *lm_sym, *lnorm, *am_blk, *amonly, *loguni;
  const float *lmsum, *am_sum;
  uint8_t *weak;  // [B][tiles of 128 lattice rows][T]: the frame has weak cells in the tile
  int S, T, C, blank, rnnt_type;
  int smoothed, am_only_off;
  float both, ls, as;
  int Sp;
  double delay_penalty;
};
int launch_weak_cells(const void *lm, const void *am, int input_dtype, const SimpleLattice &lattice, int B,
                      cudaStream_t st);

// words of one bit per frame that say which cells of a lattice row are weak
__host__ __device__ inline int weak_words(int T) { return (T + 31) / 32; }

// lm_grad / am_grad without the one-hot terms, the unigram term of lm_grad and what weak cells and
// frames contribute, from the gradient weights rw [B][S+1][Tp], the bits of their weak cells
// [B][S+1][weak_words(T)] and the maxima of |rw| per row (see simple_pairs_rowmax_offset)
int launch_simple_grads_pairs(const float *rw, const unsigned *weak, const float *lmsum, const float *ammax,
                              const float *amonly, const float *uni, const float *gl, const float *h,
                              float *lm_grad, float *am_grad, const void *pairs_saved, void *pairs_scratch, int B, int S, int T, int C, int Tp,
                              bool exact, cudaStream_t st);

}  // namespace frnnt
