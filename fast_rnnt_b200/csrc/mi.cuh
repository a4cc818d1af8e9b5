// What the two families of mutual-information sweeps share (mi.cu: one row per thread,
// both precisions; mi_f32.cu: float, an utterance over a cluster of CTAs): the boundary
// box and the layout of the lattice scratch.
#pragma once
#include "common.cuh"

namespace frnnt {

struct MiBox {
  int s0, t0, sb, tb;  // origin and extents (s_end - s_begin, t_end - t_begin)
};

__device__ __forceinline__ MiBox load_box(const int64_t *boundary, int b, int S, int T) {
  MiBox box{0, 0, S, T};
  if (boundary != nullptr) {
    // clamped so that a malformed row can never index outside the tensors
    int s0 = (int)boundary[4 * b + 0], t0 = (int)boundary[4 * b + 1];
    int s1 = (int)boundary[4 * b + 2], t1 = (int)boundary[4 * b + 3];
    s0 = max(0, min(s0, S));
    t0 = max(0, min(t0, T));
    s1 = max(s0, min(s1, S));
    t1 = max(t0, min(t1, T));
    box = MiBox{s0, t0, s1 - s0, t1 - t0};
  }
  return box;
}

// lattice scratch: the weight exponents by anti-diagonal, [B][S+T+1][pitch]
__host__ __device__ inline int lattice_pitch(int S) { return (S + 1 + 31) & ~31; }
// followed, per utterance, by two vectors of edge_elems() values ([B][2][S+T+65]): when the
// lattice has more rows than one launch holds it is swept in row blocks; the forward sweep
// passes p of a block's last row, the backward sweep the x-gradients of a block's first
// row, to the next launch through them.  All lattices come first, so that each starts on a
// multiple of 32 values.
__host__ __device__ inline size_t edge_elems(int S, int T) { return (size_t)(S + T + 1 + 64); }
__host__ __device__ inline size_t lattice_elems(int S, int T) { return (size_t)(S + T + 1) * lattice_pitch(S); }
__host__ __device__ inline size_t lattice_elems_per_utt(int S, int T) {
  return lattice_elems(S, T) + 2 * edge_elems(S, T);
}
template <typename real>
__device__ __forceinline__ real *lattice_of(real *lattice, int b, int S, int T) {
  return lattice + (size_t)b * lattice_elems(S, T);
}
template <typename real>
__device__ __forceinline__ real *edges_of(real *lattice, int b, int B, int S, int T) {
  return lattice + (size_t)B * lattice_elems(S, T) + (size_t)b * 2 * edge_elems(S, T);
}

__device__ __forceinline__ void bar_sync_named(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// What the lattice scratch holds of a cell: double the exponent of its backward weight (share of
// the x-predecessor), p[s-1][t+o] + px[s-1][t+o] - p[s][t]; float the weight itself, or kMiDead
// where the exponent is not finite (no path reaches the cell; it passes no gradient on).
constexpr float kMiDead = -1.f;
__device__ __forceinline__ float mi_weight(float exponent) {
  const float w = expf(exponent);
  return w - w == 0.f ? w : kMiDead;
}
__device__ __forceinline__ float lattice_value(float exponent) { return mi_weight(exponent); }
__device__ __forceinline__ double lattice_value(double exponent) { return exponent; }
// weight from what the lattice holds; not finite or negative: no gradient
__device__ __forceinline__ float weight_of(float value) { return value; }
__device__ __forceinline__ double weight_of(double value) { return exp(value); }

// float sweeps (mi_f32.cu).  `lattice` must be 16-byte aligned; the forward takes NULL when
// the whole lattice fits one launch (S + 1 <= kMiF32Rows) and no backward sweep follows.
// `tries` bounds every wait between the CTAs of a cluster.
constexpr int kMiF32Rows = 512, kMiTries = 1 << 22;
int launch_mi_forward_f32(const float *px, const float *py, const int64_t *boundary, float *p, float *ans,
                          float *lattice, int B, int S, int T, int modified, cudaStream_t st,
                          int tries = kMiTries);
int launch_mi_backward_f32(float *lattice, const int64_t *boundary, const float *ans_grad, float *px_grad,
                           float *py_grad, float *origin_grad, int B, int S, int T, int modified,
                           cudaStream_t st, int tries = kMiTries);

}  // namespace frnnt
