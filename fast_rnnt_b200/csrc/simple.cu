// "Simple" (factorised joiner) log-prob lattices and their gradient:
// get_rnnt_logprobs and get_rnnt_logprobs_smoothed of the reference
// (fast_rnnt/python/fast_rnnt/rnnt_loss.py:160-227 and :1246-1369), which the
// reference composes from ~20-40 ATen kernels plus autograd.
//
//   N[b,s,t]  = log( sum_c e^{lm[b,s,c]-lmmax[b,s]} e^{am[b,t,c]-ammax[b,t]} + tiny ) + lmmax + ammax
//   px[b,s,t] = am[b,t,y_bs] + lm[b,s,y_bs] - N[b,s,t]      (t < T; -inf at t = T and t = t_end)
//   py[b,s,t] = am[b,t,blank] + lm[b,s,blank] - N[b,s,t]
//   smoothed:  x*(1-l-a) + x_lmonly*l + x_amonly*a with the lm-only softmax
//              normalizer, the batch-wide unigram and the am-only normalizer.
//
// Forward  = row statistics (max, sum exp) -> [unigram, am-only normalizer] ->
//            batched contraction with the exp() applied while the operand tiles
//            are staged and log()+max in the epilogue -> lattice assembly.
// Backward = analytic: with W = -(g_px + g_py)/(M + tiny) the two contractions
//            dlm = L .* (W A), dam = A .* (W^T L) plus the one-hot gather terms
//            and the lm-only / am-only / unigram terms.  The row maxima are
//            treated as constants: N does not depend on them analytically.
//
// This file holds the fp32/fp64 SIMT version of the contraction (FMA pipes,
// shared-memory tiles); it is the general path for both dtypes.
#include <stdlib.h>
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "lsm_band.cuh"
#include "simple_pairs.cuh"

namespace frnnt {

template <typename real> __device__ __forceinline__ real tiny_v();
template <> __device__ __forceinline__ float tiny_v<float>() { return 1.17549435e-38f; }
template <> __device__ __forceinline__ double tiny_v<double>() { return 2.2250738585072014e-308; }

static inline size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

// ---- buffers -----------------------------------------------------------------
// "saved": what the forward keeps for the backward.
struct SavedLayout {
  size_t norm, lmmax, lmsum, ammax, amonly, uni, loguni, total;
  SavedLayout(size_t es, int B, int S, int T, int C) {
    size_t o = 0;
    norm = o;   o += align_up(es * (size_t)B * (S + 1) * T);
    lmmax = o;  o += align_up(es * (size_t)B * (S + 1));
    lmsum = o;  o += align_up(es * (size_t)B * (S + 1));
    ammax = o;  o += align_up(es * (size_t)B * T);
    amonly = o; o += align_up(es * (size_t)B * T);
    uni = o;    o += align_up(es * (size_t)C);
    loguni = o; o += align_up(es * (size_t)C);
    total = o;
  }
};

constexpr int kColChunkRows = 32;  // rows folded by one CTA of the column-sum kernels

// row pitch of the gradient-weight matrix (16-byte aligned rows for the tensor-core path)
static inline int rw_pitch(int T) { return (T + 3) & ~3; }

// "scratch": temporaries of one call.
struct ScratchLayout {
  size_t rw, sgx, sgy, cgx, cgy, gl, h, partial, dp, rowdot, weak, weak_row, total;
  int nchunk;
  ScratchLayout(size_t es, int B, int S, int T, int C) {
    size_t o = 0;
    const size_t rows_max = (size_t)B * (T > S + 1 ? T : S + 1);
    nchunk = (int)((rows_max + kColChunkRows - 1) / kColChunkRows);
    rw = o;      o += align_up(es * (size_t)B * (S + 1) * rw_pitch(T));  // gradient weights, rows padded to 4
    sgx = o;     o += align_up(es * (size_t)B * (S + 1));      // sum_t gx, sum_t gy
    sgy = o;     o += align_up(es * (size_t)B * (S + 1));
    cgx = o;     o += align_up(es * (size_t)B * T);            // sum_s gx, sum_s gy
    cgy = o;     o += align_up(es * (size_t)B * T);
    gl = o;      o += align_up(es * (size_t)B * (S + 1));      // weight of the lm-only softmax
    h = o;       o += align_up(es * (size_t)B * T);            // weight of the am-only normalizer
    partial = o; o += align_up(es * (size_t)nchunk * C);       // column-sum partials
    dp = o;      o += align_up(es * (size_t)C);                // d loss / d unigram-softmax mean
    rowdot = o;  o += align_up(es * (size_t)B * (S + 1));
    weak = o;    o += align_up((size_t)B * (S + 1) * weak_words(T) * 4);  // bits of the weak cells
    weak_row = o; o += align_up((size_t)B * (S + 1));          // lattice row has any
    total = o;
  }
};

// ---- row statistics ------------------------------------------------------------
// one warp per row: max and sum(exp(x - max))
template <typename real>
__global__ void row_stats_kernel(const real *__restrict__ x, real *__restrict__ rmax,
                                 real *__restrict__ rsum, long long rows, int C) {
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarps) {
    const real *src = x + row * (long long)C;
    real m = neg_inf<real>();
    for (int c = lane; c < C; c += 32) m = max(m, src[c]);
    m = warp_max(m);
    real s = 0;
    for (int c = lane; c < C; c += 32) s += exp_r(src[c] - m);
    s = warp_sum(s);
    if (lane == 0) {
      rmax[row] = m;
      rsum[row] = s;
    }
  }
}

// one warp per row: the maximum alone (all that is needed of the am rows), 16-byte loads
// when the rows allow them
template <typename real>
__global__ void row_max_kernel(const real *__restrict__ x, real *__restrict__ rmax, long long rows,
                               int C, int vec_ok) {
  constexpr int VW = 16 / sizeof(real);
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarps) {
    const real *src = x + row * (long long)C;
    real m = neg_inf<real>();
    if (vec_ok) {
      const float4 *v4 = reinterpret_cast<const float4 *>(src);
      for (int c = lane; c < C / VW; c += 32) {
        const float4 q = v4[c];
        const real *e = reinterpret_cast<const real *>(&q);
#pragma unroll
        for (int i = 0; i < VW; ++i) m = max(m, e[i]);
      }
    } else {
      for (int c = lane; c < C; c += 32) m = max(m, src[c]);
    }
    m = warp_max(m);
    if (lane == 0) rmax[row] = m;
  }
}

// partial[chunk][c] = sum over the chunk's rows of f(row, c); one thread per column
//   MODE 0: softmax(lm row)[c]                      (unigram)
//   MODE 1: h[row] * e^{am[row,c]-ammax[row]} / Z[row]   (d unigram via the am-only normalizer)
template <typename real, int MODE>
__global__ void column_partial_kernel(const real *__restrict__ x, const real *__restrict__ rmax,
                                      const real *__restrict__ aux, const real *__restrict__ h,
                                      real *__restrict__ partial, long long rows, int C) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const long long r0 = (long long)blockIdx.y * kColChunkRows;
  const long long r1 = min(rows, r0 + kColChunkRows);
  real acc = 0;
#pragma unroll 8
  for (long long r = r0; r < r1; ++r) {
    const real e = exp_r(x[r * C + c] - rmax[r]);
    if (MODE == 0) {
      acc += e / aux[r];  // aux = sum exp
    } else {
      // aux = am-only normalizer (log Z + ammax)  ->  1/Z = e^{ammax - aux}
      acc += h[r] * e * exp_r(rmax[r] - aux[r]);
    }
  }
  partial[(size_t)blockIdx.y * C + c] = acc;
}

template <typename real>
__global__ void unigram_final_kernel(const real *__restrict__ partial, int nchunk, long long rows,
                                     int C, real *__restrict__ uni, real *__restrict__ loguni) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  real acc = 0;
#pragma unroll 8
  for (int j = 0; j < nchunk; ++j) acc += partial[(size_t)j * C + c];
  const real u = acc / (real)rows + tiny_v<real>();
  uni[c] = u;
  loguni[c] = log_r(u);
}

// one warp per am row: log(sum_c e^{am-ammax} u[c]) + ammax
template <typename real>
__global__ void am_only_norm_kernel(const real *__restrict__ am, const real *__restrict__ ammax,
                                    const real *__restrict__ uni, real *__restrict__ amonly,
                                    long long rows, int C) {
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarps) {
    const real *src = am + row * (long long)C;
    const real m = ammax[row];
    real z = 0;
#pragma unroll 8
    for (int c = lane; c < C; c += 32) z += exp_r(src[c] - m) * uni[c];
    z = warp_sum(z);
    if (lane == 0) amonly[row] = log_r(z) + m;
  }
}

// ---- the contraction (SIMT) ---------------------------------------------------------
// C[m][n] = sum_k X(m,k) * Y(n,k); the problem policy supplies the (transformed)
// operands, says which index is contiguous in memory, and consumes the result.
template <typename real, int BM, int BN, int BK, int TM, int TN, typename Prob>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) contraction_kernel(Prob prob) {
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int PAD = 4;
  __shared__ real Xs[BK][BM + PAD];
  __shared__ real Ys[BK][BN + PAD];
  prob.set_batch(blockIdx.z);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  real acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0;

  const int K = prob.K();
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll 4
    for (int idx = tid; idx < BM * BK; idx += NT) {
      const int k = Prob::X_K_CONTIG ? idx % BK : idx / BM;
      const int m = Prob::X_K_CONTIG ? idx / BK : idx % BM;
      Xs[k][m] = prob.x(m0 + m, k0 + k);
    }
#pragma unroll 4
    for (int idx = tid; idx < BN * BK; idx += NT) {
      const int k = Prob::Y_K_CONTIG ? idx % BK : idx / BN;
      const int n = Prob::Y_K_CONTIG ? idx / BK : idx % BN;
      Ys[k][n] = prob.y(n0 + n, k0 + k);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      real a[TM], bq[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = Xs[k][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) bq[j] = Ys[k][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] += a[i] * bq[j];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) prob.store(m0 + ty * TM + i, n0 + tx * TN + j, acc[i][j]);
}

// N[s][t] = log(sum_c L[s][c] A[t][c] + tiny) + lmmax[s] + ammax[t]
template <typename real>
struct NormProb {
  static constexpr bool X_K_CONTIG = true, Y_K_CONTIG = true;
  const real *lm, *am, *lmmax, *ammax;
  real *norm;
  int S1, T, C;
  __device__ void set_batch(int b) {
    lm += (size_t)b * S1 * C;
    am += (size_t)b * T * C;
    lmmax += (size_t)b * S1;
    ammax += (size_t)b * T;
    norm += (size_t)b * S1 * T;
  }
  __device__ int K() const { return C; }
  __device__ real x(int s, int c) const {
    return (s < S1 && c < C) ? exp_r(lm[(size_t)s * C + c] - lmmax[s]) : (real)0;
  }
  __device__ real y(int t, int c) const {
    return (t < T && c < C) ? exp_r(am[(size_t)t * C + c] - ammax[t]) : (real)0;
  }
  __device__ void store(int s, int t, real acc) const {
    if (s < S1 && t < T) norm[(size_t)s * T + t] = log_r(acc + tiny_v<real>()) + lmmax[s] + ammax[t];
  }
};

// dlm[s][c] = -L[s][c] * sum_t Rw[s][t] A[t][c]  - gl[s] P[s][c] + P[s][c] (dP[c] - rowdot[s])
template <typename real>
struct LmGradProb {
  static constexpr bool X_K_CONTIG = true, Y_K_CONTIG = false;
  const real *rw, *am, *ammax, *lm, *lmmax, *lmsum, *gl, *dp, *rowdot;
  real *lm_grad;
  int S1, T, C, Tp;
  __device__ void set_batch(int b) {
    rw += (size_t)b * S1 * Tp;
    am += (size_t)b * T * C;
    ammax += (size_t)b * T;
    lm += (size_t)b * S1 * C;
    lmmax += (size_t)b * S1;
    lmsum += (size_t)b * S1;
    if (gl) gl += (size_t)b * S1;
    if (rowdot) rowdot += (size_t)b * S1;
    lm_grad += (size_t)b * S1 * C;
  }
  __device__ int K() const { return T; }
  __device__ real x(int s, int t) const { return (s < S1 && t < T) ? rw[(size_t)s * Tp + t] : (real)0; }
  __device__ real y(int c, int t) const {
    return (c < C && t < T) ? exp_r(am[(size_t)t * C + c] - ammax[t]) : (real)0;
  }
  __device__ void store(int s, int c, real acc) const {
    if (s >= S1 || c >= C) return;
    const real L = exp_r(lm[(size_t)s * C + c] - lmmax[s]);
    real v = -(L * acc);
    if (gl != nullptr) {
      const real P = L / lmsum[s];
      v -= gl[s] * P;
      if (dp != nullptr) v += P * (dp[c] - rowdot[s]);
    }
    lm_grad[(size_t)s * C + c] = v;
  }
};

// dam[t][c] = -A[t][c] * sum_s Rw[s][t] L[s][c]  - h[t] A[t][c] u[c] / Z[t]
template <typename real>
struct AmGradProb {
  static constexpr bool X_K_CONTIG = false, Y_K_CONTIG = false;
  const real *rw, *lm, *lmmax, *am, *ammax, *h, *uni, *amonly;
  real *am_grad;
  int S1, T, C, Tp;
  __device__ void set_batch(int b) {
    rw += (size_t)b * S1 * Tp;
    lm += (size_t)b * S1 * C;
    lmmax += (size_t)b * S1;
    am += (size_t)b * T * C;
    ammax += (size_t)b * T;
    if (h) {
      h += (size_t)b * T;
      amonly += (size_t)b * T;
    }
    am_grad += (size_t)b * T * C;
  }
  __device__ int K() const { return S1; }
  __device__ real x(int t, int s) const { return (t < T && s < S1) ? rw[(size_t)s * Tp + t] : (real)0; }
  __device__ real y(int c, int s) const {
    return (c < C && s < S1) ? exp_r(lm[(size_t)s * C + c] - lmmax[s]) : (real)0;
  }
  __device__ void store(int t, int c, real acc) const {
    if (t >= T || c >= C) return;
    const real A = exp_r(am[(size_t)t * C + c] - ammax[t]);
    real v = -(A * acc);
    if (h != nullptr) v -= h[t] * A * uni[c] * exp_r(ammax[t] - amonly[t]);
    am_grad[(size_t)t * C + c] = v;
  }
};

template <typename real> struct TileCfg;
template <> struct TileCfg<float> { static constexpr int BM = 128, BN = 128, BK = 16, TM = 8, TN = 8; };
template <> struct TileCfg<double> { static constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4; };

template <typename real, typename Prob>
static int launch_contraction(const Prob &prob, int M, int N, int B, cudaStream_t st) {
  using Cfg = TileCfg<real>;
  dim3 grid((unsigned)((N + Cfg::BN - 1) / Cfg::BN), (unsigned)((M + Cfg::BM - 1) / Cfg::BM),
            (unsigned)B);
  FRNNT_KERNEL(contraction_kernel<real, Cfg::BM, Cfg::BN, Cfg::BK, Cfg::TM, Cfg::TN, Prob>
               <<<grid, (Cfg::BM / Cfg::TM) * (Cfg::BN / Cfg::TN), 0, st>>>(prob));
  FRNNT_CUDA(cudaGetLastError());
  return FRNNT_OK;
}

// ---- weak cells (simple_pairs.cuh): float32 products where the planes do not hold ---------------------
// acc[m][n] = sum_k X(m,k) Y(n,k) of one 64 x 64 tile, 16 entries per thread.  What bounds it is the
// latency of its loads (few tiles, long reductions): the operands of the next 16 k are
// fetched into registers while this slice's products run, and two buffers in shared memory leave
// one barrier per slice.  An operand says how a thread's four values of a slice are fetched and
// where (and through which function) they are placed.
constexpr int kWeakTile = 64, kWeakBK = 16, kWeakThreads = 256, kWeakPitch = kWeakTile + 4;
typedef float WeakSlice[kWeakBK][kWeakPitch];

template <class X, class Y>
__device__ __forceinline__ void weak_product(X &x, Y &y, int K, WeakSlice (&Xs)[2], WeakSlice (&Ys)[2],
                                             float (&acc)[4][4]) {
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  float xv[4], yv[4];
  x.fetch(0, K, xv);
  y.fetch(0, K, yv);
  for (int k0 = 0, buf = 0; k0 < K; k0 += kWeakBK, buf ^= 1) {
    x.place(k0, xv, Xs[buf]);
    y.place(k0, yv, Ys[buf]);
    __syncthreads();
    if (k0 + kWeakBK < K) {
      x.fetch(k0 + kWeakBK, K, xv);
      y.fetch(k0 + kWeakBK, K, yv);
    }
#pragma unroll
    for (int k = 0; k < kWeakBK; ++k) {
      const float4 a = *reinterpret_cast<const float4 *>(&Xs[buf][k][4 * ty]);
      const float4 b = *reinterpret_cast<const float4 *>(&Ys[buf][k][4 * tx]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += av[i] * bv[j];
    }
  }
  __syncthreads();  // the buffers are free again
}

// e^{row - max} of 64 rows, k along the row: thread <-> (row tid / 16 + 16 e, k tid % 16)
template <typename TIn>
struct WeakRows {
  const TIn *row[4];  // nullptr: no such row
  float mx[4];
  __device__ void fetch(int k0, int K, float (&v)[4]) const {
    const int k = k0 + threadIdx.x % 16;
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = row[e] != nullptr && k < K ? in_f32(row[e][k]) : -INFINITY;
  }
  __device__ void place(int, const float (&v)[4], WeakSlice &s) const {
#pragma unroll
    for (int e = 0; e < 4; ++e) s[threadIdx.x % 16][threadIdx.x / 16 + 16 * e] = expf(v[e] - mx[e]);
  }
};

// A CTA takes 64 lattice rows (constrained: 63, and the one that px of the last needs) and the
// blockIdx.x-th 64 of the frames that have weak cells among them; it leaves at once where there
// are none.  All its cells go through the product, the weak ones are replaced, and py and px
// follow from the normalizers.  64 x (100, 500) x 500: 4 us with nothing weak, 211 us with every
// cell weak; 16 x (59, 293) x 4233: 2 and 273 us.
template <typename TIn>
__global__ void __launch_bounds__(kWeakThreads)
weak_cells_kernel(const TIn *__restrict__ lm, const TIn *__restrict__ am, SimpleLattice q) {
  __shared__ __align__(16) WeakSlice Xs[2], Ys[2];
  __shared__ int frames[kWeakTile], counts[8];
  __shared__ uint8_t replaced[kWeakTile][16];  // bits of four rows each, per frame
  const int tid = threadIdx.x, lane = tid & 31, b = blockIdx.z;
  const bool constrained = q.rnnt_type == FRNNT_CONSTRAINED;
  const int s0 = blockIdx.y * (constrained ? kWeakTile - 1 : kWeakTile);
  const int S1 = q.S + 1, T = q.T, C = q.C;
  // flags per 128 rows; constrained lattices have one such tile
  const uint8_t *weak = q.weak + ((size_t)b * ((S1 + 127) / 128) + (constrained ? 0 : s0 / 128)) * T;
  bool any = false;
  for (int t = tid; t < T; t += kWeakThreads) any |= weak[t];
  if (!__syncthreads_or(any)) return;
  const int first = blockIdx.x * kWeakTile;
  int found = 0;
  for (int t0 = 0; t0 < T; t0 += kWeakThreads) {
    const int t = t0 + tid;
    const bool w = t < T && weak[t];
    const unsigned m = __ballot_sync(0xffffffffu, w);
    if (lane == 0) counts[tid >> 5] = __popc(m);
    __syncthreads();
    int at = found - first + __popc(m & ((1u << lane) - 1u));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i < tid >> 5) at += counts[i];
      found += counts[i];
    }
    if (w && at >= 0 && at < kWeakTile) frames[at] = t;
    __syncthreads();
  }
  const int nframes = min(kWeakTile, found - first), rows = min(kWeakTile, S1 - s0);
  if (nframes <= 0) return;
  const size_t bs0 = (size_t)b * S1 + s0, bt0 = (size_t)b * T;
  WeakRows<TIn> x, y;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int m = tid / 16 + 16 * e;
    x.row[e] = m < rows ? lm + (bs0 + m) * C : nullptr;
    x.mx[e] = m < rows ? q.lmmax[bs0 + m] : 0.f;
    y.row[e] = m < nframes ? am + (bt0 + frames[m]) * C : nullptr;
    y.mx[e] = m < nframes ? q.ammax[bt0 + frames[m]] : 0.f;
  }
  float acc[4][4] = {};
  weak_product(x, y, C, Xs, Ys, acc);
  const int tx = tid % 16, ty = tid / 16;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = 4 * tx + j;
    if (n >= nframes) break;
    const size_t bt = bt0 + frames[n];
    const float ax = q.ammax[bt], asum = q.am_sum[bt];
    unsigned bits = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int s = 4 * ty + i;
      if (s >= rows || !(acc[i][j] < weak_bound(q.lmsum[bs0 + s], asum))) continue;
      bits |= 1u << i;
      q.norm[(bs0 + s) * T + frames[n]] = logf(acc[i][j] + 1.17549435e-38f) + q.lmmax[bs0 + s] + ax;
    }
    replaced[n][ty] = (uint8_t)bits;
  }
  __syncthreads();
  const int T1 = q.rnnt_type == FRNNT_REGULAR ? T + 1 : T;
  const bool am_on = q.smoothed && !q.am_only_off;
  for (int idx = tid; idx < nframes * kWeakTile; idx += kWeakThreads) {
    const int n = idx / kWeakTile, t = frames[n], i = idx % kWeakTile, s = s0 + i;
    const bool here = replaced[n][i / 4] >> (i % 4) & 1;
    const bool next = constrained && i + 1 < kWeakTile && (replaced[n][(i + 1) / 4] >> ((i + 1) % 4) & 1);
    if (!here && !next) continue;
    const size_t bt = bt0 + t;
    auto py_of = [&](int k) {
      const size_t bs = bs0 + k;
      float v = q.am_blk[bt] + q.lm_blk[bs] - q.norm[bs * T + t];
      if (q.smoothed) v = v * q.both + (q.lm_blk[bs] - q.lnorm[bs]) * q.ls;
      if (am_on) v += (q.am_blk[bt] + q.loguni[q.blank] - q.amonly[bt]) * q.as;
      return v;
    };
    if (here) q.py[(bs0 + i) * T + t] = py_of(i);
    if (s >= q.S || (constrained && i == kWeakTile - 1)) continue;  // (that row is the next CTA's first)
    const size_t bs = bs0 + i;
    const float px_am = q.am_sym[bt * q.Sp + s], px_lm = q.lm_sym[bs];
    float v = px_am + px_lm - q.norm[bs * T + t];
    if (q.smoothed) v = v * q.both + (px_lm - q.lnorm[bs]) * q.ls;
    if (am_on) {
      long long c = q.symbols[(size_t)b * q.S + s];
      if (c < 0 || c >= C) c = q.blank;
      v += (px_am + q.loguni[c] - q.amonly[bt]) * q.as;
    }
    if (q.rnnt_type == FRNNT_REGULAR) {
      if (q.boundary != nullptr && (long long)t == (long long)q.boundary[4 * b + 3]) v = -INFINITY;
    } else if (constrained) {
      v += py_of(i + 1);
    }
    if (q.delay_penalty > 0.0) v = add_rn(v, delay_penalty_at<float>(q.boundary, b, T, t, q.delay_penalty));
    q.px[((size_t)b * q.S + s) * T1 + t] = v;
  }
}

// calls f with lm and am as pointers to their type
template <class F>
static void with_input_type(int input_dtype, const void *lm, const void *am, F f) {
  if (input_dtype == FRNNT_F16)
    f((const __half *)lm, (const __half *)am);
  else if (input_dtype == FRNNT_BF16)
    f((const __nv_bfloat16 *)lm, (const __nv_bfloat16 *)am);
  else
    f((const float *)lm, (const float *)am);
}

int launch_weak_cells(const void *lm, const void *am, int input_dtype, const SimpleLattice &lattice, int B,
                      cudaStream_t st) {
  const int step = lattice.rnnt_type == FRNNT_CONSTRAINED ? kWeakTile - 1 : kWeakTile;
  const dim3 grid((unsigned)((lattice.T + kWeakTile - 1) / kWeakTile), (unsigned)((lattice.S + step) / step),
                  (unsigned)B);
  with_input_type(input_dtype, lm, am, [&](auto *l, auto *a) {
    FRNNT_KERNEL(weak_cells_kernel<<<grid, kWeakThreads, 0, st>>>(l, a, lattice));
  });
  FRNNT_CUDA(cudaGetLastError());
  return FRNNT_OK;
}

// What weak cells add to the gradients, dlm[s][c] -= L[s][c] sum_t Rw[s][t] A[t][c] and
// dam[t][c] -= A[t][c] sum_s Rw[s][t] L[s][c] over the weak cells, and the am-only term of frames
// whose am-only normalizer is weak.
template <typename TIn>
struct WeakGrads {
  const TIn *lm, *am;
  const float *rw;
  const unsigned *weak;      // bits of the weak cells, [B][S1][words]
  const uint8_t *weak_row;   // [B][S1]
  const float *lmmax, *ammax, *amonly, *h, *uni;
  float *lm_grad, *am_grad;
  int B, S1, T, C, Tp;
};
// Rw of the weak cells of 64 rows of lm or am, k through a list of frames resp. lattice rows;
// neighbouring threads on neighbouring frames either way
struct WeakWeights {
  const float *rw;
  const unsigned *weak;
  const int *list;
  bool is_lm;
  int m0, M, Tp, words;
  unsigned word[4];
  int bit[4];
  __device__ int k_of(int e) const { return is_lm ? threadIdx.x % 16 : threadIdx.x / 64 + 4 * e; }
  __device__ int m_of(int e) const { return is_lm ? threadIdx.x / 16 + 16 * e : threadIdx.x % 64; }
  // the weight and the word that says whether it counts: neither load waits for the other
  __device__ void fetch(int k0, int K, float (&v)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = k0 + k_of(e), m = m0 + m_of(e);
      v[e] = 0.f, word[e] = 0u, bit[e] = 0;
      if (k >= K || m >= M) continue;
      const int at = list[k], s = is_lm ? m : at, t = is_lm ? at : m;
      word[e] = weak[(size_t)s * words + t / 32];
      bit[e] = t % 32;
      v[e] = rw[(size_t)s * Tp + t];
    }
  }
  __device__ void place(int, const float (&v)[4], WeakSlice &s) const {
#pragma unroll
    for (int e = 0; e < 4; ++e) s[k_of(e)][m_of(e)] = word[e] >> bit[e] & 1u ? v[e] : 0.f;
  }
};
// e^{row - max}, rows through the list, 64 columns: thread <-> (column tid % 64, k tid / 64 + 4 e)
template <typename TIn>
struct WeakColumns {
  const TIn *x;
  const float *mx;
  const int *list;
  int n0, C;
  float m[4];
  __device__ void fetch(int k0, int K, float (&v)[4]) {
    const int c = n0 + threadIdx.x % 64;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = k0 + threadIdx.x / 64 + 4 * e;
      const bool ok = k < K && c < C;
      v[e] = ok ? in_f32(x[(size_t)list[k] * C + c]) : -INFINITY;
      m[e] = ok ? mx[list[k]] : 0.f;
    }
  }
  __device__ void place(int, const float (&v)[4], WeakSlice &s) const {
#pragma unroll
    for (int e = 0; e < 4; ++e) s[threadIdx.x / 64 + 4 * e][threadIdx.x % 64] = expf(v[e] - m[e]);
  }
};

// A CTA takes 64 rows of lm (of am) and every lm_split-th (am_split-th) 64 columns; it leaves at once
// when the rows have nothing weak.  The frames (lattice rows) that some of its rows need are
// listed, kWeakList candidates at a time, and the product runs over the list.  64 x (100, 500) x
// 500: 4.5 us with nothing weak, 507 us with every cell weak (the whole gradient 750 us then; the
// FMA pipe for every cell 660); 16 x (59, 293) x 4233: 4.7 and 450 us (670; 660).  128 x 128 tiles
// without prefetch, as the FMA pipe's, took two to seven times as long for either kernel.
constexpr int kWeakList = 1024;
template <typename TIn>
__global__ void __launch_bounds__(kWeakThreads, 3)
weak_grads_kernel(const WeakGrads<TIn> g, int lm_split, int am_split) {
  __shared__ __align__(16) WeakSlice Xs[2], Ys[2];
  __shared__ int list[kWeakList], counts[8];
  const int tid = threadIdx.x, lane = tid & 31, tx = tid % 16, ty = tid / 16;
  const int words = weak_words(g.T);
  const int lm_tiles = (g.S1 + kWeakTile - 1) / kWeakTile, am_tiles = (g.T + kWeakTile - 1) / kWeakTile;
  const long long lm_ctas = (long long)g.B * lm_tiles * lm_split;
  const bool is_lm = blockIdx.x < lm_ctas;
  const int split = is_lm ? lm_split : am_split, tiles = is_lm ? lm_tiles : am_tiles;
  const int cta = (int)(is_lm ? blockIdx.x : blockIdx.x - lm_ctas), item = cta / split;
  const int b = item / tiles, m0 = kWeakTile * (item % tiles);
  const int M = is_lm ? g.S1 : g.T, depth = is_lm ? g.T : g.S1;
  const size_t lm0 = (size_t)b * g.S1, am0 = (size_t)b * g.T;
  bool cells = false, frames = false;
  const int end = is_lm ? min(m0 + kWeakTile, g.S1) : g.S1;
  for (int s = (is_lm ? m0 : 0) + tid; s < end; s += kWeakThreads) cells |= g.weak_row[lm0 + s];
  if (!is_lm && g.h != nullptr && tid < kWeakTile && m0 + tid < g.T)
    frames = am_only_weak(g.ammax[am0 + m0 + tid], g.amonly[am0 + m0 + tid]);
  cells = __syncthreads_or(cells);
  frames = __syncthreads_or(frames);
  if (!cells && !frames) return;
  const unsigned *weak = g.weak + lm0 * words;
  const float *rw = g.rw + lm0 * g.Tp;
  for (int n0 = (cta % split) * kWeakTile; n0 < g.C; n0 += split * kWeakTile) {
    float acc[4][4] = {};
    for (int d0 = 0; cells && d0 < depth; d0 += kWeakList) {
      int K = 0;
      for (int k0 = d0; k0 < min(depth, d0 + kWeakList); k0 += kWeakThreads) {
        const int k = k0 + tid;
        unsigned used = 0;
        if (k < depth) {
          if (is_lm) {
            for (int s = m0; s < end; ++s) used |= weak[(size_t)s * words + k / 32] >> (k % 32) & 1u;
          } else {
            used = weak[(size_t)k * words + m0 / 32];
            if (m0 / 32 + 1 < words) used |= weak[(size_t)k * words + m0 / 32 + 1];
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, used != 0);
        if (lane == 0) counts[tid >> 5] = __popc(m);
        __syncthreads();
        int at = K + __popc(m & ((1u << lane) - 1u));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i < tid >> 5) at += counts[i];
          K += counts[i];
        }
        if (used != 0) list[at] = k;
        __syncthreads();
      }
      WeakColumns<TIn> y{is_lm ? g.am + am0 * g.C : g.lm + lm0 * g.C, is_lm ? g.ammax + am0 : g.lmmax + lm0, list, n0,
                         g.C, {}};
      WeakWeights x{rw, weak, list, is_lm, m0, M, g.Tp, words, {}, {}};
      weak_product(x, y, K, Xs, Ys, acc);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + 4 * ty + i;
      if (m >= M) break;
      const size_t row = (is_lm ? lm0 : am0) + m;
      const float own_max = is_lm ? g.lmmax[row] : g.ammax[row];
      const TIn *own = (is_lm ? g.lm : g.am) + row * g.C;
      float *grad = (is_lm ? g.lm_grad : g.am_grad) + row * g.C;
      // the am-only term of a weak frame: h u[c] / Z
      const float frame = frames && am_only_weak(own_max, g.amonly[row]) ? g.h[row] * expf(own_max - g.amonly[row]) : 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = n0 + 4 * tx + j;
        if (c >= g.C) break;
        float v = acc[i][j];
        if (frame != 0.f) v += frame * g.uni[c];
        if (v != 0.f) grad[c] -= expf(in_f32(own[c]) - own_max) * v;
      }
    }
  }
}

// ---- lattice assembly -------------------------------------------------------------
struct SmoothCfg {
  int smoothed;
  // the am-only branch is left out: am_only_scale == 0.  The reference multiplies the
  // branch by 1e-20 in that case (rnnt_loss.py:1346-1351), which changes an fp32 / fp64
  // px or py only if that value is exactly 0; its three extra passes (unigram, am-only
  // normalizer) are not worth that
  int am_only_off;
  double both, ls, as;  // 1-l-a, lm-only scale, am-only scale (zero lm scale replaced by 1e-20)
  double delay_penalty = 0.0;  // added to px by the lattice-writing kernels when positive
};

template <typename real>
__global__ void assemble_kernel(const real *__restrict__ lm, const real *__restrict__ am,
                                const int64_t *__restrict__ symbols,
                                const int64_t *__restrict__ boundary, const real *__restrict__ norm,
                                const real *__restrict__ lmmax, const real *__restrict__ lmsum,
                                const real *__restrict__ amonly, const real *__restrict__ loguni,
                                real *__restrict__ px, real *__restrict__ py, int S, int T, int C,
                                int blank, int rnnt_type, SmoothCfg cfg) {
  const int b = blockIdx.z, s = blockIdx.y;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int S1 = S + 1;
  const int T1 = (rnnt_type == FRNNT_REGULAR) ? T + 1 : T;
  if (t > T) return;
  const real ninf = neg_inf<real>();
  const real both = (real)cfg.both, ls = (real)cfg.ls, as = (real)cfg.as;
  const real *lmrow = lm + ((size_t)b * S1 + s) * C;
  real lm_only_norm = 0;
  if (cfg.smoothed) lm_only_norm = log_r(lmsum[(size_t)b * S1 + s]) + lmmax[(size_t)b * S1 + s];

  // py at (s, t) and, for the constrained type, at (s+1, t)
  auto py_at = [&](int ss) -> real {
    const real *amrow = am + ((size_t)b * T + t) * C;
    const real *lr = lm + ((size_t)b * S1 + ss) * C;
    const real py_am = amrow[blank], py_lm = lr[blank];
    real v = py_am + py_lm - norm[((size_t)b * S1 + ss) * T + t];
    if (cfg.smoothed) {
      const real lnorm = log_r(lmsum[(size_t)b * S1 + ss]) + lmmax[(size_t)b * S1 + ss];
      const real v_lm = py_lm - lnorm;
      v = v * both + v_lm * ls;
      if (!cfg.am_only_off) v += (py_am + loguni[blank] - amonly[(size_t)b * T + t]) * as;
    }
    return v;
  };

  if (t < T) py[((size_t)b * S1 + s) * T + t] = py_at(s);

  if (s < S && t < T1) {
    int y = (int)symbols[(size_t)b * S + s];
    if (y < 0 || y >= C) y = blank;
    const real px_lm = lmrow[y];
    real px_am = ninf, v;
    if (t < T) {
      px_am = am[((size_t)b * T + t) * C + y];
      v = px_am + px_lm - norm[((size_t)b * S1 + s) * T + t];
    } else {
      v = px_am + px_lm;  // the -inf column of the regular type
    }
    if (cfg.smoothed) {
      const real v_lm = px_lm - lm_only_norm;
      v = v * both + v_lm * ls;
      if (!cfg.am_only_off) {
        real v_am = px_am + loguni[y];
        if (t < T) v_am -= amonly[(size_t)b * T + t];
        v += v_am * as;
      }
    }
    if (rnnt_type == FRNNT_REGULAR) {
      if (boundary != nullptr && (long long)t == (long long)boundary[4 * b + 3]) v = ninf;
    } else if (rnnt_type == FRNNT_CONSTRAINED) {
      v += py_at(s + 1);
    }
    if (cfg.delay_penalty > 0.0) v = add_rn(v, delay_penalty_at<real>(boundary, b, T, t, cfg.delay_penalty));
    px[((size_t)b * S + s) * T1 + t] = v;
  }
}

// ---- backward helpers -------------------------------------------------------------
// Gradients that actually reach the un-masked lattice entries:
//   gx: px_grad with the t = t_end column of the regular type dropped
//   gy: py_grad, plus px_grad[s-1] for the constrained type (px += py[s+1])
template <typename real>
struct EffGrads {
  const real *g_px, *g_py;
  const int64_t *boundary;
  int S, T, T1, rnnt_type;
  __device__ real gx(int b, int s, int t) const {
    if (s >= S || t >= T1) return 0;
    if (rnnt_type == FRNNT_REGULAR && boundary != nullptr &&
        (long long)t == (long long)boundary[4 * b + 3])
      return 0;
    return g_px[((size_t)b * S + s) * T1 + t];
  }
  __device__ real gy(int b, int s, int t) const {
    if (t >= T) return 0;
    real v = g_py[((size_t)b * (S + 1) + s) * T + t];
    if (rnnt_type == FRNNT_CONSTRAINED && s >= 1) v += g_px[((size_t)b * S + s - 1) * T1 + t];
    return v;
  }
};

// Rw[b,s,t] = both * (gx + gy) / (M + tiny),   1/(M+tiny) = e^{lmmax + ammax - N}
template <typename real>
__global__ void grad_weight_kernel(EffGrads<real> eg, const real *__restrict__ norm,
                                   const real *__restrict__ lmmax, const real *__restrict__ ammax,
                                   real *__restrict__ rw, real both, int Tp) {
  const int b = blockIdx.z, s = blockIdx.y;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= Tp) return;
  const size_t o = ((size_t)b * (eg.S + 1) + s) * Tp + t;
  if (t >= eg.T) {  // row padding
    rw[o] = 0;
    return;
  }
  const size_t i = ((size_t)b * (eg.S + 1) + s) * eg.T + t;
  const real w = both * (eg.gx(b, s, t) + eg.gy(b, s, t));
  const real inv = exp_r(lmmax[(size_t)b * (eg.S + 1) + s] + ammax[(size_t)b * eg.T + t] - norm[i]);
  rw[o] = (w == 0) ? (real)0 : w * inv;
}

// The two kernels above and below in one pass, for the tensor-core path: one CTA per lattice
// row (b, s) writes the row of Rw, the row sums of gx (all T1 columns) and gy, and the
// row's largest finite |Rw| (which sets the scale of the fp16 planes Rw is split into).  Weak cells
// (simple_pairs.cuh) do not go into the planes: their bits go to `weak`, weak_row says whether
// the row has any.
template <typename real>
__global__ void __launch_bounds__(128)
grad_weight_rows_kernel(EffGrads<real> eg, const real *__restrict__ norm, const real *__restrict__ lmmax,
                        const real *__restrict__ ammax, const real *__restrict__ lmsum,
                        const float *__restrict__ am_sum, real *__restrict__ rw, real *__restrict__ sgx,
                        real *__restrict__ sgy, float *__restrict__ rowmax, unsigned *__restrict__ weak,
                        uint8_t *__restrict__ weak_row, real both, int Tp) {
  __shared__ real red[3][4];
  const int row = blockIdx.x, b = row / (eg.S + 1), s = row % (eg.S + 1);
  const real lmx = lmmax[row];
  const float lms = (float)lmsum[row];
  const int words = weak_words(eg.T);
  bool any_weak = false;
  real ax = 0, ay = 0, mx = 0;
  const int n = max(Tp, eg.T1);
  for (int t0 = 0; t0 < n; t0 += 128) {
    const int t = t0 + threadIdx.x;
    bool is_weak = false;
    if (t < n) {
      const real gx = eg.gx(b, s, t), gy = eg.gy(b, s, t);
      ax += gx;
      ay += gy;
      if (t < Tp) {
        real v = 0;
        if (t < eg.T) {
          const real w = both * (gx + gy);
          const real inv = exp_r(lmx + ammax[(size_t)b * eg.T + t] - norm[(size_t)row * eg.T + t]);
          v = (w == 0) ? (real)0 : w * inv;
          // 1 / z against the bound; a cell without weight counts nowhere
          is_weak = w != 0 && (float)inv * weak_bound(lms, am_sum[(size_t)b * eg.T + t]) > 1.f;
        }
        rw[(size_t)row * Tp + t] = v;
        if (!is_weak && v - v == 0) mx = max(mx, v < 0 ? -v : v);
      }
    }
    const unsigned bits = __ballot_sync(0xffffffffu, is_weak);
    if ((threadIdx.x & 31) == 0 && t / 32 < words) weak[(size_t)row * words + t / 32] = bits;
    any_weak |= is_weak;
  }
  ax = warp_sum(ax);
  ay = warp_sum(ay);
  mx = warp_max(mx);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) red[0][w] = ax, red[1][w] = ay, red[2][w] = mx;
  any_weak = __syncthreads_or(any_weak);
  if (threadIdx.x == 0) {
    weak_row[row] = any_weak;
    sgx[row] = (red[0][0] + red[0][1]) + (red[0][2] + red[0][3]);
    sgy[row] = (red[1][0] + red[1][1]) + (red[1][2] + red[1][3]);
    rowmax[row] = (float)max(max(red[2][0], red[2][1]), max(red[2][2], red[2][3]));
  }
}

// one warp per (b, s): sums over t of gx (all T1 columns) and gy
template <typename real>
__global__ void grad_row_sums_kernel(EffGrads<real> eg, real *__restrict__ sgx,
                                     real *__restrict__ sgy, int B) {
  const int lane = threadIdx.x & 31;
  const int row = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (row >= B * (eg.S + 1)) return;
  const int b = row / (eg.S + 1), s = row % (eg.S + 1);
  real ax = 0, ay = 0;
  for (int t = lane; t < eg.T1; t += 32) {
    ax += eg.gx(b, s, t);
    ay += eg.gy(b, s, t);
  }
  ax = warp_sum(ax);
  ay = warp_sum(ay);
  if (lane == 0) {
    sgx[row] = ax;
    sgy[row] = ay;
  }
}

// sums over s for 32 frames per CTA: lane <-> frame, the 8 warps take every 8th row
// each (contiguous 128-byte loads, all of a warp's rows independent), then the eight
// partial sums are added in warp order
constexpr int kColSumWarps = 8;
template <typename real>
__global__ void __launch_bounds__(32 * kColSumWarps)
grad_col_sums_kernel(EffGrads<real> eg, real *__restrict__ cgx, real *__restrict__ cgy, int B) {
  __shared__ real px_part[kColSumWarps][32], py_part[kColSumWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b = blockIdx.y, t = blockIdx.x * 32 + lane;
  real ax = 0, ay = 0;
  if (t < eg.T) {
#pragma unroll 4
    for (int s = w; s <= eg.S; s += kColSumWarps) {
      ax += eg.gx(b, s, t);
      ay += eg.gy(b, s, t);
    }
  }
  px_part[w][lane] = ax;
  py_part[w][lane] = ay;
  __syncthreads();
  if (w == 0 && t < eg.T) {
    ax = px_part[0][lane];
    ay = py_part[0][lane];
    for (int q = 1; q < kColSumWarps; ++q) {
      ax += px_part[q][lane];
      ay += py_part[q][lane];
    }
    cgx[(size_t)b * eg.T + t] = ax;
    cgy[(size_t)b * eg.T + t] = ay;
  }
}

// v[i] = alpha * (a[i] + b[i])
template <typename real>
__global__ void scaled_sum_kernel(const real *a, const real *b, real *v, real alpha, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = alpha * (a[i] + b[i]);
}

// one-hot terms of lm_grad: symbol column gets cx*sgx, blank column gets cx*sgy
template <typename real>
__global__ void lm_onehot_kernel(const int64_t *__restrict__ symbols, const real *__restrict__ sgx,
                                 const real *__restrict__ sgy, real *__restrict__ lm_grad, int B,
                                 int S, int C, int blank, real coef) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= B * (S + 1)) return;
  const int b = row / (S + 1), s = row % (S + 1);
  real *g = lm_grad + (size_t)row * C;
  if (s < S) {
    int y = (int)symbols[(size_t)b * S + s];
    if (y < 0 || y >= C) y = blank;
    g[y] += coef * sgx[row];
  }
  g[blank] += coef * sgy[row];
}

// one-hot terms of am_grad: for every s the symbol column gets coef*gx[s][t]; blank gets coef*cgy[t]
template <typename real>
__global__ void am_onehot_kernel(EffGrads<real> eg, const int64_t *__restrict__ symbols,
                                 const real *__restrict__ cgy, real *__restrict__ am_grad, int B,
                                 int C, int blank, real coef) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= B * eg.T) return;
  const int b = idx / eg.T, t = idx % eg.T;
  real *g = am_grad + (size_t)idx * C;
  // fire-and-forget adds: this thread owns row (b, t), and adds issued by one
  // thread to one address are applied in program order, so the sum is deterministic.
  // Eight gradient loads are issued before their adds (the adds would otherwise keep
  // the next load from starting).
  for (int s0 = 0; s0 < eg.S; s0 += 8) {
    real v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = s0 + u < eg.S ? eg.gx(b, s0 + u, t) : (real)0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (s0 + u >= eg.S || v[u] == 0) continue;
      int y = (int)symbols[(size_t)b * eg.S + s0 + u];
      if (y < 0 || y >= C) y = blank;
      atomicAdd(&g[y], coef * v[u]);
    }
  }
  atomicAdd(&g[blank], coef * cgy[idx]);
}

// d loss / d log-unigram[c] = as * ( sum_{b,s: y_bs = c} sgx[b,s]  +  [c = blank] sum_{b,s} sgy[b,s] )
// then dP[c] = (dlogu[c] / u[c] - du[c]) / rows      (du holds +sum h A / Z)
constexpr int kUniRows = 128;  // threads per CTA, too
template <typename real>
__global__ void __launch_bounds__(kUniRows) unigram_grad_kernel(const int64_t *__restrict__ symbols,
                                    const real *__restrict__ sgx, const real *__restrict__ sgy,
                                    const real *__restrict__ du_partial, int nchunk,
                                    const real *__restrict__ uni, real *__restrict__ dp, int B,
                                    int S, int C, int blank, real as) {
  // The rows go through shared memory, 128 at a time (symbol or -1, and the two sums): read from
  // global memory by every thread they cost one dependent load after the other: 109 us for
  // 16 x 60 rows and 147 partials, 33 us this way with eight partials in flight.
  __shared__ int sym[kUniRows];
  __shared__ real sx[kUniRows], sy[kUniRows];
  const int c = blockIdx.x * kUniRows + threadIdx.x;
  const int rows = B * (S + 1);
  real acc = 0;
  for (int r0 = 0; r0 < rows; r0 += kUniRows) {
    const int row = r0 + threadIdx.x;
    if (row < rows) {
      const int b = row / (S + 1), s = row % (S + 1);
      int y = -1;
      if (s < S) {
        const long long q = symbols[(size_t)b * S + s];
        y = q < 0 || q >= C ? blank : (int)q;
      }
      sym[threadIdx.x] = y;
      sx[threadIdx.x] = sgx[row];
      sy[threadIdx.x] = sgy[row];
    }
    __syncthreads();
    const int n = min(kUniRows, rows - r0);
#pragma unroll 8
    for (int i = 0; i < n; ++i) {
      if (sym[i] == c) acc += sx[i];
      if (c == blank) acc += sy[i];
    }
    __syncthreads();
  }
  if (c >= C) return;
  real du = 0;
  for (int j0 = 0; j0 < nchunk; j0 += 8) {
    real v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = j0 + u < nchunk ? du_partial[(size_t)(j0 + u) * C + c] : (real)0;
#pragma unroll
    for (int u = 0; u < 8; ++u) du += v[u];
  }
  dp[c] = (as * acc / uni[c] - du) / (real)((long long)B * (S + 1));
}

// one warp per lm row: rowdot = sum_c softmax(lm row)[c] * dP[c]
template <typename real>
__global__ void row_dot_kernel(const real *__restrict__ lm, const real *__restrict__ lmmax,
                               const real *__restrict__ lmsum, const real *__restrict__ dp,
                               real *__restrict__ rowdot, long long rows, int C) {
  const int lane = threadIdx.x & 31;
  const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= rows) return;
  const real *src = lm + row * (long long)C;
  const real m = lmmax[row];
  real acc = 0;
#pragma unroll 8
  for (int c = lane; c < C; c += 32) acc += exp_r(src[c] - m) * dp[c];
  acc = warp_sum(acc);
  if (lane == 0) rowdot[row] = acc / lmsum[row];
}

// The same sum and what it stands for, lm_grad[row][c] += P[row][c] (dP[c] - rowdot[row]), for the
// tensor-core path: one CTA per lm row, which the second pass finds in the caches.  P in
// float32: dP[c] goes up to 1 / (rows u[c]) for a symbol that is improbable in every row, where
// the planes would lose P.
__global__ void __launch_bounds__(256)
lm_unigram_grad_kernel(const float *__restrict__ lm, const float *__restrict__ lmmax,
                       const float *__restrict__ lmsum, const float *__restrict__ dp,
                       float *__restrict__ lm_grad, int C) {
  __shared__ float part[8];
  const long long row = blockIdx.x;
  const float *src = lm + row * C;
  float *dst = lm_grad + row * C;
  const float m = lmmax[row], sum = lmsum[row];
  float acc = 0.f;
#pragma unroll 4
  for (int c = threadIdx.x; c < C; c += 256) acc += expf(src[c] - m) * dp[c];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  acc = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) acc += part[w];
  const float rowdot = acc / sum;
#pragma unroll 4
  for (int c = threadIdx.x; c < C; c += 256) dst[c] += expf(src[c] - m) / sum * (dp[c] - rowdot);
}

// tensor-core (tcgen05, 3xTF32) contraction, FRNNT_CONTRACTION=tf32 or tall constrained lattices:
// float32 with 16-byte aligned rows; what else the fp16-pair engine does not take (float64,
// tall constrained lattices with an odd vocabulary) runs on the SIMT path.  The
// environment variable FRNNT_CONTRACTION=simt forces the SIMT path (for tests).
bool norm_umma_supported(const void *lm, const void *am, int S1, int T, int C);
int launch_norm_umma(const float *lm, const float *am, const float *lmmax, const float *ammax,
                     float *norm, int B, int S1, int T, int C, cudaStream_t st);
int launch_simple_grads_umma(const float *lm, const float *am, const float *lmmax,
                             const float *lmsum, const float *ammax, const float *amonly,
                             const float *uni, const float *rw, const float *gl, const float *h,
                             const float *dp, const float *rowdot, float *lm_grad, float *am_grad,
                             int B, int S1, int T, int C, int Tp, cudaStream_t st);

// buffers of the caller's that only the FMA pipe, which moves single values, can work in
static bool off_16_bytes(const void *saved, const void *scratch) {
  return (uintptr_t)saved % 16 != 0 || (uintptr_t)scratch % 16 != 0;
}

template <typename real>
static bool use_tensor_cores(const void *lm, const void *am, const void *saved, const void *scratch, int S1, int T,
                             int C) {
  if (sizeof(real) != 4 || off_16_bytes(saved, scratch)) return false;
  const char *mode = getenv("FRNNT_CONTRACTION");
  if (mode != nullptr && strcmp(mode, "simt") == 0) return false;
  return norm_umma_supported(lm, am, S1, T, C);
}

// the fp16-pair engine (FRNNT_CONTRACTION=tf32 keeps the 3xTF32 kernels, =simt the FMA pipe)
template <typename real>
static bool use_pairs(const void *lm, const void *am, const void *saved, const void *scratch, int S1, int T, int C,
                      int rnnt_type) {
  if (sizeof(real) != 4 || off_16_bytes(saved, scratch)) return false;
  const char *mode = getenv("FRNNT_CONTRACTION");
  if (mode != nullptr && (strcmp(mode, "simt") == 0 || strcmp(mode, "tf32") == 0)) return false;
  return simple_pairs_supported(lm, am, S1, T, C, rnnt_type);
}

static int simple_check(int dtype, int B, int S, int T, int C, int blank, int rnnt_type) {
  FRNNT_REQUIRE(check_dtype(dtype) || is_half_input(dtype), FRNNT_EINVAL,
                "dtype must be FRNNT_F32, FRNNT_F64, or FRNNT_F16 / FRNNT_BF16 for 16-bit lm and am");
  FRNNT_REQUIRE(B >= 0 && S >= 0 && T >= 0 && C >= 1, FRNNT_EINVAL,
                "bad sizes B=%d S=%d T=%d C=%d", B, S, T, C);
  FRNNT_REQUIRE(blank >= 0 && blank < C, FRNNT_EINVAL, "blank=%d outside [0,%d)", blank, C);
  FRNNT_REQUIRE(rnnt_type >= 0 && rnnt_type <= 2, FRNNT_EINVAL, "bad rnnt_type %d", rnnt_type);
  FRNNT_REQUIRE(B <= 65535 && S + 1 <= 65535, FRNNT_EUNSUPPORTED, "B or S too large for the grid");
  return FRNNT_OK;
}

static SmoothCfg make_cfg(int smoothed, double lm_only_scale, double am_only_scale) {
  SmoothCfg cfg;
  cfg.smoothed = smoothed;
  cfg.both = 1.0 - lm_only_scale - am_only_scale;
  // exact zeros would turn -inf * 0 into nan (rnnt_loss.py:1346-1351)
  cfg.ls = lm_only_scale == 0.0 ? 1.0e-20 : lm_only_scale;
  cfg.am_only_off = smoothed && am_only_scale == 0.0;
  cfg.as = am_only_scale;
  if (!smoothed) {
    cfg.both = 1.0;
    cfg.ls = 0.0;
    cfg.as = 0.0;
  }
  return cfg;
}

static inline int warps_grid(long long rows) {
  long long want = (rows + 7) / 8;
  if (want < 1) want = 1;
  return (int)(want < (long long)sm_count() * 32 ? want : (long long)sm_count() * 32);
}

template <typename real>
static int simple_forward_impl(const void *lm_, const void *am_, const int64_t *symbols,
                               const int64_t *boundary, int blank, int rnnt_type, SmoothCfg cfg,
                               void *px, void *py, void *saved, void *scratch, int B, int S, int T,
                               int C, cudaStream_t st, int input_dtype = FRNNT_F32) {
  const real *lm = (const real *)lm_, *am = (const real *)am_;  // not dereferenced for 16-bit inputs
  const int S1 = S + 1;
  SavedLayout sv(sizeof(real), B, S, T, C);
  ScratchLayout sc(sizeof(real), B, S, T, C);
  char *svb = (char *)saved, *scb = (char *)scratch;
  real *norm = (real *)(svb + sv.norm), *lmmax = (real *)(svb + sv.lmmax);
  real *lmsum = (real *)(svb + sv.lmsum), *ammax = (real *)(svb + sv.ammax);
  real *amonly = (real *)(svb + sv.amonly), *uni = (real *)(svb + sv.uni);
  real *loguni = (real *)(svb + sv.loguni), *partial = (real *)(scb + sc.partial);
  const long long lm_rows = (long long)B * S1, am_rows = (long long)B * T;

  const bool pairs = use_pairs<real>(lm, am, saved, nullptr, S1, T, C, rnnt_type);
  FRNNT_REQUIRE(!is_half_input(input_dtype) || (pairs && (!cfg.smoothed || cfg.am_only_off)), FRNNT_EUNSUPPORTED,
                "16-bit inputs are read by the tensor-core path without the am-only branch only "
                "(frnnt_simple_reads_16bit_inputs)");
  void *pairs_saved = svb + sv.total;
  if (pairs) {
    int rc0 = launch_simple_forward_pairs(lm_, am_, symbols, boundary, blank,
                                          rnnt_type, cfg.smoothed, cfg.am_only_off, (float)cfg.both,
                                          (float)cfg.ls, (float)cfg.as, (float *)px, (float *)py, (float *)norm,
                                          (float *)lmmax, (float *)lmsum, (float *)ammax, (const float *)amonly,
                                          (const float *)loguni, pairs_saved, B, S, T, C, 0, st, cfg.delay_penalty,
                                          input_dtype);
    if (rc0 != FRNNT_OK) return rc0;
  } else {
    FRNNT_KERNEL(row_stats_kernel<real><<<warps_grid(lm_rows), 256, 0, st>>>(lm, lmmax, lmsum, lm_rows, C));
    constexpr int VW = 16 / sizeof(real);
    const int vec_ok = C % VW == 0 && (uintptr_t)am % 16 == 0;
    FRNNT_KERNEL(row_max_kernel<real><<<warps_grid(am_rows), 256, 0, st>>>(am, ammax, am_rows, C, vec_ok));
  }
  FRNNT_CUDA(cudaGetLastError());
  if (cfg.smoothed && !cfg.am_only_off) {
    const int nchunk = (int)((lm_rows + kColChunkRows - 1) / kColChunkRows);
    dim3 g1((unsigned)((C + 127) / 128), (unsigned)nchunk);
    FRNNT_KERNEL(column_partial_kernel<real, 0><<<g1, 128, 0, st>>>(lm, lmmax, lmsum, nullptr, partial, lm_rows, C));
    FRNNT_KERNEL(unigram_final_kernel<real><<<(C + 127) / 128, 128, 0, st>>>(partial, nchunk, lm_rows, C, uni, loguni));
    FRNNT_KERNEL(am_only_norm_kernel<real><<<warps_grid(am_rows), 256, 0, st>>>(am, ammax, uni, amonly, am_rows, C));
    FRNNT_CUDA(cudaGetLastError());
  }
  int rc;
  if (pairs)
    return launch_simple_forward_pairs(lm_, am_, symbols, boundary, blank,
                                       rnnt_type, cfg.smoothed, cfg.am_only_off, (float)cfg.both,
                                       (float)cfg.ls, (float)cfg.as, (float *)px, (float *)py, (float *)norm,
                                       (float *)lmmax, (float *)lmsum, (float *)ammax, (const float *)amonly,
                                       (const float *)loguni, pairs_saved, B, S, T, C, 1, st, cfg.delay_penalty,
                                       input_dtype);
  if (use_tensor_cores<real>(lm, am, saved, nullptr, S1, T, C)) {
    rc = launch_norm_umma((const float *)lm, (const float *)am, (const float *)lmmax,
                          (const float *)ammax, (float *)norm, B, S1, T, C, st);
  } else {
    NormProb<real> prob{lm, am, lmmax, ammax, norm, S1, T, C};
    rc = launch_contraction<real>(prob, S1, T, B, st);
  }
  if (rc != FRNNT_OK) return rc;
  dim3 g2((unsigned)((T + 1 + 127) / 128), (unsigned)S1, (unsigned)B);
  FRNNT_KERNEL(assemble_kernel<real><<<g2, 128, 0, st>>>(lm, am, symbols, boundary, norm, lmmax, lmsum, amonly,
                                            loguni, (real *)px, (real *)py, S, T, C, blank,
                                            rnnt_type, cfg));
  FRNNT_CUDA(cudaGetLastError());
  return FRNNT_OK;
}

template <typename real>
static int simple_backward_impl(const void *lm_, const void *am_, const int64_t *symbols,
                                const int64_t *boundary, int blank, int rnnt_type, SmoothCfg cfg,
                                int am_only_active, const void *px_grad, const void *py_grad,
                                const void *saved, void *scratch, void *lm_grad_, void *am_grad_,
                                int B, int S, int T, int C, cudaStream_t st, int input_dtype) {
  const real *lm = (const real *)lm_, *am = (const real *)am_;  // 16-bit inputs: only weak_grads_kernel reads them
  real *lm_grad = (real *)lm_grad_, *am_grad = (real *)am_grad_;
  const int S1 = S + 1;
  const int T1 = rnnt_type == FRNNT_REGULAR ? T + 1 : T;
  SavedLayout sv(sizeof(real), B, S, T, C);
  ScratchLayout sc(sizeof(real), B, S, T, C);
  const char *svb = (const char *)saved;
  char *scb = (char *)scratch;
  const real *norm = (const real *)(svb + sv.norm), *lmmax = (const real *)(svb + sv.lmmax);
  const real *lmsum = (const real *)(svb + sv.lmsum), *ammax = (const real *)(svb + sv.ammax);
  const real *amonly = (const real *)(svb + sv.amonly), *uni = (const real *)(svb + sv.uni);
  real *rw = (real *)(scb + sc.rw), *sgx = (real *)(scb + sc.sgx), *sgy = (real *)(scb + sc.sgy);
  real *cgx = (real *)(scb + sc.cgx), *cgy = (real *)(scb + sc.cgy);
  real *gl = (real *)(scb + sc.gl), *h = (real *)(scb + sc.h);
  real *partial = (real *)(scb + sc.partial), *dp = (real *)(scb + sc.dp);
  real *rowdot = (real *)(scb + sc.rowdot);
  const long long lm_rows = (long long)B * S1, am_rows = (long long)B * T;
  EffGrads<real> eg{(const real *)px_grad, (const real *)py_grad, boundary, S, T, T1, rnnt_type};

  const int Tp = rw_pitch(T);
  const bool pairs = use_pairs<real>(lm, am, saved, scratch, S1, T, C, rnnt_type) && T > 0;
  dim3 g3((unsigned)((Tp + 127) / 128), (unsigned)S1, (unsigned)B);
  const float *am_sum = (const float *)(svb + sv.total + simple_pairs_amsum_offset(B, S, T, C));
  unsigned *weak = (unsigned *)(scb + sc.weak);
  uint8_t *weak_row = (uint8_t *)(scb + sc.weak_row);
  if (pairs) {
    // one pass: Rw, the row sums and the row maxima of |Rw| (first floats of the pairs scratch)
    FRNNT_KERNEL(grad_weight_rows_kernel<real><<<(unsigned)lm_rows, 128, 0, st>>>(
        eg, norm, lmmax, ammax, lmsum, am_sum, rw, sgx, sgy,
        (float *)(scb + sc.total + simple_pairs_rowmax_offset(B, S, T, C)), weak, weak_row, (real)cfg.both, Tp));
  } else {
    if (T > 0)
      FRNNT_KERNEL(grad_weight_kernel<real><<<g3, 128, 0, st>>>(eg, norm, lmmax, ammax, rw, (real)cfg.both, Tp));
    FRNNT_KERNEL(grad_row_sums_kernel<real><<<(int)((lm_rows * 32 + 255) / 256), 256, 0, st>>>(eg, sgx, sgy, B));
  }
  if (T > 0)
    FRNNT_KERNEL(grad_col_sums_kernel<real><<<dim3((unsigned)((T + 31) / 32), (unsigned)B), 32 * kColSumWarps, 0,
                                              st>>>(eg, cgx, cgy, B));
  FRNNT_CUDA(cudaGetLastError());

  const real *gl_p = nullptr, *h_p = nullptr, *dp_p = nullptr, *rowdot_p = nullptr;
  if (cfg.smoothed) {
    // gl[b,s] = ls * (sgx + sgy);  h[b,t] = as * (cgx + cgy)
    FRNNT_KERNEL(scaled_sum_kernel<real><<<(int)((lm_rows + 255) / 256), 256, 0, st>>>(sgx, sgy, gl, (real)cfg.ls,
                                                                      lm_rows));
    gl_p = gl;
    if (am_only_active && T > 0) {
      FRNNT_KERNEL(scaled_sum_kernel<real><<<(int)((am_rows + 255) / 256), 256, 0, st>>>(cgx, cgy, h, (real)cfg.as,
                                                                        am_rows));
      h_p = h;
      const int nchunk = (int)((am_rows + kColChunkRows - 1) / kColChunkRows);
      dim3 g1((unsigned)((C + 127) / 128), (unsigned)nchunk);
      FRNNT_KERNEL(column_partial_kernel<real, 1><<<g1, 128, 0, st>>>(am, ammax, amonly, h, partial, am_rows, C));
      FRNNT_KERNEL(unigram_grad_kernel<real><<<(C + kUniRows - 1) / kUniRows, kUniRows, 0, st>>>(symbols, sgx, sgy, partial, nchunk,
                                                            uni, dp, B, S, C, blank, (real)cfg.as));
      if (!pairs)
        FRNNT_KERNEL(row_dot_kernel<real><<<(int)((lm_rows * 32 + 255) / 256), 256, 0, st>>>(lm, lmmax, lmsum, dp,
                                                                           rowdot, lm_rows, C));
      dp_p = dp;
      rowdot_p = rowdot;
    }
    FRNNT_CUDA(cudaGetLastError());
  }

  int rc;
  if (pairs) {
    rc = launch_simple_grads_pairs((const float *)rw, weak, (const float *)lmsum, (const float *)ammax,
                                   (const float *)amonly, (const float *)uni, (const float *)gl_p,
                                   (const float *)h_p, (float *)lm_grad, (float *)am_grad, svb + sv.total,
                                   scb + sc.total, B, S, T, C, Tp,
                                   simple_pairs_exact(lm_, am_, C, input_dtype), st);
    if (rc != FRNNT_OK) return rc;
    if (dp_p != nullptr)
      FRNNT_KERNEL(lm_unigram_grad_kernel<<<(unsigned)lm_rows, 256, 0, st>>>(
          (const float *)lm, (const float *)lmmax, (const float *)lmsum, (const float *)dp_p, (float *)lm_grad, C));
    // four CTAs per SM for either side, where there are as many: a tile's columns over several
    // (eight: 6% faster where everything is weak, 7 instead of 4.5 us where nothing is)
    const long long tiles_c = (C + kWeakTile - 1) / kWeakTile, most = (long long)sm_count() * 4;
    const long long lm_items = (long long)B * ((S1 + kWeakTile - 1) / kWeakTile);
    const long long am_items = (long long)B * ((T + kWeakTile - 1) / kWeakTile);
    const int lm_split = (int)std::min(tiles_c, std::max(1LL, most / lm_items));
    const int am_split = (int)std::min(tiles_c, std::max(1LL, most / am_items));
    const unsigned ctas = (unsigned)(lm_items * lm_split + am_items * am_split);
    with_input_type(input_dtype, lm_, am_, [&](auto *l, auto *a) {
      using TIn = std::remove_const_t<std::remove_pointer_t<decltype(l)>>;
      const WeakGrads<TIn> g{l, a, (const float *)rw, weak, weak_row, (const float *)lmmax, (const float *)ammax,
                             (const float *)amonly, (const float *)h_p, (const float *)uni, (float *)lm_grad,
                             (float *)am_grad, B, S1, T, C, Tp};
      FRNNT_KERNEL(weak_grads_kernel<<<ctas, kWeakThreads, 0, st>>>(g, lm_split, am_split));
    });
    FRNNT_CUDA(cudaGetLastError());
  } else if (use_tensor_cores<real>(lm, am, saved, scratch, S1, T, C)) {
    rc = launch_simple_grads_umma((const float *)lm, (const float *)am, (const float *)lmmax,
                                  (const float *)lmsum, (const float *)ammax, (const float *)amonly,
                                  (const float *)uni, (const float *)rw, (const float *)gl_p,
                                  (const float *)h_p, (const float *)dp_p, (const float *)rowdot_p,
                                  (float *)lm_grad, (float *)am_grad, B, S1, T, C, Tp, st);
    if (rc != FRNNT_OK) return rc;
  } else {
    LmGradProb<real> p1{rw, am, ammax, lm, lmmax, lmsum, gl_p, dp_p, rowdot_p, lm_grad, S1, T, C, Tp};
    rc = launch_contraction<real>(p1, S1, C, B, st);
    if (rc != FRNNT_OK) return rc;
    AmGradProb<real> p2{rw, lm, lmmax, am, ammax, h_p, uni, amonly, am_grad, S1, T, C, Tp};
    rc = launch_contraction<real>(p2, T, C, B, st);
    if (rc != FRNNT_OK) return rc;
  }

  const real coef_lm = (real)cfg.both + (real)cfg.ls;
  const real coef_am = (real)cfg.both + (am_only_active || !cfg.smoothed ? (real)cfg.as : (real)0);
  FRNNT_KERNEL(lm_onehot_kernel<real><<<(int)((lm_rows + 127) / 128), 128, 0, st>>>(symbols, sgx, sgy, lm_grad, B, S, C,
                                                                   blank, coef_lm));
  FRNNT_KERNEL(am_onehot_kernel<real><<<(int)((am_rows + 127) / 128), 128, 0, st>>>(eg, symbols, cgy, am_grad, B, C,
                                                                   blank, coef_am));
  FRNNT_CUDA(cudaGetLastError());
  return FRNNT_OK;
}

}  // namespace frnnt

using namespace frnnt;

// float32 calls may take the tensor-core path, whose planes and tables follow the regular areas
extern "C" size_t frnnt_simple_saved_bytes(int dtype, int B, int S, int T, int C) {
  if (is_half_input(dtype)) dtype = FRNNT_F32;
  if (!check_dtype(dtype) || B < 0 || S < 0 || T < 0 || C < 0) return 0;
  return SavedLayout(dtype_size(dtype), B, S, T, C).total +
         (dtype == FRNNT_F32 ? SimplePairsLayout(B, S, T, C).saved_bytes : 0);
}

extern "C" size_t frnnt_simple_scratch_bytes(int dtype, int B, int S, int T, int C) {
  if (is_half_input(dtype)) dtype = FRNNT_F32;
  if (!check_dtype(dtype) || B < 0 || S < 0 || T < 0 || C < 0) return 0;
  return ScratchLayout(dtype_size(dtype), B, S, T, C).total +
         (dtype == FRNNT_F32 ? SimplePairsLayout(B, S, T, C).scratch_bytes : 0);
}

extern "C" int frnnt_simple_reads_16bit_inputs(int S, int T, int C, int rnnt_type, int smoothed,
                                               double am_only_scale) {
  if (S < 0 || T < 1 || C < 1) return 0;
  if (smoothed && am_only_scale != 0.0) return 0;
  // 256-byte aligned rows stand in for the caller's tensors (torch's allocations are)
  return use_pairs<float>((const void *)256, (const void *)256, nullptr, nullptr, S + 1, T, C, rnnt_type) ? 1 : 0;
}

extern "C" int frnnt_simple_logprobs_forward(int dtype, const void *lm, const void *am,
                                             const int64_t *symbols, const int64_t *boundary,
                                             int blank, int rnnt_type, int smoothed,
                                             double lm_only_scale, double am_only_scale,
                                             double delay_penalty, void *px, void *py, void *saved,
                                             void *scratch, int B, int S, int T, int C, void *stream) {
  int rc = simple_check(dtype, B, S, T, C, blank, rnnt_type);
  if (rc != FRNNT_OK) return rc;
  if (B == 0) return FRNNT_OK;
  FRNNT_REQUIRE(lm && (am || T == 0) && (symbols || S == 0) && py && (px || S == 0) && saved &&
                    scratch,
                FRNNT_EINVAL, "NULL argument");
  SmoothCfg cfg = make_cfg(smoothed, lm_only_scale, am_only_scale);
  cfg.delay_penalty = delay_penalty > 0.0 ? delay_penalty : 0.0;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype != FRNNT_F64)
    return simple_forward_impl<float>(lm, am, symbols, boundary, blank, rnnt_type, cfg, px, py,
                                      saved, scratch, B, S, T, C, st, dtype);
  return simple_forward_impl<double>(lm, am, symbols, boundary, blank, rnnt_type, cfg, px, py,
                                     saved, scratch, B, S, T, C, st);
}

extern "C" int frnnt_simple_logprobs_backward(int dtype, const void *lm, const void *am,
                                              const int64_t *symbols, const int64_t *boundary,
                                              int blank, int rnnt_type, int smoothed,
                                              double lm_only_scale, double am_only_scale,
                                              const void *px_grad, const void *py_grad,
                                              const void *saved, void *scratch, void *lm_grad,
                                              void *am_grad, int B, int S, int T, int C,
                                              void *stream) {
  int rc = simple_check(dtype, B, S, T, C, blank, rnnt_type);
  if (rc != FRNNT_OK) return rc;
  if (B == 0) return FRNNT_OK;
  FRNNT_REQUIRE(lm && (am || T == 0) && (symbols || S == 0) && py_grad && (px_grad || S == 0) &&
                    saved && scratch && lm_grad && (am_grad || T == 0),
                FRNNT_EINVAL, "NULL argument");
  SmoothCfg cfg = make_cfg(smoothed, lm_only_scale, am_only_scale);
  // With am_only_scale == 0 the reference still scales the am-only branch by 1e-20; its
  // gradient (<= 1e-19 relative) is below the resolution of either dtype and is skipped.
  const int am_only_active = smoothed && am_only_scale != 0.0;
  cudaStream_t st = (cudaStream_t)stream;
  if (is_half_input(dtype)) {
    FRNNT_REQUIRE(use_pairs<float>(lm, am, saved, scratch, S + 1, T, C, rnnt_type) && T > 0 && !am_only_active,
                  FRNNT_EUNSUPPORTED, "16-bit inputs: see frnnt_simple_reads_16bit_inputs");
  }
  if (dtype != FRNNT_F64)
    return simple_backward_impl<float>(lm, am, symbols, boundary, blank, rnnt_type, cfg,
                                       am_only_active, px_grad, py_grad, saved, scratch, lm_grad,
                                       am_grad, B, S, T, C, st, dtype);
  return simple_backward_impl<double>(lm, am, symbols, boundary, blank, rnnt_type, cfg,
                                      am_only_active, px_grad, py_grad, saved, scratch, lm_grad,
                                      am_grad, B, S, T, C, st, dtype);
}
