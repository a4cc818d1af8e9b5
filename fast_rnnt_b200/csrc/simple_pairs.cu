// The "simple" lattices (get_rnnt_logprobs / get_rnnt_logprobs_smoothed,
// fast_rnnt/python/fast_rnnt/rnnt_loss.py:66-227 and :1135-1369) on the fp16-pair
// tensor-core engine (umma_pairs.cuh), float32 path:
//
//   forward   one pass over lm and am takes the row maxima and writes
//             exp(x - rowmax) as fp16 planes (the operands of every product below; they
//             are kept for the backward) plus a few per-row scalars;
//             N^T[t][s] = sum_c A[t][c] L[s][c] per utterance on the tensor cores (TMA-fed),
//             whose epilogue takes the log, adds the maxima back, gathers am[t][symbol],
//             am[t][blank], applies the smoothing interpolation, the -inf at t_end and
//             px += py[s+1] (constrained) and writes the normalizer, px and py -- lane <->
//             frame, so every store is a coalesced row segment of the [s][t] lattices
//             (rnnt_loss.py:174-227, :1296-1367);
//   backward  the gradient weights Rw[s][t] (simple.cu) become planes, and
//             dlm[s][c] = -L[s][c] * sum_t Rw[s][t] A[t][c],
//             dam[t][c] = -A[t][c] * sum_s Rw[s][t] L[s][c]
//             run on the same engine, L and A read back from the planes in the epilogue;
//   weak cells (simple_pairs.cuh) are computed in float32, forward and backward.
#include <cuda_fp16.h>

#include <type_traits>

#include "lsm_band.cuh"
#include "simple_pairs.cuh"
#include "umma_pairs.cuh"

namespace frnnt {

constexpr float kExpScale = 16384.f;             // exp(x - max) <= 1
constexpr float kExpInv2 = 1.f / (16384.f * 16384.f);
constexpr int kSpParts = 1024;

static inline size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

SimplePairsLayout::SimplePairsLayout(int B, int S, int T, int C) {
  const size_t S1 = (size_t)S + 1;
  Cp = (C + 63) / 64 * 64;
  Tq = (T + 63) / 64 * 64;
  Sp = (S + 31) / 32 * 32;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t r = o;
    o += up256(bytes);
    return r;
  };
  lp_hi = take((size_t)B * S1 * Cp * 2);
  lp_lo = take((size_t)B * S1 * Cp * 2);
  ap_hi = take((size_t)B * T * Cp * 2);
  ap_lo = take((size_t)B * T * Cp * 2);
  lm_blk = take((size_t)B * S1 * 4);
  lm_sym = take((size_t)B * S1 * 4);
  lnorm = take((size_t)B * S1 * 4);
  am_blk = take((size_t)B * T * 4);
  am_sym = take((size_t)B * T * Sp * 4);
  am_sum = take((size_t)B * T * 4);
  weak = take((size_t)B * ((S1 + kPairTile - 1) / kPairTile) * T);
  saved_bytes = o;
  o = 0;
  rw_hi = take((size_t)B * S1 * Tq * 2);
  rw_lo = take((size_t)B * S1 * Tq * 2);
  parts = take(std::max<size_t>(kSpParts, (size_t)B * S1) * 4);
  inv_scale = take((size_t)B * 4);
  scratch_bytes = o;
}

size_t simple_pairs_rowmax_offset(int B, int S, int T, int C) { return SimplePairsLayout(B, S, T, C).parts; }
size_t simple_pairs_amsum_offset(int B, int S, int T, int C) { return SimplePairsLayout(B, S, T, C).am_sum; }

bool simple_pairs_supported(const void *lm, const void *am, int S1, int T, int C, int rnnt_type) {
  (void)lm, (void)am;  // rows of any alignment: see rows_by_four
  if (C < 1 || S1 < 1 || T < 1) return false;
  // px += py[s+1] is carried from column to column inside one tile of 128 lattice rows
  if (rnnt_type == FRNNT_CONSTRAINED && S1 > kPairTile) return false;
  return true;
}

// Four entries of a row at a time as one 16-byte (8-byte) load, TMA stores of the gradients: for
// vocabularies that are a multiple of 4 and 16-byte aligned tensors.  Everything else reads
// single entries and stores gradient boxes row by row.  16 x (59, 293) x 4233, forward and
// backward: normalizer 76, lm / am gradient 52 / 90, planes 40 us, against 1503, 294 / 248 and
// 48 us on the FMA pipe.
static bool rows_by_four(const void *a, const void *b, int C) {
  return C % 4 == 0 && (uintptr_t)a % 16 == 0 && (uintptr_t)b % 16 == 0;
}

// Which calls get the more accurate form of the products (EXACT: a fresh accumulator per 64 values of
// the reduction instead of 128, the small products first): those whose rows of 4-byte values
// are not all 16-byte aligned.  The FMA pipe used to serve them, and its float32 sums are more
// accurate than 128 truncating tensor-core additions.  Relative errors of px and of the am
// gradient in 1e-8, 160 x 41 cells of unit normals, C = 64 / 128 / 500: in groups of 128 8.1,
// 14.2, 11.9 and 9.0, 16.8, 10.2; in groups of 64 6.0, 5.5, 4.9 and 7.9, 7.0, 6.1; on the FMA pipe
// 4.9, 4.9, 6.0 and 7.4, 6.7, 6.1.  16-bit rows get what their float32 copies get, which are
// aligned.
bool simple_pairs_exact(const void *lm, const void *am, int C, int input_dtype) {
  return is_half_input(input_dtype) ? C % 4 != 0 : !rows_by_four(lm, am, C);
}

// ---- forward, pass 1: row maxima, exp planes, per-row scalars -----------------------------------
// entries 4 v .. 4 v + 3 of a row of C; VEC: as one load, else singly, -inf beyond the row (exp: 0)
template <bool VEC, typename TIn>
__device__ __forceinline__ float4 row_load4(const TIn *row, int v, int C) {
  if (VEC) return in_load4(row, v);
  const int c = 4 * v;
  return make_float4(in_f32(row[c]), c + 1 < C ? in_f32(row[c + 1]) : -INFINITY,
                     c + 2 < C ? in_f32(row[c + 2]) : -INFINITY, c + 3 < C ? in_f32(row[c + 3]) : -INFINITY);
}

// Rows first_row .. rows - 1 of lm (rows 0 .. B*S1-1) and am (the rest), G warps each, each lane keeping K vectors of four
// entries: a row of up to 128 G K entries is read once.  What bounds the kernel is HBM (read
// 4 C, write 4 C bytes a row); re-reading what one warp cannot keep made rows of 5000 entries
// take 1.4 times as long (64 x (60, 400) x 5000: 312 -> 226 us, 157 at the copy rate;
// 16 x (59, 293) x 4233, single entries: 74 -> 40 us).
template <typename TIn, bool VEC, int G, int K>
__global__ void __launch_bounds__(256)
exp_planes_kernel(const TIn *__restrict__ lm, const TIn *__restrict__ am,
                  const int64_t *__restrict__ symbols, __half *__restrict__ lp_hi,
                  __half *__restrict__ lp_lo, __half *__restrict__ ap_hi, __half *__restrict__ ap_lo,
                  float *__restrict__ lmmax, float *__restrict__ lmsum, float *__restrict__ ammax,
                  float *__restrict__ lm_blk, float *__restrict__ lm_sym, float *__restrict__ lnorm,
                  float *__restrict__ am_blk, float *__restrict__ am_sym, float *__restrict__ am_sum,
                  float *__restrict__ px, int B, int S, int T, int C, int Cp, int Sp, int blank, int regular, long long first_row,
                  long long rows) {
  constexpr int LANES = 32 * G, RPB = 8 / G;  // threads of a row, rows of a CTA
  __shared__ float part[8];
  const int lane = threadIdx.x % LANES, slot = threadIdx.x / LANES;
  const int S1 = S + 1, nvec = (C + 3) / 4;
  const long long rows_lm = (long long)B * S1;
  auto over_group = [&](float v, bool is_max) {
    v = is_max ? warp_max(v) : warp_sum(v);
    if (G > 1) {
      __syncthreads();
      if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
      __syncthreads();
      v = part[slot * G];
#pragma unroll
      for (int w = 1; w < G; ++w) v = is_max ? fmaxf(v, part[slot * G + w]) : v + part[slot * G + w];
    }
    return v;
  };
  for (long long row0 = first_row + (long long)blockIdx.x * RPB; row0 < rows; row0 += (long long)gridDim.x * RPB) {
    // a CTA's last rows may not exist; they take part in the barriers of the others
    const bool valid = row0 + slot < rows;
    if (G == 1 && !valid) break;
    const long long row = valid ? row0 + slot : rows - 1;
    const bool is_lm = row < rows_lm;
    const long long r = is_lm ? row : row - rows_lm;
    const TIn *src = (is_lm ? lm : am) + r * C;
    uint2 *dh = reinterpret_cast<uint2 *>((is_lm ? lp_hi : ap_hi) + r * Cp);
    uint2 *dl = reinterpret_cast<uint2 *>((is_lm ? lp_lo : ap_lo) + r * Cp);
    float4 keep[K];
    float m = -INFINITY;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int v = lane + LANES * j;
      if (v < nvec) keep[j] = row_load4<VEC>(src, v, C);
    }
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (lane + LANES * j < nvec) m = fmaxf(fmaxf(m, fmaxf(keep[j].x, keep[j].y)), fmaxf(keep[j].z, keep[j].w));
    for (int v = lane + LANES * K; v < nvec; v += LANES) {
      const float4 q = row_load4<VEC>(src, v, C);
      m = fmaxf(fmaxf(m, fmaxf(q.x, q.y)), fmaxf(q.z, q.w));
    }
    m = over_group(m, true);
    float sum = 0.f;
    auto one = [&](int v, const float4 &q) {
      const float e[4] = {expf(q.x - m), expf(q.y - m), expf(q.z - m), expf(q.w - m)};
#pragma unroll
      for (int i = 0; i < 4; ++i) sum += e[i];
      uint2 hi, lo;
      fp16_pair4(e, kExpScale, hi, lo);
      if (valid) dh[v] = hi, dl[v] = lo;
    };
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int v = lane + LANES * j;
      if (v < nvec) one(v, keep[j]);
    }
    for (int v = lane + LANES * K; v < nvec; v += LANES) one(v, row_load4<VEC>(src, v, C));
    sum = over_group(sum, false);
    if (!valid) continue;
    if (!is_lm) {
      // am[t][symbol of every lattice row]: gathered here, where the row has just been read
      // (L1 hits), so that the product's epilogue reads them as whole 128-byte lines
      const TIn *x = am + r * C;
      const int64_t *sy = symbols + (size_t)div_rows(r, T) * S;
      float *dst = am_sym + (size_t)r * Sp;
      for (int s = lane; s < Sp; s += LANES) {
        float v = 0.f;
        if (s < S) {
          long long y = sy[s];
          if (y < 0 || y >= C) y = blank;
          v = in_f32(x[y]);
        }
        dst[s] = v;
      }
    }
    if (lane == 0) {
      const TIn *x = (is_lm ? lm : am) + r * C;
      if (is_lm) {
        const int b = (int)div_rows(r, S1), s = mod_rows(r, S1);
        lmmax[r] = m;
        lmsum[r] = sum;
        lnorm[r] = logf(sum) + m;
        lm_blk[r] = in_f32(x[blank]);
        if (s < S) {
          long long y = symbols[(size_t)b * S + s];
          if (y < 0 || y >= C) y = blank;
          lm_sym[r] = in_f32(x[y]);
          // the -inf column of the regular type, which no frame owns
          if (regular) px[((size_t)b * S + s) * (T + 1) + T] = -INFINITY;
        }
      } else {
        ammax[r] = m;
        am_sum[r] = sum;
        am_blk[r] = in_f32(x[blank]);
      }
    }
  }
}

// ---- forward, pass 2: the normalizer product and the lattices ----------------------------------
// tile rows = frames t, tile columns = lattice rows s
// EXACT (simple_pairs_exact): a fresh accumulator per 64 values of the reduction and logf instead of
// __logf
template <bool EXACT>
struct NormPairExt : SimpleLattice {
  static constexpr bool kBatched = true, kCustomStore = true;
  static constexpr int kGroup = EXACT ? 1 : kPairGroup;
  struct Row {
    float ammax_t, am_blk_t, amonly_t, py_next, pen, am_sum_t;
    const float *amrow;
    long long t_end;
    bool weak;
  };
  __device__ void row_begin(Row &r, int b, int t, int) const {
    const size_t bt = (size_t)b * T + t;
    r.ammax_t = ammax[bt];
    r.am_blk_t = am_blk[bt];
    r.amonly_t = (smoothed && !am_only_off) ? amonly[bt] : 0.f;
    r.amrow = am_sym + bt * Sp;
    r.t_end = (rnnt_type == FRNNT_REGULAR && boundary != nullptr) ? (long long)boundary[4 * b + 3] : -1;
    r.py_next = 0.f;
    r.pen = delay_penalty_at<float>(boundary, b, T, t, delay_penalty);
    r.am_sum_t = am_sum[bt];
    r.weak = false;
  }
  __device__ void prefetch(Row &, int, int, int) const {}
  __device__ void finish(Row &, int, int, int, float (&)[16], int) const {}
  __device__ void row_end(Row &r, int b, int t, int s0) const {
    weak[((size_t)b * ((S + kPairTile) / kPairTile) + s0 / kPairTile) * T + t] = r.weak;
  }
  // per-column data of a tile in the warp's 4 KB of shared memory: one 16-byte entry
  // (lmmax, lm[blank], lm[symbol], lm-only normalizer), the symbol and the row's share of the
  // bound on weak cells per lattice row
  struct Cols {
    float4 q[kPairTile];
    int sym[kPairTile];
    float bound[kPairTile];
  };
  __device__ void tile_begin(int b, int s0, uint8_t *box, int lane) const {
    Cols *c = reinterpret_cast<Cols *>(box);
    const int S1 = S + 1;
#pragma unroll
    for (int j = 0; j < kPairTile / 32; ++j) {
      const int i = lane + 32 * j, s = s0 + i;
      if (s < S1) {
        const size_t bs = (size_t)b * S1 + s;
        c->bound[i] = weak_bound(lmsum[bs], 0.f);
        long long y = blank;
        float ls_ = 0.f;
        if (s < S) {
          ls_ = lm_sym[bs];
          y = symbols[(size_t)b * S + s];
          if (y < 0 || y >= C) y = blank;
        }
        c->q[i] = make_float4(lmmax[bs], lm_blk[bs], ls_, lnorm[bs]);
        c->sym[i] = (int)y;
      }
    }
  }
  // columns from the last to the first: px of row s needs py of row s + 1 (constrained).
  // The epilogue runs on one warp per scheduler, i.e. at the latency of its instructions:
  // it is written to be short (one 16-byte shared-memory load per cell, the log on the
  // special-function unit: |error| of lg2.approx is 2^-22, i.e. 1.6e-7 on the normalizer,
  // no more than the rounding of an exact float32 log of this magnitude).
  __device__ void store_box(Row &r, int b, int t, int s0, int c0, float (&v0)[16], float (&v1)[16],
                            const uint8_t *box) const {
    const Cols *c = reinterpret_cast<const Cols *>(box);
    const int S1 = S + 1, T1 = rnnt_type == FRNNT_REGULAR ? T + 1 : T;
    // am[t][symbol] of the box's lattice rows: one 128-byte line per frame
    float pxam[32];
    if (s0 + c0 < Sp) {
      const float4 *g = reinterpret_cast<const float4 *>(r.amrow + s0 + c0);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 q = g[i];
        pxam[4 * i] = q.x, pxam[4 * i + 1] = q.y, pxam[4 * i + 2] = q.z, pxam[4 * i + 3] = q.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) pxam[i] = 0.f;
    }
    float *nrow = norm + ((size_t)b * S1 + s0 + c0 + 31) * T + t;
    float *yrow = py + ((size_t)b * S1 + s0 + c0 + 31) * T + t;
    float *xrow = px + ((size_t)b * S + s0 + c0 + 31) * T1 + t;
    const bool am_on = smoothed && !am_only_off;
    const float lu_blank = am_on ? loguni[blank] : 0.f;
    const float am_y = am_on ? (r.am_blk_t + lu_blank - r.amonly_t) * as : 0.f;
    float zmin = INFINITY;  // of z less the row's share of the bound
#pragma unroll
    for (int i = 31; i >= 0; --i, nrow -= T, yrow -= T, xrow -= T1) {
      const int s = s0 + c0 + i;
      if (s > S) continue;
      const float acc = i < 16 ? v0[i & 15] : v1[i & 15];
      const float4 q = c->q[c0 + i];
      const float z = acc * kExpInv2 + 1.17549435e-38f;
      zmin = fminf(zmin, z - c->bound[c0 + i]);
      const float nv = (EXACT ? logf(z) : __logf(z)) + q.x + r.ammax_t;
      *nrow = nv;
      float vy = r.am_blk_t + q.y - nv;
      if (smoothed) vy = vy * both + (q.y - q.w) * ls + am_y;
      *yrow = vy;
      if (s < S) {
        float v = pxam[i] + q.z - nv;
        if (smoothed) {
          v = v * both + (q.z - q.w) * ls;
          if (am_on) v += (pxam[i] + loguni[c->sym[c0 + i]] - r.amonly_t) * as;
        }
        if (rnnt_type == FRNNT_REGULAR) {
          if ((long long)t == r.t_end) v = -INFINITY;
        } else if (rnnt_type == FRNNT_CONSTRAINED) {
          v += r.py_next;
        }
        if (delay_penalty > 0.0) v = __fadd_rn(v, r.pen);
        *xrow = v;
      }
      r.py_next = vy;
    }
    r.weak |= zmin < weak_bound(0.f, r.am_sum_t);
  }
};

// ---- backward products --------------------------------------------------------------------------
// what both epilogues share: the 32 plane values (exp(x - max) * 2^14) of the row's next box
struct PlaneRow {
  uint4 h[4], l[4];
  __device__ void load(const __half *hi, const __half *lo, size_t off) {
    const uint4 *ph = reinterpret_cast<const uint4 *>(hi + off);
    const uint4 *pl = reinterpret_cast<const uint4 *>(lo + off);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = ph[i], l[i] = pl[i];
  }
  __device__ void get(int half, float (&e)[16]) const {
    __align__(16) __half hh[16], ll[16];
    *reinterpret_cast<uint4 *>(hh) = h[2 * half];
    *reinterpret_cast<uint4 *>(hh + 8) = h[2 * half + 1];
    *reinterpret_cast<uint4 *>(ll) = l[2 * half];
    *reinterpret_cast<uint4 *>(ll + 8) = l[2 * half + 1];
#pragma unroll
    for (int i = 0; i < 16; ++i) e[i] = (__half2float(hh[i]) + __half2float(ll[i])) * (1.f / kExpScale);
  }
};

// dlm[s][c] = -L[s][c] * sum_t Rw[s][t] A[t][c]  (+ lm-only term)
template <bool ROW_STORE, bool EXACT>
struct LmGradPairExt {
  static constexpr bool kBatched = true, kCustomStore = false, kRowStore = ROW_STORE;
  static constexpr int kGroup = EXACT ? 1 : kPairGroup;
  const __half *lp_hi, *lp_lo;
  const float *inv_rw, *lmsum, *gl;
  int S1, Cp;
  struct Row {
    float sc, inv_sum, g;
    PlaneRow pl;
  };
  __device__ void row_begin(Row &r, int b, int s, int n0) const {
    const size_t row = (size_t)b * S1 + s;
    r.sc = inv_rw[b] * (1.f / kExpScale);
    r.inv_sum = gl != nullptr ? 1.f / lmsum[row] : 0.f;
    r.g = gl != nullptr ? gl[row] : 0.f;
    (void)n0;
  }
  // the planes are padded to whole 64-entry blocks, so a box is always readable
  __device__ void prefetch(Row &r, int b, int s, int n) const {
    if (n < Cp) r.pl.load(lp_hi, lp_lo, ((size_t)b * S1 + s) * Cp + n);
  }
  __device__ void finish(Row &r, int, int, int, float (&v)[16], int half) const {
    float L[16];
    r.pl.get(half, L);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float o = -(L[i] * (v[i] * r.sc));
      if (gl != nullptr) {
        const float P = L[i] * r.inv_sum;
        o -= r.g * P;
      }
      v[i] = o;
    }
  }
  __device__ void row_end(Row &, int, int, int) const {}
  template <class R> __device__ void store_box(R &, int, int, int, int, float (&)[16], float (&)[16], const uint8_t *) const {}
  __device__ void tile_begin(int, int, uint8_t *, int) const {}
};

// dam[t][c] = -A[t][c] * sum_s Rw[s][t] L[s][c]  (+ am-only term)
template <bool ROW_STORE, bool EXACT>
struct AmGradPairExt {
  static constexpr bool kBatched = true, kCustomStore = false, kRowStore = ROW_STORE;
  static constexpr int kGroup = EXACT ? 1 : kPairGroup;
  const __half *ap_hi, *ap_lo;
  const float *inv_rw, *ammax, *h, *uni, *amonly;
  int T, C, Cp;
  struct Row {
    float sc, w;
    PlaneRow pl;
  };
  __device__ void row_begin(Row &r, int b, int t, int) const {
    const size_t row = (size_t)b * T + t;
    r.sc = inv_rw[b] * (1.f / kExpScale);
    // a weak frame gets the term in float32 later
    r.w = h != nullptr && !am_only_weak(ammax[row], amonly[row]) ? h[row] * expf(ammax[row] - amonly[row]) : 0.f;
  }
  __device__ void prefetch(Row &r, int b, int t, int n) const {
    if (n < Cp) r.pl.load(ap_hi, ap_lo, ((size_t)b * T + t) * Cp + n);
  }
  __device__ void finish(Row &r, int, int, int c0, float (&v)[16], int half) const {
    float A[16];
    r.pl.get(half, A);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float o = -(A[i] * (v[i] * r.sc));
      if (h != nullptr && c0 + i < C) o -= r.w * A[i] * uni[c0 + i];
      v[i] = o;
    }
  }
  __device__ void row_end(Row &, int, int, int) const {}
  template <class R> __device__ void store_box(R &, int, int, int, int, float (&)[16], float (&)[16], const uint8_t *) const {}
  __device__ void tile_begin(int, int, uint8_t *, int) const {}
};

// Rw [B][S1][Tp] float without the weak cells -> planes [B][S1][Tq], columns Tp..Tq-1 zero (they are
// inside the tensor maps only as padding up to T, never beyond it, but the backward's second product
// reads rows as its reduction index and must not meet stale data).  One scale per utterance
// (blockIdx.y), so that its planes do not depend on the weights of the others.
__global__ void __launch_bounds__(256)
sp_split_kernel(const float *__restrict__ x, const unsigned *__restrict__ weak, int S1, int Tp, int Tq,
                int weak_words, const float *__restrict__ part, __half *__restrict__ hi,
                __half *__restrict__ lo, float *__restrict__ inv_scale) {
  // the maxima of the utterance's rows by all threads of each of its CTAs, four entries at a time
  // after that: 64 x 101 rows of 500 in 9.0 us (11.2 with one scale, i.e. every CTA reading all maxima)
  __shared__ float slot[8];
  const size_t row0 = (size_t)blockIdx.y * S1;
  float m = 0.f;
#pragma unroll 4
  for (int i = threadIdx.x; i < S1; i += 256) m = fmaxf(m, part[row0 + i]);
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) slot[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) m = fmaxf(m, slot[w]);
  const float scale = fp16_pair_scale(m);
  if (blockIdx.x == 0 && threadIdx.x == 0) inv_scale[blockIdx.y] = 1.f / scale;
  const int nvec = Tq / 4;  // Tp is a multiple of 4, too
  const long long n = (long long)S1 * nvec;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    const size_t r = row0 + div_rows(i, nvec);
    const int q = mod_rows(i, nvec), c = 4 * q;
    uint2 h = make_uint2(0u, 0u), l = h;
    if (c < Tp) {
      const float4 q4 = *reinterpret_cast<const float4 *>(x + r * Tp + c);
      const unsigned w = weak[r * weak_words + c / 32] >> (c % 32);
      const float v[4] = {w & 1u ? 0.f : q4.x, w & 2u ? 0.f : q4.y, w & 4u ? 0.f : q4.z, w & 8u ? 0.f : q4.w};
      fp16_pair4(v, scale, h, l);
    }
    reinterpret_cast<uint2 *>(hi)[r * nvec + q] = h;
    reinterpret_cast<uint2 *>(lo)[r * nvec + q] = l;
  }
}

int launch_simple_forward_pairs(const void *lm, const void *am, const int64_t *symbols,
                                const int64_t *boundary, int blank, int rnnt_type, int smoothed,
                                int am_only_off, float both, float ls, float as, float *px, float *py,
                                float *norm, float *lmmax, float *lmsum, float *ammax,
                                const float *amonly, const float *loguni, void *pairs_saved, int B, int S,
                                int T, int C, int stage, cudaStream_t st, double delay_penalty, int input_dtype) {
  const SimplePairsLayout L(B, S, T, C);
  uint8_t *sv = (uint8_t *)pairs_saved;
  __half *lp_hi = (__half *)(sv + L.lp_hi), *lp_lo = (__half *)(sv + L.lp_lo);
  __half *ap_hi = (__half *)(sv + L.ap_hi), *ap_lo = (__half *)(sv + L.ap_lo);
  float *lm_blk = (float *)(sv + L.lm_blk), *lm_sym = (float *)(sv + L.lm_sym);
  float *lnorm = (float *)(sv + L.lnorm), *am_blk = (float *)(sv + L.am_blk);
  float *am_sym = (float *)(sv + L.am_sym), *am_sum = (float *)(sv + L.am_sum);
  const int S1 = S + 1;
  if (stage == 0) {
    const long long rows_lm = (long long)B * S1, rows = rows_lm + (long long)B * T;
    const bool vec = rows_by_four(lm, am, C);
#define FRNNT_EXP_PLANES_AS(TIn, VEC, G, K, FIRST, LAST)                                                            \
  FRNNT_KERNEL(exp_planes_kernel<TIn, VEC, G, K>                                                                    \
               <<<(int)std::min<long long>((((LAST) - (FIRST)) * G + 7) / 8, (long long)sm_count() * 32), 256, 0, st>>>( \
                   (const TIn *)lm, (const TIn *)am, symbols, lp_hi, lp_lo, ap_hi, ap_lo, lmmax, lmsum, ammax,      \
                   lm_blk, lm_sym, lnorm, am_blk, am_sym, am_sum, px, B, S, T, C, L.Cp, L.Sp, blank,                        \
                   rnnt_type == FRNNT_REGULAR, FIRST, LAST))
    // Rows up to 512: lanes keep 16 entries.  Longer rows: lm, whose sum of exponentials counts,
    // stays with one warp per row (the order of that sum is kept); am, by far the most rows, goes
    // to as many warps as 32 entries a lane take
#define FRNNT_EXP_PLANES_BY(TIn, VEC)                          \
  do {                                                         \
    if (C <= 512) {                                            \
      FRNNT_EXP_PLANES_AS(TIn, VEC, 1, 4, 0LL, rows);          \
    } else {                                                   \
      FRNNT_EXP_PLANES_AS(TIn, VEC, 1, 4, 0LL, rows_lm);       \
      if (C <= 1024)                                           \
        FRNNT_EXP_PLANES_AS(TIn, VEC, 1, 8, rows_lm, rows);    \
      else if (C <= 2048)                                      \
        FRNNT_EXP_PLANES_AS(TIn, VEC, 2, 8, rows_lm, rows);    \
      else if (C <= 4096)                                      \
        FRNNT_EXP_PLANES_AS(TIn, VEC, 4, 8, rows_lm, rows);    \
      else                                                     \
        FRNNT_EXP_PLANES_AS(TIn, VEC, 8, 8, rows_lm, rows);    \
    }                                                          \
  } while (0)
#define FRNNT_EXP_PLANES(TIn)            \
  do {                                   \
    if (vec)                             \
      FRNNT_EXP_PLANES_BY(TIn, true);    \
    else                                 \
      FRNNT_EXP_PLANES_BY(TIn, false);   \
  } while (0)
    if (input_dtype == FRNNT_F16) {
      FRNNT_EXP_PLANES(__half);
    } else if (input_dtype == FRNNT_BF16) {
      FRNNT_EXP_PLANES(__nv_bfloat16);
    } else {
      FRNNT_EXP_PLANES(float);
    }
#undef FRNNT_EXP_PLANES
#undef FRNNT_EXP_PLANES_BY
#undef FRNNT_EXP_PLANES_AS
    FRNNT_CUDA(cudaGetLastError());
    return FRNNT_OK;
  }
  CUtensorMap mah, mal, mbh, mbl;
  int rc = make_pair_map(&mah, ap_hi, T, C, L.Cp, false, B, (long long)T * L.Cp);
  if (rc == FRNNT_OK) rc = make_pair_map(&mal, ap_lo, T, C, L.Cp, false, B, (long long)T * L.Cp);
  if (rc == FRNNT_OK) rc = make_pair_map(&mbh, lp_hi, S1, C, L.Cp, false, B, (long long)S1 * L.Cp);
  if (rc == FRNNT_OK) rc = make_pair_map(&mbl, lp_lo, S1, C, L.Cp, false, B, (long long)S1 * L.Cp);
  if (rc != FRNNT_OK) return rc;
  const LinShape shape{T, S1, C, ((C + kPairBK - 1) / kPairBK) * kPairBK, (T + kPairTile - 1) / kPairTile,
                       (S1 + kPairTile - 1) / kPairTile, B};
  // the policy stores the lattices itself; the engine's output map is unused and is made
  // over the normalizer buffer only because it has to be a valid map
  const SimpleLattice lattice{
      norm,   px,     py,    am_sym,  symbols, boundary, lmmax,     ammax,    lm_blk, lm_sym,      lnorm, am_blk,
      amonly, loguni, lmsum, am_sum,  sv + L.weak, S, T, C, blank,  rnnt_type, smoothed, am_only_off, both,  ls,
      as,     L.Sp,   delay_penalty};
  auto product = [&](auto exact) {
    return launch_pair_umma<false, false>(mah, mal, mbh, mbl, norm, shape,
                                          NormPairExt<decltype(exact)::value>{lattice}, st);
  };
  rc = simple_pairs_exact(lm, am, C, input_dtype) ? product(std::true_type{}) : product(std::false_type{});
  if (rc != FRNNT_OK) return rc;
  return launch_weak_cells(lm, am, input_dtype, lattice, B, st);
}

int launch_simple_grads_pairs(const float *rw, const unsigned *weak, const float *lmsum, const float *ammax,
                              const float *amonly, const float *uni, const float *gl, const float *h,
                              float *lm_grad, float *am_grad, const void *pairs_saved, void *pairs_scratch, int B, int S, int T, int C, int Tp,
                              bool exact, cudaStream_t st) {
  const SimplePairsLayout L(B, S, T, C);
  const uint8_t *sv = (const uint8_t *)pairs_saved;
  uint8_t *sc = (uint8_t *)pairs_scratch;
  const __half *lp_hi = (const __half *)(sv + L.lp_hi), *lp_lo = (const __half *)(sv + L.lp_lo);
  const __half *ap_hi = (const __half *)(sv + L.ap_hi), *ap_lo = (const __half *)(sv + L.ap_lo);
  __half *rw_hi = (__half *)(sc + L.rw_hi), *rw_lo = (__half *)(sc + L.rw_lo);
  float *parts = (float *)(sc + L.parts), *inv_rw = (float *)(sc + L.inv_scale);
  const int S1 = S + 1, Cp = L.Cp, Tq = L.Tq;

  CUtensorMap a1h, a1l, b1h, b1l, a2h, a2l, b2h, b2l;
  int rc = make_pair_map(&a1h, rw_hi, S1, T, Tq, false, B, (long long)S1 * Tq);      // Rw [s][t], K = t
  if (rc == FRNNT_OK) rc = make_pair_map(&a1l, rw_lo, S1, T, Tq, false, B, (long long)S1 * Tq);
  if (rc == FRNNT_OK) rc = make_pair_map(&b1h, ap_hi, T, C, Cp, true, B, (long long)T * Cp);   // A [t][c], K = t rows
  if (rc == FRNNT_OK) rc = make_pair_map(&b1l, ap_lo, T, C, Cp, true, B, (long long)T * Cp);
  if (rc == FRNNT_OK) rc = make_pair_map(&a2h, rw_hi, S1, T, Tq, true, B, (long long)S1 * Tq);  // Rw^T: K = s rows
  if (rc == FRNNT_OK) rc = make_pair_map(&a2l, rw_lo, S1, T, Tq, true, B, (long long)S1 * Tq);
  if (rc == FRNNT_OK) rc = make_pair_map(&b2h, lp_hi, S1, C, Cp, true, B, (long long)S1 * Cp);  // L [s][c], K = s rows
  if (rc == FRNNT_OK) rc = make_pair_map(&b2l, lp_lo, S1, C, Cp, true, B, (long long)S1 * Cp);
  if (rc != FRNNT_OK) return rc;

  // the caller left max |rw| per row in `parts`
  const long long per_utt = ((long long)S1 * (Tq / 4) + 255) / 256;
  const dim3 grid((unsigned)std::min(per_utt, std::max<long long>(1, (long long)sm_count() * 16 / B)), (unsigned)B);
  FRNNT_KERNEL(sp_split_kernel<<<grid, 256, 0, st>>>(rw, weak, S1, Tp, Tq, weak_words(T), parts, rw_hi, rw_lo, inv_rw));
  FRNNT_CUDA(cudaGetLastError());

  const int ctiles = (C + kPairTile - 1) / kPairTile;
  const LinShape lm_shape{S1, C, T, ((T + kPairBK - 1) / kPairBK) * kPairBK, (S1 + kPairTile - 1) / kPairTile, ctiles, B};
  const LinShape am_shape{T, C, S1, ((S1 + kPairBK - 1) / kPairBK) * kPairBK, (T + kPairTile - 1) / kPairTile, ctiles, B};
  auto products = [&](auto row_store, auto more_exact) {
    constexpr bool kRow = decltype(row_store)::value, kExact = decltype(more_exact)::value;
    const LmGradPairExt<kRow, kExact> lm_ext{lp_hi, lp_lo, inv_rw, lmsum, gl, S1, Cp};
    const int r = launch_pair_umma<false, true>(a1h, a1l, b1h, b1l, lm_grad, lm_shape, lm_ext, st);
    if (r != FRNNT_OK) return r;
    const AmGradPairExt<kRow, kExact> am_ext{ap_hi, ap_lo, inv_rw, ammax, h, uni, amonly, T, C, Cp};
    return launch_pair_umma<true, true>(a2h, a2l, b2h, b2l, am_grad, am_shape, am_ext, st);
  };
  // TMA stores where the gradients' rows allow them, whatever the rows of lm and am
  if (!rows_by_four(lm_grad, am_grad, C)) return products(std::true_type{}, std::true_type{});
  return exact ? products(std::false_type{}, std::true_type{}) : products(std::false_type{}, std::false_type{});
}

}  // namespace frnnt
