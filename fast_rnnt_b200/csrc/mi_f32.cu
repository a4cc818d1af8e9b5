// Mutual-information sweeps for float lattices: an utterance over a cluster of CTAs.
// The recursion, the boundary box and the lattice scratch are those of mi.cu.
//
// What bounds both sweeps is the chain of s_end + t_end anti-diagonals, each waiting for the
// one before; bytes and operations are far from any limit.  So the time is (number of
// diagonals) x (time of one step), and everything here shortens the step:
//
//   * ONE compute warp per CTA, lane l owning R neighbouring rows: 32 R rows, and a single value
//     per lane and step travels between threads (a warp shuffle).  R = 1 up to 32 rows (180
//     cycles a forward step), else 2 (235: the second row's instructions mostly fit into the
//     latency of the first row's chain; four rows were 2.3 times a step of two);
//   * a taller lattice is split over a cluster of up to 8 CTAs.  CTA w works two chunks of 16
//     diagonals behind CTA w - 1 (forward; the other way round in the backward): the compute
//     warp leaves the edge row in shared memory, an otherwise idle warp sends it, a chunk at
//     a time, to the neighbour (st.async, counted by an mbarrier per chunk); an mbarrier in
//     the other direction bounds how far the sender runs ahead.  Measured slower, in cycles a
//     step: the compute warp sending each value itself + 55; a cluster barrier or a release at
//     cluster scope per chunk, which waits for the helpers' global stores, + 45 to 80;
//     several compute warps on one SM, which share its schedulers with their helpers;
//   * helper warps move everything between global memory and shared memory, one chunk ahead
//     (px, py, weights) and one behind (weights, gradients).  The rings are [16
//     diagonals][rows], so that a compute lane fetches or leaves its R rows in one access;
//     the pitch (rows + 4) keeps the transposing accesses of the helpers free of bank
//     conflicts.  The warp that shares the compute warp's scheduler is the one that only
//     sends the edge row;
//   * cells outside the box need no test in the forward chain: they are fed x = -inf, y = 0,
//     which keeps rows that have not begun at -inf and the origin at 0;
//   * the forward's helpers turn the exponents a - p[s][t] that its compute warp leaves in
//     shared memory into the backward weights (kMiDead: a cell that passes no gradient on), so
//     that the helpers of the backward only copy them in and the gradients out.
//
// Forward / backward of 64 x (100, 500): 79 / 25 us, with one row per thread 113 / 62; of
// 6 x (423, 2211): 316 / 102 us, before 1240 / 1252.
#include <cooperative_groups.h>

#include "mi.cuh"

namespace frnnt {

constexpr int kStep = 16;      // anti-diagonals per chunk
constexpr int kHelpers = 6;    // helper warps: 1, 2, 3, 5, 6, 7 of eight (0 computes)
constexpr int kThreads = 256;
constexpr int kEdgeRing = 128;  // edge-row values kept (eight chunks)
constexpr int kMaxCluster = 8;

// if (cond) acc = x + y, as one predicated instruction (a select would lengthen the chain)
__device__ __forceinline__ void add_if(float &acc, bool cond, float x, float y) {
  asm("{\n.reg .pred q;\nsetp.ne.s32 q, %3, 0;\n@q add.f32 %0, %1, %2;\n}"
      : "+f"(acc)
      : "f"(x), "f"(y), "r"((int)cond));
}

// LogAdd with the values of log_add(): a difference that is not finite, or too large for exp()
// to count, leaves the larger operand.  expf and log1pf are the library's on purpose: a faster
// pair (one ex2 and a polynomial of the same error, 0.7 of this kernel's time) rounds a few
// cells in a thousand to a neighbouring float32, and prune ranges are an argmax that such
// neighbours can move.
__device__ __forceinline__ float log_add_f32(float a, float b) {
  const float d = a - b;
  float r = a < b ? b : a;
  add_if(r, fabsf(d) < 150.f, r, log1pf(expf(-fabsf(d))));
  return r;
}

template <int R> struct Vec;
template <> struct Vec<1> { using type = float; };
template <> struct Vec<2> { using type = float2; };
template <> struct Vec<4> { using type = float4; };

template <int R>
__device__ __forceinline__ void load_rows(float (&v)[R], const float *src) {
  *reinterpret_cast<typename Vec<R>::type *>(v) = *reinterpret_cast<const typename Vec<R>::type *>(src);
}
template <int R>
__device__ __forceinline__ void store_rows(float *dst, const float (&v)[R]) {
  *reinterpret_cast<typename Vec<R>::type *>(dst) = *reinterpret_cast<const typename Vec<R>::type *>(v);
}

// ---- cluster --------------------------------------------------------------------
__device__ __forceinline__ int cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
__device__ __forceinline__ int cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return (int)r;
}
// address of `p` (own shared memory) in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ unsigned peer_address(const void *p, int rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(a)
               : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
// `v` to an address in a peer's shared memory; counts four bytes at that CTA's mbarrier `bar`
__device__ __forceinline__ void peer_send(unsigned address, float v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(address),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}

// Hand-over of the edge row between neighbouring CTAs, chunks numbered in the order of the sweep.
// Each side has one mbarrier per slot of the edge ring (chunk mod 8): `full` in the consumer's
// shared memory, `taken` in the producer's.  Every wait is bounded.  One that runs out makes all
// later ones of its warp give up at once; the CTA goes on with NaN for the edge row, which the
// recursion carries to every cell behind it, to the CTAs and row blocks that follow, and so to
// the score, the remaining gradients and the origin's.
constexpr int kSlots = kEdgeRing / kStep;

__device__ __forceinline__ void slot_init(uint64_t *bars) {
  for (int i = 0; i < 2 * kSlots; ++i)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(bars + i)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// "taken" carries no data: what it lets the producer overwrite has been read into registers
__device__ __forceinline__ void slot_arrive(unsigned peer_bars, int chunk) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(peer_bars + 8 * (chunk % kSlots)) : "memory");
}
// the receiver's own arrival: `steps` values are to come for this chunk
__device__ __forceinline__ void slot_expect(uint64_t *bars, int chunk, int steps) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(bars + chunk % kSlots)),
               "r"(4 * steps)
               : "memory");
}
// true: nothing came within `tries` looks (or the warp has given up before)
__device__ __forceinline__ bool slot_wait(const uint64_t *bars, int chunk, bool failed, int tries) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(bars + chunk % kSlots);
  const unsigned parity = (chunk / kSlots) & 1;
  for (int spin = 0; !failed && spin < tries; ++spin) {
    unsigned done;
    asm volatile("{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n"
                 "selp.u32 %0, 1, 0, q;\n}"
                 : "=r"(done)
                 : "r"(a), "r"(parity)
                 : "memory");
    if (done) return false;
  }
  return true;
}
__device__ __forceinline__ void cluster_sync() { cooperative_groups::this_cluster().sync(); }
// The end of a CTA.  The neighbours may still be writing here until all have arrived; a warp that gave
// up waiting has not seen its last values arrive, so it stays for 64 us, some fifty times as
// long as they are under way at most.
__device__ __forceinline__ void leave_cluster(bool failed) {
  cluster_sync();
  for (int i = 0; failed && i < 64; ++i) __nanosleep(1000);
}

template <int R>
struct MiShape {
  static constexpr int kRows = 32 * R;                        // lattice rows of a CTA
  static constexpr int kRing = kRows + 4;                     // pitch of a ring
  static constexpr int kTasks = kRows / (2 * R);              // 2 R rows x 16 diagonals each
  static constexpr int kTasksPerWarp = (kTasks + kHelpers - 1) / kHelpers;
  static constexpr int kQuads = kRows / 4 * kStep;            // of weights in a chunk, four rows each
  static constexpr int kQuadsPerLane = (kQuads + kHelpers * 32 - 1) / (kHelpers * 32);
  static constexpr int kGroup = 8;                            // steps whose inputs are fetched together
  static constexpr size_t kSmem = ((size_t)6 * kStep * kRing + kEdgeRing + 2 * kStep) * sizeof(float) + 2 * kSlots * sizeof(uint64_t);
};

// -----------------------------------------------------------------------------
// forward
// -----------------------------------------------------------------------------
// BLOCKED: the launch covers lattice rows [row0, row0 + kMiF32Rows) only
template <int R, bool CLUSTER, bool MODIFIED, bool WRITE_P, bool BLOCKED>
__global__ void __launch_bounds__(kThreads)
mi_forward_f32_kernel(const float *__restrict__ px, const float *__restrict__ py,
                      const int64_t *__restrict__ boundary, float *__restrict__ p, float *__restrict__ ans,
                      float *__restrict__ lattice, int B, int S, int T, int row0_arg, int tries) {
  using M = MiShape<R>;
  constexpr int ROWS = M::kRows, PITCH = M::kRing, G = M::kGroup;
  constexpr int off = MODIFIED ? -1 : 0;
  extern __shared__ __align__(16) float smem[];
  float *ringx = smem;                           // [2][kStep][PITCH]
  float *ringy = ringx + 2 * kStep * PITCH;      // [2][kStep][PITCH]
  float *ringw = ringy + 2 * kStep * PITCH;      // [2][kStep][PITCH]  exponents of the weights
  // p by block diagonal (mod kEdgeRing) of the row above this CTA's first row
  float *above = ringw + 2 * kStep * PITCH;
  // [kSlots] edge row arrived from the CTA above, [kSlots] edge row taken by the CTA below
  uint64_t *bars = reinterpret_cast<uint64_t *>(above + kEdgeRing);
  float *own = reinterpret_cast<float *>(bars + 2 * kSlots);  // [2][kStep]  p of this CTA's last row
  const int rank = CLUSTER ? cluster_rank() : 0, ranks = CLUSTER ? cluster_size() : 1;
  const int row0 = BLOCKED ? row0_arg : 0;
  const int b = blockIdx.x / ranks;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int T1 = MODIFIED ? T : T + 1;
  const MiBox box = load_box(boundary, b, S, T);
  // block row i <-> lattice row row0 + i, block diagonal k = i + t'; this CTA holds block rows
  // [first, first + ROWS)
  const int ib = min(ranks * ROWS - 1, box.sb - row0);
  if (ib < 0) return;                            // the whole cluster
  const int first = rank * ROWS;
  const int nd = ib + box.tb + 1;
  const int nchunks = (nd + kStep - 1) / kStep;
  const float *X = px + (size_t)b * S * T1;
  const float *Y = py + (size_t)b * (S + 1) * T;
  const int lpitch = lattice_pitch(S);
  const float ninf = -INFINITY;
  float *edge = lattice != nullptr ? edges_of(lattice, b, B, S, T) : nullptr;
  const int blk = row0 / kMiF32Rows;
  float *edge_out = edge + (size_t)(blk & 1) * edge_elems(S, T);
  const float *edge_in = edge + (size_t)((blk + 1) & 1) * edge_elems(S, T);
  const bool keep = lattice != nullptr;
  const bool has_rows = first <= ib;

  for (int j = threadIdx.x; j < kEdgeRing; j += kThreads) above[j] = ninf;
  if (CLUSTER) {
    if (threadIdx.x == 0) slot_init(bars);
    cluster_sync();
    if (!has_rows) {
      cluster_sync();  // the one at the end
      return;
    }
  }

  // Helper warps.  A lane takes R rows of one diagonal at a time: fetch() reads
  // x = px[s0+i-1][t0+t'+o] and y = py[s0+i][t0+t'-1] of the cells (row i, diagonal k) of
  // chunk c into registers, place() stores them in the rings one barrier later, so
  // that a whole chunk's time covers the latency of global memory.
  const bool helper = (warp & 3) != 0;
  const int hw = warp - 1 - (warp >> 2), hj = lane & (kStep - 1), half = lane / kStep;
  float xv[M::kTasksPerWarp][R], yv[M::kTasksPerWarp][R], ev = ninf;
  auto fetch = [&](int c) {
#pragma unroll
    for (int n = 0; n < M::kTasksPerWarp; ++n) {
      const int task = hw + n * kHelpers;
      const int q0 = first + R * (2 * task + half);
      const int tp0 = c * kStep + hj - q0;  // t' of the first row's cell
      const float *xs = X + (long long)(box.s0 + row0 + q0 - 1) * T1 + (box.t0 + tp0 + off);
      const float *ys = Y + (long long)(box.s0 + row0 + q0) * T + (box.t0 + tp0 - 1);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool row_ok = q0 + r <= ib && task < M::kTasks;
        const bool vx = row_ok && row0 + q0 + r >= 1 && (unsigned)(tp0 - r + off) < (unsigned)(box.tb + off + 1);
        const bool vy = row_ok && (unsigned)(tp0 - r - 1) < (unsigned)box.tb;
        xv[n][r] = vx ? xs[(long long)r * (T1 - 1)] : ninf;
        yv[n][r] = vy ? ys[(long long)r * (T - 1)] : 0.f;
      }
    }
    if (BLOCKED && rank == 0 && row0 > 0 && hw == 0 && lane < kStep) {
      // p of cell (row0 - 1, t') of the block above; the steps of a chunk read diagonals up to
      // kStep * c + kStep - 2
      const int d = c * kStep - 1 + lane;
      ev = d + 1 <= box.tb ? edge_in[row0 + d] : ninf;
    }
  };
  auto place = [&](int c) {
#pragma unroll
    for (int n = 0; n < M::kTasksPerWarp; ++n) {
      const int task = hw + n * kHelpers;
      const int at = ((c & 1) * kStep + hj) * PITCH + R * (2 * task + half);
      if (task < M::kTasks) {
        store_rows<R>(ringx + at, xv[n]);
        store_rows<R>(ringy + at, yv[n]);
      }
    }
    if (BLOCKED && rank == 0 && row0 > 0 && hw == 0 && lane < kStep)
      above[(c * kStep - 1 + lane + kEdgeRing) % kEdgeRing] = ev;
  };
  // weights of what chunk c left in ringw, four rows of one diagonal at a time
  float *L = keep ? lattice_of(lattice, b, S, T) + (size_t)row0 * lpitch + row0 : nullptr;
  auto weights = [&](int c) {
#pragma unroll
    for (int n = 0; n < M::kQuadsPerLane; ++n) {
      const int q = (n * kHelpers + hw) * 32 + lane;
      const int l0 = 4 * (q % (ROWS / 4)), j = q / (ROWS / 4), q0 = first + l0;
      const int k = c * kStep + j;
      if (q >= M::kQuads || k < 0 || k >= nd || row0 + q0 >= lpitch) continue;
      float w[4];
      load_rows<4>(w, ringw + ((c & 1) * kStep + j) * PITCH + l0);
#pragma unroll
      for (int r = 0; r < 4; ++r) w[r] = mi_weight(w[r]);
      store_rows<4>(L + (size_t)k * lpitch + q0, w);
    }
  };

  if (BLOCKED) __syncthreads();  // `above` is filled by the helpers, too
  if (helper) {
    fetch(0);
    place(0);
    if (nchunks > 1) fetch(1);
  }
  __syncthreads();

  const int i0 = first + lane * R;               // this lane's first block row
  float p_cur[R], p_old[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    // the origin: LogAdd(-inf, 0 + 0) = 0 at its only step
    p_cur[r] = row0 + i0 + r == 0 ? 0.f : ninf;
    p_old[r] = ninf;
  }
  float *P = WRITE_P ? p + (size_t)b * (S + 1) * (T + 1) : nullptr;
  // this CTA's last row for the one below, by the warp that has nothing else to do
  const bool has_next = CLUSTER && first + ROWS <= ib;
  const bool sender = CLUSTER && warp == 4;
  const unsigned next = has_next ? peer_address(above, rank + 1) : 0u;
  const unsigned next_full = has_next ? peer_address(bars, rank + 1) : 0u;
  const unsigned prev_taken = CLUSTER && rank > 0 ? peer_address(bars + kSlots, rank - 1) : 0u;
  bool late = false;
  auto pass_on = [&](int c) {
    if (rank > 0 && lane == 0) slot_arrive(prev_taken, c);
    if (has_next && lane < min(kStep, nd - c * kStep)) {
      if (c >= kSlots - 1) late = slot_wait(bars + kSlots, c - (kSlots - 1), late, tries);
      peer_send(next + 4 * ((c * kStep + lane) & (kEdgeRing - 1)), late ? NAN : own[(c & 1) * kStep + lane],
                next_full + 8 * (c % kSlots));
    }
  };
  bool failed = false;

  for (int c = 0; c < nchunks; ++c) {
    if (helper) {
      if (c + 1 < nchunks) place(c + 1);
      if (c + 2 < nchunks) fetch(c + 2);
      if (keep && c >= 1) weights(c - 1);
    } else if (warp == 0) {
      if (CLUSTER && rank > 0) {
        // (after a failure no more arrivals: the barrier's phase may not have ended)
        if (lane == 0 && !failed) slot_expect(bars, c, min(kStep, nd - c * kStep));
        failed = slot_wait(bars, c, failed, tries);
      }
      float *rw = ringw + (c & 1) * kStep * PITCH + lane * R;
      const float *rx = ringx + (c & 1) * kStep * PITCH + lane * R;
      const float *ry = ringy + (c & 1) * kStep * PITCH + lane * R;
      const int nstep = min(kStep, nd - c * kStep);
      float x[2][G][R], y[2][G][R], nb[2][G];
      auto inputs = [&](int j0, int s) {
#pragma unroll
        for (int u = 0; u < G; ++u) {
          load_rows<R>(x[s][u], rx + (j0 + u) * PITCH);
          load_rows<R>(y[s][u], ry + (j0 + u) * PITCH);
          nb[s][u] = above[(c * kStep + j0 + u - 1 + off) & (kEdgeRing - 1)];
          if (CLUSTER && failed) nb[s][u] = NAN;
        }
      };
      auto step = [&](int j, const float (&xs)[R], const float (&ys)[R], float from_above) {
        const int k = c * kStep + j;
        const float up = __shfl_up_sync(0xffffffffu, MODIFIED ? p_old[R - 1] : p_cur[R - 1], 1);
        float pn[R], dl[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float a;
          if (r == 0) {
            a = from_above + xs[0];
            add_if(a, lane != 0, up, xs[0]);
          } else {
            a = (MODIFIED ? p_old[r - 1] : p_cur[r - 1]) + xs[r];
          }
          pn[r] = log_add_f32(a, p_cur[r] + ys[r]);
          dl[r] = a - pn[r];  // exponent of this cell's backward weight
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          p_old[r] = p_cur[r];
          p_cur[r] = pn[r];
        }
        if (CLUSTER && lane == 31) own[(c & 1) * kStep + j] = p_cur[R - 1];
        if (keep) store_rows<R>(rw + j * PITCH, dl);
        if (BLOCKED && i0 + R == kMiF32Rows) edge_out[row0 + k] = p_cur[R - 1];
        if (WRITE_P) {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int i = i0 + r, tp = k - i;
            if (i <= ib && tp >= 0 && tp <= box.tb)
              P[(size_t)(box.s0 + row0 + i) * (T + 1) + box.t0 + tp] = p_cur[r];
          }
        }
      };
      inputs(0, 0);
      if (nstep == kStep) {
#pragma unroll
        for (int j0 = 0; j0 < kStep; j0 += G) {
          const int s = (j0 / G) & 1;
          if (j0 + G < kStep) inputs(j0 + G, s ^ 1);
#pragma unroll
          for (int u = 0; u < G; ++u) step(j0 + u, x[s][u], y[s][u], nb[s][u]);
        }
      } else {  // the last chunk ends with diagonal nd - 1
#pragma unroll 1
        for (int j0 = 0; j0 < nstep; j0 += G) {
          inputs(j0, 0);
#pragma unroll
          for (int u = 0; u < G; ++u)
            if (j0 + u < nstep) step(j0 + u, x[0][u], y[0][u], nb[0][u]);
        }
      }
    } else if (sender && c >= 1) {
      pass_on(c - 1);
    }
    __syncthreads();
  }
  if (helper && keep) weights(nchunks - 1);
  if (sender) pass_on(nchunks - 1);
  // the last step of a row is diagonal nd - 1, where the last row reaches its end
  if (warp == 0) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (row0 + i0 + r == box.sb) ans[b] = p_cur[r];
  }
  if (CLUSTER) leave_cluster(failed);
}

// -----------------------------------------------------------------------------
// backward
// -----------------------------------------------------------------------------
template <int R, bool CLUSTER, bool MODIFIED, bool BLOCKED>
__global__ void __launch_bounds__(kThreads)
mi_backward_f32_kernel(float *__restrict__ lattice, const int64_t *__restrict__ boundary,
                       const float *__restrict__ ans_grad, float *__restrict__ px_grad,
                       float *__restrict__ py_grad, float *__restrict__ origin_grad, int B, int S, int T,
                       int row0_arg, int tries) {
  using M = MiShape<R>;
  constexpr int ROWS = M::kRows, PITCH = M::kRing, G = M::kGroup;
  constexpr int off = MODIFIED ? -1 : 0;
  extern __shared__ __align__(16) float smem[];
  float *ringx = smem;                           // [2][kStep][PITCH]  d/dpx
  float *ringy = ringx + 2 * kStep * PITCH;      // [2][kStep][PITCH]  d/dpy
  float *ringw = ringy + 2 * kStep * PITCH;      // [2][kStep][PITCH]  weights
  // x-gradients by block diagonal (mod kEdgeRing) of the row below this CTA's last row
  float *below = ringw + 2 * kStep * PITCH;
  // [kSlots] edge row arrived from the CTA below, [kSlots] edge row taken by the CTA above
  uint64_t *bars = reinterpret_cast<uint64_t *>(below + kEdgeRing);
  float *own = reinterpret_cast<float *>(bars + 2 * kSlots);  // [2][kStep]  this CTA's first row
  const int rank = CLUSTER ? cluster_rank() : 0, ranks = CLUSTER ? cluster_size() : 1;
  const int row0 = BLOCKED ? row0_arg : 0;
  const int b = blockIdx.x / ranks;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int T1 = MODIFIED ? T : T + 1;
  const MiBox box = load_box(boundary, b, S, T);
  const int ib = min(ranks * ROWS - 1, box.sb - row0);
  const int first = rank * ROWS;
  const int nd = ib >= 0 ? ib + box.tb + 1 : 0;
  const int nchunks = (nd + kStep - 1) / kStep;
  float *GX = px_grad + (size_t)b * S * T1;
  float *GY = py_grad + (size_t)b * (S + 1) * T;
  const int lpitch = lattice_pitch(S);
  const float *LT = lattice_of(lattice, b, S, T);
  float *edge = edges_of(lattice, b, B, S, T);
  const int blk = row0 / kMiF32Rows;
  float *edge_out = edge + (size_t)(blk & 1) * edge_elems(S, T);
  const float *edge_in = edge + (size_t)((blk + 1) & 1) * edge_elems(S, T);
  const bool block_below = BLOCKED && row0 + kMiF32Rows <= box.sb;
  const bool has_rows = first <= ib;

  for (int j = threadIdx.x; j < kEdgeRing; j += kThreads) below[j] = 0.f;
  if (BLOCKED) __syncthreads();  // `below` is filled by the helpers, too

  // the chunk of diagonals that is the n-th of the sweep
  auto chunk_of = [&](int n) { return nchunks - 1 - n; };

  // Helper warps.  fetch() reads the weights of the it-th chunk into registers (four rows of one
  // diagonal per lane), place() stores them in the ring one barrier later; drain() writes the
  // gradients of a chunk out, a lane taking R rows of one diagonal at a time.
  const bool helper = (warp & 3) != 0;
  const int hw = warp - 1 - (warp >> 2), hj = lane & (kStep - 1), half = lane / kStep;
  float wv[M::kQuadsPerLane][4], ev = 0.f;
  auto fetch = [&](int it) {
#pragma unroll
    for (int n = 0; n < M::kQuadsPerLane; ++n) {
      const int q = (n * kHelpers + hw) * 32 + lane;
      const int q0 = first + 4 * (q % (ROWS / 4)), k = chunk_of(it) * kStep + q / (ROWS / 4);
#pragma unroll
      for (int r = 0; r < 4; ++r) wv[n][r] = kMiDead;
      if (q < M::kQuads && q0 <= ib && k >= 0 && k < nd)
        load_rows<4>(wv[n], LT + (size_t)(row0 + k) * lpitch + row0 + q0);
    }
    if (BLOCKED && rank == ranks - 1 && hw == 0 && lane < kStep) {
      // what cell (row0 + kMiF32Rows, t') of the block below sent up, by its block diagonal
      const int d = chunk_of(it) * kStep + 1 - off + lane;
      ev = block_below && d >= kMiF32Rows && d - kMiF32Rows <= box.tb ? edge_in[row0 + d] : 0.f;
    }
  };
  auto place = [&](int it) {
#pragma unroll
    for (int n = 0; n < M::kQuadsPerLane; ++n) {
      const int q = (n * kHelpers + hw) * 32 + lane;
      const int l0 = 4 * (q % (ROWS / 4)), j = q / (ROWS / 4);
      const int tp0 = chunk_of(it) * kStep + j - first - l0;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        // first column: only an x-predecessor (regular) or none; first row: only a y-predecessor;
        // what the lattice holds outside the box is not defined
        if (tp0 - r == 0) wv[n][r] = MODIFIED ? kMiDead : 1.f;
        if (r == 0 && row0 + first + l0 == 0) wv[n][r] = 0.f;
        if (first + l0 + r > ib || (unsigned)(tp0 - r) > (unsigned)box.tb) wv[n][r] = kMiDead;
      }
      if (q < M::kQuads) store_rows<4>(ringw + ((it & 1) * kStep + j) * PITCH + l0, wv[n]);
    }
    if (BLOCKED && rank == ranks - 1 && hw == 0 && lane < kStep)
      below[(chunk_of(it) * kStep + 1 - off + lane) & (kEdgeRing - 1)] = ev;
  };
  auto drain = [&](int it) {
    const int c = chunk_of(it);
#pragma unroll
    for (int n = 0; n < M::kTasksPerWarp; ++n) {
      const int task = hw + n * kHelpers;
      const int l0 = R * (2 * task + half), q0 = first + l0;
      if (task >= M::kTasks) continue;
      const int at = ((it & 1) * kStep + hj) * PITCH + l0;
      float gx[R], gy[R];
      load_rows<R>(gx, ringx + at);
      load_rows<R>(gy, ringy + at);
      const int tp0 = c * kStep + hj - q0;
      float *xs = GX + (long long)(box.s0 + row0 + q0 - 1) * T1 + (box.t0 + tp0 + off);
      float *ys = GY + (long long)(box.s0 + row0 + q0) * T + (box.t0 + tp0 - 1);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool row_ok = q0 + r <= ib;
        if (row_ok && row0 + q0 + r >= 1 && (unsigned)(tp0 - r + off) < (unsigned)(box.tb + off + 1))
          xs[(long long)r * (T1 - 1)] = gx[r];
        if (row_ok && (unsigned)(tp0 - r - 1) < (unsigned)box.tb) ys[(long long)r * (T - 1)] = gy[r];
      }
    }
  };

  if (CLUSTER && threadIdx.x == 0) slot_init(bars);
  const bool works = has_rows && nchunks > 0;
  if (helper && works) {
    fetch(0);
    place(0);
    if (nchunks > 1) fetch(1);
  }
  if (CLUSTER)
    cluster_sync();
  else
    __syncthreads();

  if (helper && row0 == 0) {
    // exact zeros outside the boundary box (mutual_information_cpu.cu:161-166), dealt out over
    // the cluster's helpers
    const int lw = rank * kHelpers + hw, nlw = ranks * kHelpers;
    const int cx_lo = box.t0, cx_hi = box.t0 + box.tb + off;  // inclusive, in-box columns of px_grad
    for (int r = lw; r < S; r += nlw) {
      const bool in_rows = r >= box.s0 && r < box.s0 + box.sb;
      if (in_rows && cx_lo == 0 && cx_hi == T1 - 1) continue;
      for (int col = lane; col < T1; col += 32)
        if (!in_rows || col < cx_lo || col > cx_hi) GX[(size_t)r * T1 + col] = 0;
    }
    const int cy_lo = box.t0, cy_hi = box.t0 + box.tb - 1;
    for (int r = lw; r <= S; r += nlw) {
      const bool in_rows = r >= box.s0 && r <= box.s0 + box.sb;
      if (in_rows && cy_lo == 0 && cy_hi == T - 1) continue;
      for (int col = lane; col < T; col += 32)
        if (!in_rows || col < cy_lo || col > cy_hi) GY[(size_t)r * T + col] = 0;
    }
  }

  const int i0 = first + lane * R;
  float g1_cur[R], g1_old[R], g2_cur[R];
  float g_first = 0.f;  // gradient of the first row's cell handled last: what reaches the origin
  const float g_end = ans_grad[b];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    g1_cur[r] = g1_old[r] = 0.f;
    // cell (sb, tb) is its row's first step (diagonal nd - 1)
    g2_cur[r] = row0 + i0 + r == box.sb ? g_end : 0.f;
  }
  // this CTA's first row for the one above, by the warp that has nothing else to do
  const bool has_next = CLUSTER && first + ROWS <= ib;  // rows below
  const bool sender = CLUSTER && warp == 4;
  const unsigned previous = CLUSTER && rank > 0 ? peer_address(below, rank - 1) : 0u;
  const unsigned previous_full = CLUSTER && rank > 0 ? peer_address(bars, rank - 1) : 0u;
  const unsigned next_taken = has_next ? peer_address(bars + kSlots, rank + 1) : 0u;
  bool late = false;
  auto pass_on = [&](int it) {
    const int c = chunk_of(it);
    if (has_next && lane == 0) slot_arrive(next_taken, it);
    if (rank > 0 && lane < min(kStep, nd - c * kStep)) {
      if (it >= kSlots - 1) late = slot_wait(bars + kSlots, it - (kSlots - 1), late, tries);
      peer_send(previous + 4 * ((c * kStep + lane) & (kEdgeRing - 1)), late ? NAN : own[(it & 1) * kStep + lane],
                previous_full + 8 * (it % kSlots));
    }
  };
  bool failed = false;

  for (int it = 0; works && it < nchunks; ++it) {
    const int c = chunk_of(it);
    if (helper) {
      if (it + 1 < nchunks) place(it + 1);
      if (it + 2 < nchunks) fetch(it + 2);
      if (it >= 1) drain(it - 1);
    } else if (warp == 0) {
      if (has_next) {
        if (lane == 0 && !failed) slot_expect(bars, it, min(kStep, nd - c * kStep));
        failed = slot_wait(bars, it, failed, tries);
      }
      float *rx = ringx + (it & 1) * kStep * PITCH + lane * R;
      float *ry = ringy + (it & 1) * kStep * PITCH + lane * R;
      const float *rw = ringw + (it & 1) * kStep * PITCH + lane * R;
      const int nstep = min(kStep, nd - c * kStep);
      float w[2][G][R], nb[2][G];
      auto inputs = [&](int j0, int s) {
#pragma unroll
        for (int u = 0; u < G; ++u) {
          load_rows<R>(w[s][u], rw + (j0 + u) * PITCH);
          nb[s][u] = below[(c * kStep + j0 + u + 1 - off) & (kEdgeRing - 1)];
          if (CLUSTER && failed) nb[s][u] = NAN;
        }
      };
      auto step = [&](int j, const float (&wt)[R], float edge_below) {
        const int k = c * kStep + j;
        const float up = __shfl_down_sync(0xffffffffu, MODIFIED ? g1_old[0] : g1_cur[0], 1);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float g;
          if (r == R - 1) {
            g = edge_below + g2_cur[r];
            add_if(g, lane != 31, up, g2_cur[r]);
          } else {  // row r + 1 is still at the step before
            g = (MODIFIED ? g1_old[r + 1] : g1_cur[r + 1]) + g2_cur[r];
          }
          if (r == 0) g_first = g;
          if (MODIFIED) g1_old[r] = g1_cur[r];
          g1_cur[r] = fmaxf(wt[r], 0.f) * g;                  // share of the x-predecessor
          g2_cur[r] = (wt[r] < 0.f ? 0.f : 1.f - wt[r]) * g;  // share of the y-predecessor
        }
        store_rows<R>(rx + j * PITCH, g1_cur);
        store_rows<R>(ry + j * PITCH, g2_cur);
        if (CLUSTER && lane == 0) own[(it & 1) * kStep + j] = g1_cur[0];
        if (BLOCKED && row0 > 0 && i0 == 0) edge_out[row0 + k] = g1_cur[0];
      };
      if (nstep == kStep) {
        inputs(kStep - G, 0);
#pragma unroll
        for (int j0 = kStep - G; j0 >= 0; j0 -= G) {
          const int s = ((kStep - G - j0) / G) & 1;
          if (j0 > 0) inputs(j0 - G, s ^ 1);
#pragma unroll
          for (int u = G - 1; u >= 0; --u) step(j0 + u, w[s][u], nb[s][u]);
        }
      } else {  // the first chunk begins with diagonal nd - 1
#pragma unroll 1
        for (int j0 = (nstep - 1) / G * G; j0 >= 0; j0 -= G) {
          inputs(j0, 0);
#pragma unroll
          for (int u = G - 1; u >= 0; --u)
            if (j0 + u < nstep) step(j0 + u, w[0][u], nb[0][u]);
        }
      }
    } else if (sender && it >= 1) {
      pass_on(it - 1);
    }
    __syncthreads();
  }
  if (helper && works) drain(nchunks - 1);
  if (sender && works) pass_on(nchunks - 1);
  if (threadIdx.x == 0 && rank == 0 && row0 == 0 && origin_grad != nullptr) origin_grad[b] = g_first;
  if (CLUSTER) leave_cluster(failed);
}

// -----------------------------------------------------------------------------
// host side
// -----------------------------------------------------------------------------
template <bool CLUSTER, class Kernel, class... Args>
static int launch(Kernel kern, int B, int ranks, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)B * (unsigned)ranks);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ranks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CLUSTER ? 1 : 0;
  count_launch();
  FRNNT_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
  return FRNNT_OK;
}

template <bool MODIFIED, bool WRITE_P>
static int forward_f32(const float *px, const float *py, const int64_t *boundary, float *p, float *ans,
                       float *lattice, int B, int S, int T, int tries, cudaStream_t st) {
  if (S + 1 <= MiShape<1>::kRows)
    return launch<false>(mi_forward_f32_kernel<1, false, MODIFIED, WRITE_P, false>, B, 1, MiShape<1>::kSmem, st, px,
                         py, boundary, p, ans, lattice, B, S, T, 0, tries);
  if (S + 1 <= MiShape<2>::kRows)
    return launch<false>(mi_forward_f32_kernel<2, false, MODIFIED, WRITE_P, false>, B, 1, MiShape<2>::kSmem, st, px,
                         py, boundary, p, ans, lattice, B, S, T, 0, tries);
  if (S + 1 <= kMiF32Rows)
    return launch<true>(mi_forward_f32_kernel<2, true, MODIFIED, WRITE_P, false>, B,
                        (S + MiShape<2>::kRows) / MiShape<2>::kRows, MiShape<2>::kSmem, st, px, py, boundary, p, ans,
                        lattice, B, S, T, 0, tries);
  // more rows than one cluster holds: one launch per block of rows, top to bottom
  for (int row0 = 0; row0 <= S; row0 += kMiF32Rows) {
    const int rc = launch<true>(mi_forward_f32_kernel<2, true, MODIFIED, WRITE_P, true>, B, kMaxCluster,
                                MiShape<2>::kSmem, st, px, py, boundary, p, ans, lattice, B, S, T, row0, tries);
    if (rc != FRNNT_OK) return rc;
  }
  return FRNNT_OK;
}

template <bool MODIFIED>
static int backward_f32(float *lattice, const int64_t *boundary, const float *ans_grad, float *px_grad,
                        float *py_grad, float *origin_grad, int B, int S, int T, int tries,
                        cudaStream_t st) {
  if (S + 1 <= MiShape<1>::kRows)
    return launch<false>(mi_backward_f32_kernel<1, false, MODIFIED, false>, B, 1, MiShape<1>::kSmem, st, lattice,
                         boundary, ans_grad, px_grad, py_grad, origin_grad, B, S, T, 0, tries);
  if (S + 1 <= MiShape<2>::kRows)
    return launch<false>(mi_backward_f32_kernel<2, false, MODIFIED, false>, B, 1, MiShape<2>::kSmem, st, lattice,
                         boundary, ans_grad, px_grad, py_grad, origin_grad, B, S, T, 0, tries);
  if (S + 1 <= kMiF32Rows)
    return launch<true>(mi_backward_f32_kernel<2, true, MODIFIED, false>, B,
                        (S + MiShape<2>::kRows) / MiShape<2>::kRows, MiShape<2>::kSmem, st, lattice, boundary,
                        ans_grad, px_grad, py_grad, origin_grad, B, S, T, 0, tries);
  // bottom to top
  for (int row0 = (S / kMiF32Rows) * kMiF32Rows; row0 >= 0; row0 -= kMiF32Rows) {
    const int rc = launch<true>(mi_backward_f32_kernel<2, true, MODIFIED, true>, B, kMaxCluster, MiShape<2>::kSmem,
                                st, lattice, boundary, ans_grad, px_grad, py_grad, origin_grad, B, S, T, row0, tries);
    if (rc != FRNNT_OK) return rc;
  }
  return FRNNT_OK;
}
static_assert(kMaxCluster * MiShape<2>::kRows == kMiF32Rows, "a full cluster holds a block");

int launch_mi_forward_f32(const float *px, const float *py, const int64_t *boundary, float *p, float *ans,
                          float *lattice, int B, int S, int T, int modified, cudaStream_t st,
                          int tries) {
  if (p != nullptr)
    return modified ? forward_f32<true, true>(px, py, boundary, p, ans, lattice, B, S, T, tries, st)
                    : forward_f32<false, true>(px, py, boundary, p, ans, lattice, B, S, T, tries, st);
  return modified ? forward_f32<true, false>(px, py, boundary, p, ans, lattice, B, S, T, tries, st)
                  : forward_f32<false, false>(px, py, boundary, p, ans, lattice, B, S, T, tries, st);
}

int launch_mi_backward_f32(float *lattice, const int64_t *boundary, const float *ans_grad, float *px_grad,
                           float *py_grad, float *origin_grad, int B, int S, int T, int modified,
                           cudaStream_t st, int tries) {
  return modified ? backward_f32<true>(lattice, boundary, ans_grad, px_grad, py_grad, origin_grad, B, S, T, tries, st)
                  : backward_f32<false>(lattice, boundary, ans_grad, px_grad, py_grad, origin_grad, B, S, T, tries, st);
}

}  // namespace frnnt
