// Factorisations executed by one thread block of TTB_THREADS threads:
// Householder QR, Jacobi SVD and pivoted Gaussian elimination.
//
// The matrices of tensor-train work are small (columns a bond, rows a bond
// times a mode), so what bounds their factorisation on one SM is the chain
// of column steps: a reduction, a scale factor, an update, a barrier.  The
// register-tiled routines keep whole columns in registers, eight lanes to a
// column where the rows allow it: a column step is one dot product per
// column, three shuffle levels for four columns of a warp together, one
// update, and one block barrier in all.
//
// They are compiled once, here, and called from the kernels of the other
// files (relocatable device code): inlined into every kernel, ptxas spent
// minutes on each.
#include <cooperative_groups.h>

#include "ttb_factor.cuh"

namespace ttb {

// ---------------------------------------------------------------------------
// Householder QR
// ---------------------------------------------------------------------------

// cta_householder where each thread has one row of a step at most (m <= 1 + 32
// NV): its entries and sums, bit for bit, with a warp per column and one barrier
// a step.  That form's warp ``w`` sums the rows j + 1 + 32 w + lane, so a warp
// here makes those sums one by one and adds them in the same order.  Every warp
// scales the reflector for itself in registers; the column is overwritten a step
// later, when nobody reads it.  The warp that updates column j + 1 hands out its
// norm.  A lone solve of a 2^16-unknown Poisson system, some 230 factorisations
// of 10 to 50 rows, takes 55.1 ms where six barriers a step took 60.7 ms; the
// smallest (2^6 unknowns) 4.3 against 4.7 ms.
template <int NV>
static __device__ __noinline__ void cta_householder_short(double* W, int m, int k, i64 ldw,
                                                          double* tau) {
  constexpr int CB = NV <= 2 ? 3 : 2;  // columns of a warp in flight
  __shared__ double nsig[2];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int p = min(m, k);
  if (wid == 0) {
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < NV; ++w) {
      const int i = 1 + 32 * w + lane;
      const double x = i < m ? W[i] : 0.0;
      sum += warp_sum(fma(x, x, 0.0));
    }
    if (lane == 0) nsig[0] = sum;
  }
  __syncthreads();
  double late_beta = 0.0, late_t = 0.0, late_scale = 0.0;
  bool late_scaled = false;
  // column j as it stays: beta, the scaled reflector, its scalar
  auto finish = [&](int j) {
    double* col = W + j * ldw;
    if (late_scaled)
      for (int i = j + 1 + lane; i < m; i += 32) col[i] *= late_scale;
    if (lane == 0) {
      col[j] = late_beta;
      tau[j] = late_t;
    }
  };
  for (int j = 0; j < p; ++j) {
    const double* col = W + j * ldw;
    const double alpha = col[j], sigma = nsig[j & 1];
    if (j > 0 && wid == TTB_WARPS - 1) finish(j - 1);
    double t = 0.0, beta = alpha, scale = 0.0;
    double v[NV];
#pragma unroll
    for (int w = 0; w < NV; ++w) {
      const int i = j + 1 + 32 * w + lane;
      v[w] = i < m ? col[i] : 0.0;
    }
    if (sigma != 0.0) {
      const double nrm = sqrt(alpha * alpha + sigma);
      beta = (alpha >= 0.0) ? -nrm : nrm;
      t = (beta - alpha) / beta;
      scale = 1.0 / (alpha - beta);
#pragma unroll
      for (int w = 0; w < NV; ++w) v[w] *= scale;
    }
    late_beta = beta;
    late_t = t;
    late_scale = scale;
    late_scaled = sigma != 0.0;
    if (t != 0.0) {
      for (int c0 = j + 1 + wid; c0 < k; c0 += CB * TTB_WARPS) {
        double x[CB][NV], sw[CB], top[CB];
#pragma unroll
        for (int b = 0; b < CB; ++b) {
          const int c = c0 + b * TTB_WARPS;
          const double* from = W + c * ldw;
          top[b] = c < k ? from[j] : 0.0;
#pragma unroll
          for (int w = 0; w < NV; ++w) {
            const int i = j + 1 + 32 * w + lane;
            x[b][w] = (c < k && i < m) ? from[i] : 0.0;
          }
        }
#pragma unroll
        for (int b = 0; b < CB; ++b) sw[b] = 0.0;
#pragma unroll
        for (int w = 0; w < NV; ++w)
#pragma unroll
          for (int b = 0; b < CB; ++b) sw[b] += warp_sum(fma(v[w], x[b][w], 0.0));
        double next = 0.0;
#pragma unroll
        for (int b = 0; b < CB; ++b) {
          const int c = c0 + b * TTB_WARPS;
          if (c >= k) continue;
          double* to = W + c * ldw;
          const double wv = t * (sw[b] + top[b]);
          if (lane == 0) to[j] = top[b] - wv;
#pragma unroll
          for (int w = 0; w < NV; ++w) {
            const int i = j + 1 + 32 * w + lane;
            const double y = fma(-wv, v[w], x[b][w]);
            if (i < m) to[i] = y;
            x[b][w] = (i < m && i > j + 1) ? y : 0.0;
          }
        }
        if (c0 == j + 1) {
#pragma unroll
          for (int w = 0; w < NV; ++w) next += warp_sum(fma(x[0][w], x[0][w], 0.0));
          if (lane == 0) nsig[(j + 1) & 1] = next;
        }
      }
    } else if (wid == 0 && j + 1 < p) {
      const double* cn = W + (j + 1) * ldw;
      double next = 0.0;
#pragma unroll
      for (int w = 0; w < NV; ++w) {
        const int i = j + 2 + 32 * w + lane;
        const double x = i < m ? cn[i] : 0.0;
        next += warp_sum(fma(x, x, 0.0));
      }
      if (lane == 0) nsig[(j + 1) & 1] = next;
    }
    __syncthreads();
  }
  if (p > 0 && wid == TTB_WARPS - 1) finish(p - 1);
  __syncthreads();
}

// The general form.  The whole block works on every reflector: the trailing
// columns are taken kHC at a time, their dot products with v accumulated per
// thread over a row stripe and reduced together, and the squared norm of the
// next column is gathered during its update (one pass fewer per column).
// SHARED: W is in shared memory, and the compiler may take it for granted (R of
// 4096 x 3 takes 31 us so and 44 us through generic addresses).
constexpr int kHC = 16;
template <bool SHARED>
static __device__ __forceinline__ void householder_passes(double* W, int m, int k, i64 ldw,
                                                          double* tau, double* red,
                                                          double (&hred)[TTB_WARPS][kHC],
                                                          double (&hw)[kHC]) {
  if constexpr (SHARED) __builtin_assume(__isShared(W));
  const int p = m < k ? m : k;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double part = 0.0;
  for (int i = 1 + tid; i < m; i += TTB_THREADS) part = fma(W[i], W[i], part);
  double sigma = block_sum(part, red);
  for (int j = 0; j < p; ++j) {
    double* col = W + j * ldw;
    const double alpha = col[j];
    double t = 0.0, beta = alpha, scale = 0.0;
    if (sigma != 0.0) {
      const double nrm = sqrt(alpha * alpha + sigma);
      beta = (alpha >= 0.0) ? -nrm : nrm;
      t = (beta - alpha) / beta;
      scale = 1.0 / (alpha - beta);
    }
    __syncthreads();  // everyone has read col[j] before it is overwritten
    if (sigma != 0.0) {
      for (int i = j + 1 + tid; i < m; i += TTB_THREADS) col[i] *= scale;
    }
    if (tid == 0) {
      col[j] = beta;
      tau[j] = t;
    }
    __syncthreads();
    double next = 0.0;  // this thread's part of |column j+1, rows > j+1|^2
    for (int c0 = j + 1; c0 < k; c0 += kHC) {
      const int nc = min(kHC, k - c0);
      double* cb = W + (i64)c0 * ldw;
      if (t != 0.0) {
        double w[kHC];
#pragma unroll
        for (int q = 0; q < kHC; ++q) w[q] = 0.0;
        for (int i = j + 1 + tid; i < m; i += TTB_THREADS) {
          const double v = col[i];
#pragma unroll
          for (int q = 0; q < kHC; ++q)
            if (q < nc) w[q] = fma(v, cb[i + q * ldw], w[q]);
        }
#pragma unroll
        for (int q = 0; q < kHC; ++q) {
          const double sw = warp_sum(w[q]);
          if (lane == 0) hred[wid][q] = sw;
        }
        __syncthreads();
        if (tid < nc) {
          double sw = 0.0;
          for (int q = 0; q < TTB_WARPS; ++q) sw += hred[q][tid];
          const double wv = t * (sw + cb[j + tid * ldw]);
          hw[tid] = wv;
          cb[j + tid * ldw] -= wv;
        }
        __syncthreads();
        for (int i = j + 1 + tid; i < m; i += TTB_THREADS) {
          const double v = col[i];
#pragma unroll
          for (int q = 0; q < kHC; ++q) {
            if (q < nc) {
              const double x = fma(-hw[q], v, cb[i + q * ldw]);
              cb[i + q * ldw] = x;
              if (q == 0 && c0 == j + 1 && i > j + 1) next = fma(x, x, next);
            }
          }
        }
        __syncthreads();  // hred and hw are reused by the next chunk
      } else if (c0 == j + 1) {
        for (int i = j + 2 + tid; i < m; i += TTB_THREADS) next = fma(cb[i], cb[i], next);
      }
    }
    if (j + 1 < p) sigma = block_sum(next, red);
  }
}

// In-place Householder QR of the m x k matrix W (column step ``ldw``, unit
// row step), as LAPACK dgeqr2 lays it out: on return R is in the upper
// triangle and the reflector vectors v_j (v_j[j] = 1 implied) below the
// diagonal, with the scalars in tau[0 .. min(m,k)-1].  Each reflector is
// H = I - tau v v^T built as in dlarfg: beta = -sign(alpha) ||x||,
// tau = (beta - alpha) / beta, v = x / (alpha - beta); a column whose
// sub-diagonal part is exactly zero gets tau = 0.
static __device__ void cta_householder(double* W, int m, int k, i64 ldw, double* tau, double* red) {
  if (m <= 33) {
    cta_householder_short<1>(W, m, k, ldw, tau);
    return;
  }
  if (m <= 65) {
    cta_householder_short<2>(W, m, k, ldw, tau);
    return;
  }
  if (m <= 129) {
    cta_householder_short<4>(W, m, k, ldw, tau);
    return;
  }
  __shared__ double hred[TTB_WARPS][kHC];
  __shared__ double hw[kHC];
  if (__isShared(W)) householder_passes<true>(W, m, k, ldw, tau, red, hred, hw);
  else householder_passes<false>(W, m, k, ldw, tau, red, hred, hw);
}

// Overwrite the m x q matrix X (strided) with H_0 H_1 ... H_{p-1} X, the
// reflectors of cta_householder (applied last to first).  A warp keeps its
// columns through all reflectors, so no step needs a barrier; two columns of
// up to 128 rows at a time, held in registers between the product and the
// update.
static __device__ void cta_apply_q(const double* W, int m, int p, i64 ldw, const double* tau, Mat X,
                            int q) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (m <= 129) {
    constexpr int NV = 4;
    for (int c0 = wid; c0 < q; c0 += 2 * TTB_WARPS) {
      const int c1 = c0 + TTB_WARPS;
      const bool two = c1 < q;
      for (int j = p - 1; j >= 0; --j) {
        const double t = tau[j];
        if (t == 0.0) continue;
        const double* v = W + j * ldw;
        double x0[NV], x1[NV], vv[NV], w0 = 0.0, w1 = 0.0;
        const double top0 = X(j, c0), top1 = two ? X(j, c1) : 0.0;
#pragma unroll
        for (int r = 0; r < NV; ++r) {
          const int i = j + 1 + lane + 32 * r;
          const bool in = i < m;
          vv[r] = in ? v[i] : 0.0;
          x0[r] = in ? X(i, c0) : 0.0;
          x1[r] = in && two ? X(i, c1) : 0.0;
          if (in) {
            w0 = fma(vv[r], x0[r], w0);
            w1 = fma(vv[r], x1[r], w1);
          }
        }
        w0 = t * (warp_sum(w0) + top0);
        w1 = t * (warp_sum(w1) + top1);
        __syncwarp();
        if (lane == 0) {
          X(j, c0) = top0 - w0;
          if (two) X(j, c1) = top1 - w1;
        }
#pragma unroll
        for (int r = 0; r < NV; ++r) {
          const int i = j + 1 + lane + 32 * r;
          if (i >= m) continue;
          X(i, c0) = fma(-w0, vv[r], x0[r]);
          if (two) X(i, c1) = fma(-w1, vv[r], x1[r]);
        }
        __syncwarp();
      }
    }
    __syncthreads();
    return;
  }
  for (int c = wid; c < q; c += TTB_WARPS) {
    for (int j = p - 1; j >= 0; --j) {
      const double t = tau[j];
      if (t == 0.0) continue;
      const double* v = W + j * ldw;
      double w = 0.0;
      for (int i = j + 1 + lane; i < m; i += 32) w = fma(v[i], X(i, c), w);
      w = warp_sum(w) + X(j, c);
      w *= t;
      __syncwarp();
      if (lane == 0) X(j, c) -= w;
      for (int i = j + 1 + lane; i < m; i += 32) X(i, c) = fma(-w, v[i], X(i, c));
      __syncwarp();
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// register-tiled Householder QR
// ---------------------------------------------------------------------------

// A register tile gives a matrix column to LPC lanes of a warp: lane q of the
// column's group holds the row pairs 2 q + 2 LPC t + {0, 1}, RP rows in all
// (RP LPC rows at most).  A warp works on 32 / LPC columns at once, one per
// group, in each of its SL slots; slot s of warp w holds the columns
// G TTB_WARPS s + G w + group, G = 32 / LPC.
template <int LPC>
static __device__ __forceinline__ int tile_row(int r) {
  return 2 * LPC * (r >> 1) + 2 * (threadIdx.x & (LPC - 1)) + (r & 1);
}
template <int LPC>
static __device__ __forceinline__ int tile_col(int s) {
  constexpr int G = 32 / LPC;
  return G * (TTB_WARPS * s + (threadIdx.x >> 5)) + (threadIdx.x & 31) / LPC;
}

// Sum over a column's lanes, every one of them getting it.
template <int LPC>
static __device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = LPC / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Inner product over this lane's rows, four chains deep.
template <int RP>
static __device__ __forceinline__ double lane_dot(const double (&x)[RP], const double (&y)[RP]) {
  constexpr int C = RP >= 8 ? 4 : 2;
  double a[C];
#pragma unroll
  for (int q = 0; q < C; ++q) a[q] = 0.0;
#pragma unroll
  for (int r = 0; r < RP; ++r) a[r % C] = fma(x[r], y[r], a[r % C]);
#pragma unroll
  for (int q = 2; q < C; q += 2) {
    a[0] += a[q];
    a[1] += a[q + 1];
  }
  return a[0] + a[1];
}

// Column ``col`` of a matrix with unit row step, rows below m (zeros beyond).
// L2: past the first-level cache, for columns that other SMs write.
template <int LPC, int RP, bool L2 = false>
static __device__ __forceinline__ void tile_load(const double* col, int m, double (&x)[RP]) {
  const bool even = (reinterpret_cast<uintptr_t>(col) & 15) == 0;
#pragma unroll
  for (int r = 0; r < RP; r += 2) {
    const int i = tile_row<LPC>(r);
    if (2 * LPC * (r >> 1) + 2 * LPC <= m && even) {
      const double2* from = reinterpret_cast<const double2*>(col + i);
      double2 p;
      if constexpr (L2) p = __ldcg(from);
      else p = *from;
      x[r] = p.x;
      x[r + 1] = p.y;
    } else if constexpr (L2) {
      x[r] = i < m ? __ldcg(col + i) : 0.0;
      x[r + 1] = i + 1 < m ? __ldcg(col + i + 1) : 0.0;
    } else {
      x[r] = i < m ? col[i] : 0.0;
      x[r + 1] = i + 1 < m ? col[i + 1] : 0.0;
    }
  }
}

// Reflector j of the factored panel in W (unit row step, column step ld,
// v[j] = 1 implied, zeros above).  A panel has at most 64 columns, so only
// the first 64 rows need the test.
constexpr int kPanelMax = 64;
template <int LPC, int RP, int TEST = kPanelMax>
static __device__ __forceinline__ void hh_load(const double* W, i64 ld, int m, int j,
                                               double (&v)[RP]) {
  tile_load<LPC, RP>(W + j * ld, m, v);
#pragma unroll
  for (int r = 0; r < RP; ++r) {
    if (2 * LPC * (r >> 1) >= TEST) break;
    const int i = tile_row<LPC>(r);
    if (i <= j) v[r] = i == j ? 1.0 : 0.0;
  }
}

// beta, tau and the scale of a column's reflector (LAPACK dlarfg): alpha its
// pivot entry, sigma the squared norm below it.
static __device__ __forceinline__ void hh_scalars(double alpha, double sigma, double& beta,
                                                  double& tau, double& scale) {
  beta = alpha;
  tau = 0.0;
  scale = 0.0;
  if (sigma != 0.0) {
    const double nrm = sqrt(alpha * alpha + sigma);
    beta = (alpha >= 0.0) ? -nrm : nrm;
    tau = (beta - alpha) / beta;
    scale = __drcp_rn(alpha - beta);
  }
}

// A column in registers becomes reflector j (every group of the warp makes
// its own; the caller keeps the owner's): scaled in place below row j, beta
// at row j.  Returns tau.
template <int LPC, int RP, int TEST = kPanelMax>
static __device__ __forceinline__ double hh_make(double (&x)[RP], int j) {
  double a = 0.0, y[RP];
#pragma unroll
  for (int r = 0; r < RP; ++r) {
    const int i = tile_row<LPC>(r);
    y[r] = x[r];
    if (2 * LPC * (r >> 1) >= TEST) continue;
    if (i == j) a = x[r];
    if (i <= j) y[r] = 0.0;
  }
  // row j is held by lane (j / 2) mod LPC of each group
  a = __shfl_sync(0xffffffffu, a, (threadIdx.x & 31 & ~(LPC - 1)) + ((j >> 1) & (LPC - 1)));
  const double sigma = group_sum<LPC>(lane_dot<RP>(y, y));
  double beta, tau, scale;
  hh_scalars(a, sigma, beta, tau, scale);
  if (tau != 0.0) {
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      const int i = tile_row<LPC>(r);
      if (2 * LPC * (r >> 1) >= TEST) {
        x[r] *= scale;
      } else {
        if (i > j) x[r] *= scale;
        if (i == j) x[r] = beta;
      }
    }
  }
  return tau;
}

// Producer and consumers of a step: the warp that makes the next step's
// reflector or pivot arrives when it is in shared memory and goes on with its
// own updates; the others wait there.  Two barriers take turns (a warp cannot
// be a step ahead without all having passed the one before).
static __device__ __forceinline__ void step_arrive(int j) {
  asm volatile("bar.arrive %0, %1;" ::"r"(1 + (j & 1)), "n"(TTB_THREADS) : "memory");
}
static __device__ __forceinline__ void step_wait(int j) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + (j & 1)), "n"(TTB_THREADS) : "memory");
}

// x[at] for a warp-uniform ``at``, by halves (an indexed register array would
// go to local memory).
template <int N, int RP>
static __device__ __forceinline__ double pick_reg(const double (&x)[RP], int at, int base = 0) {
  if constexpr (N == 1) {
    return base < RP ? x[base < RP ? base : 0] : 0.0;
  } else {
    const double lo = pick_reg<N / 2, RP>(x, at, base);
    const double hi = pick_reg<N / 2, RP>(x, at, base + N / 2);
    return (at & (N / 2)) ? hi : lo;
  }
}
__host__ __device__ constexpr int ceil_pow2(int n) {
  int p = 1;
  while (p < n) p *= 2;
  return p;
}

// dst = x[at] for a warp-uniform ``at``: a chain of moves the compiler does
// not turn into an indexed array (which would put x in local memory).
template <int RP, int SL>
static __device__ __forceinline__ void pick_slot(const double (&x)[SL][RP], int at,
                                                 double (&dst)[RP]) {
#pragma unroll
  for (int r = 0; r < RP; ++r) dst[r] = x[0][r];
#pragma unroll
  for (int s = 1; s < SL; ++s)
    if (s == at) {
#pragma unroll
      for (int r = 0; r < RP; ++r) asm volatile("mov.f64 %0, %1;" : "=d"(dst[r]) : "d"(x[s][r]));
    }
}

// x[s] -= t (v . x[s]) v in every slot from ``first`` on.
template <int LPC, int RP, int SL>
static __device__ __forceinline__ void hh_reflect(double (&x)[SL][RP], const double (&v)[RP],
                                                  double t, int first) {
  double w[SL];
#pragma unroll
  for (int s = 0; s < SL; ++s) w[s] = s < first ? 0.0 : lane_dot<RP>(v, x[s]);
#pragma unroll
  for (int s = 0; s < SL; ++s) w[s] = -t * group_sum<LPC>(w[s]);
#pragma unroll
  for (int s = 0; s < SL; ++s) {
    if (s < first) continue;
#pragma unroll
    for (int r = 0; r < RP; ++r) x[s][r] = fma(w[s], v[r], x[s][r]);
  }
}

// x -= t (v . x) v for one slot, v's row pairs read from shared memory (twice:
// held in registers they would crowd out the columns).
template <int RP>
static __device__ __forceinline__ void reflect_slot(double (&x)[RP], const double2* v, double t) {
  double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int r = 0; r < RP; r += 2) {
    const double2 p = v[4 * r];
    a[r & 2] = fma(p.x, x[r], a[r & 2]);
    a[(r & 2) + 1] = fma(p.y, x[r + 1], a[(r & 2) + 1]);
  }
  const double w = -t * group_sum<8>((a[0] + a[2]) + (a[1] + a[3]));
#pragma unroll
  for (int r = 0; r < RP; r += 2) {
    const double2 p = v[4 * r];
    x[r] = fma(w, p.x, x[r]);
    x[r + 1] = fma(w, p.y, x[r + 1]);
  }
}

// Column n of a panel, in one lane group of slot x, becomes reflector n: v
// (zeros above, 1 at row n) to ``vb`` and tau to ``tb``, the other warps are
// let go, then W's column n and tau[n] are written.  Rows below m only.
template <int RP>
static __device__ __forceinline__ void publish_slot(double (&x)[RP], int n, bool mine, int m,
                                                    double2* vb, double* tb, double* wc,
                                                    double* tau) {
  double a = 0.0, c[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int r = 0; r < RP; ++r) {
    const int i = tile_row<8>(r);
    double y = x[r];
    if (16 * (r >> 1) < kPanelMax) {  // rows above the pivot end within the panel's width
      if (i == n) a = y;
      if (i <= n) y = 0.0;
    }
    c[r & 3] = fma(y, y, c[r & 3]);
  }
  a = __shfl_sync(0xffffffffu, a, (threadIdx.x & 24) + ((n >> 1) & 7));
  const double sigma = group_sum<8>((c[0] + c[2]) + (c[1] + c[3]));
  double beta, t, scale;
  hh_scalars(a, sigma, beta, t, scale);
  if (mine) {
#pragma unroll
    for (int r = 0; r < RP; r += 2) {
      const int i = tile_row<8>(r);
      double2 p = make_double2(x[r] * scale, x[r + 1] * scale);
      if (16 * (r >> 1) < kPanelMax) {
        p.x = i > n ? p.x : i == n ? 1.0 : 0.0;
        p.y = i + 1 > n ? p.y : i + 1 == n ? 1.0 : 0.0;
      }
      vb[4 * r] = p;
    }
    if ((threadIdx.x & 7) == 0) *tb = t;
  }
  __syncwarp();
  step_arrive(n);
  if (mine) {
    if ((threadIdx.x & 7) == 0) tau[n] = t;
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      const int i = tile_row<8>(r);
      if (t != 0.0) {
        if (i > n) x[r] *= scale;
        if (i == n) x[r] = beta;
      }
      if (i < m) wc[i] = x[r];
    }
  }
}

// hh_panel (below) for eight lanes a column, m <= 8 RP <= 256: reflectors go
// through shared memory, ready to use, and the warp of the next column
// updates and publishes it before its other columns, so that a column step
// costs the chain of one column.  Neighbouring columns belong to different
// warps (slot s of warp w: columns 32 s + 8 group + w), so that a publisher
// is never more than one barrier ahead; its own late reads of a reflector
// are why three buffers take turns.
template <int RP, int SL>
static __device__ __noinline__ void hh_panel8(double* W, i64 ld, int m, int k, double* tau,
                                              double2 (*vbuf)[128], double* tb) {
  static_assert(RP <= 32 && SL == 2 && TTB_WARPS == 8, "128 row pairs, two slots of 32 columns");
  const int warp = threadIdx.x >> 5, lane8 = threadIdx.x & 7, group = (threadIdx.x & 31) >> 3;
  const int p = m < k ? m : k;
  double x[SL][RP];
#pragma unroll
  for (int s = 0; s < SL; ++s) {
    const int c = 32 * s + 8 * group + warp;
    tile_load<8, RP>(W + c * ld, c < k ? m : 0, x[s]);
  }
  __syncthreads();  // every warp has its columns; the buffers are free
  int at = 2, to = 0;  // the buffers of steps j and j + 1
  for (int j = -1; j < p; ++j) {
    double t = 0.0;
    const double2* v = vbuf[at] + lane8;
    if (j >= 0) {
      if (warp != (j & 7)) step_wait(j);
      t = tb[at];
    }
    const int n = j + 1;
    int done = -1;
    if (n < p && warp == (n & 7)) {
      done = n >> 5;
      const bool mine = group == ((n >> 3) & 3);
      if (done == 0) {
        if (t != 0.0) reflect_slot<RP>(x[0], v, t);
        publish_slot<RP>(x[0], n, mine, m, vbuf[to] + lane8, tb + to, W + n * ld, tau);
      } else {
        if (t != 0.0) reflect_slot<RP>(x[1], v, t);
        publish_slot<RP>(x[1], n, mine, m, vbuf[to] + lane8, tb + to, W + n * ld, tau);
      }
    }
    if (t != 0.0) {
#pragma unroll
      for (int s = 0; s < SL; ++s)
        if (s != done && 32 * s + 24 + warp > j) reflect_slot<RP>(x[s], v, t);
    }
    at = to;
    to = to == 2 ? 0 : to + 1;
  }
#pragma unroll
  for (int s = 0; s < SL; ++s) {
    const int c = 32 * s + 8 * group + warp;
    if (c < p || c >= k) continue;
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      const int i = tile_row<8>(r);
      if (i < m) W[i + c * ld] = x[s][r];
    }
  }
  __syncthreads();
}

// Householder QR of the m x k panel in W, m <= LPC RP, k <= 32 / LPC *
// TTB_WARPS * SL <= 64, in place in LAPACK dgeqr2's layout (see
// cta_householder).  The warp that owns column j + 1 makes the next reflector
// as soon as reflector j has been applied to it, so that a column step has
// one barrier.  Bound by the chain of a column step (about 2000 cycles at 256
// rows: two reductions, a square root and two reciprocals).  256 x 64 with
// its Q took 2.92 ms column by column (a block-wide reduction and three
// barriers per 16 columns of every step) and takes 0.19 ms, its R alone 0.44
// and 0.11 ms (both with hh_panel8 up to 256 rows; this form alone 0.21 and
// 0.14 ms).
template <int LPC, int RP, int SL>
static __device__ __noinline__ void hh_panel(double* W, i64 ld, int m, int k, double* tau) {
  constexpr int G = 32 / LPC;
  const int warp = threadIdx.x >> 5;
  const int p = m < k ? m : k;
  double x[SL][RP];
#pragma unroll
  for (int s = 0; s < SL; ++s) {
    const int c = tile_col<LPC>(s);
    tile_load<LPC, RP>(W + c * ld, c < k ? m : 0, x[s]);
  }
  for (int j = -1; j < p; ++j) {
    __syncthreads();  // reflector j is in W (first: every warp has its columns)
    const double t = j >= 0 ? tau[j] : 0.0;
    // columns past j: those of slots from ``first`` on (a finished column's
    // registers are not used again)
    const int first = SL > 1 && G * (warp + 1) <= j + 1 - G * TTB_WARPS * (SL - 2) ? SL - 1 : 0;
    if (t != 0.0 && G * (TTB_WARPS * (SL - 1) + warp + 1) > j + 1) {
      double v[RP];
      hh_load<LPC, RP>(W, ld, m, j, v);
      hh_reflect<LPC, RP, SL>(x, v, t, first);
    }
    if (j + 1 < p && warp == ((j + 1) / G) % TTB_WARPS) {  // the next reflector
      double col[RP];
      const int s = (j + 1) / (G * TTB_WARPS);
      pick_slot<RP, SL>(x, s, col);
      const double tn = hh_make<LPC, RP>(col, j + 1);
      if (tile_col<LPC>(s) == j + 1) {
        if ((threadIdx.x & (LPC - 1)) == 0) tau[j + 1] = tn;
        double* wc = W + (j + 1) * ld;
#pragma unroll
        for (int r = 0; r < RP; ++r) {
          const int i = tile_row<LPC>(r);
          if (i < m) wc[i] = col[r];
        }
      }
    }
  }
#pragma unroll
  for (int s = 0; s < SL; ++s) {
    const int c = tile_col<LPC>(s);
    if (c < p || c >= k) continue;
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      const int i = tile_row<LPC>(r);
      if (i < m) W[i + c * ld] = x[s][r];
    }
  }
  __syncthreads();
}

// Where the columns of hh_columns start: the matrix X itself, the identity,
// or [top(:, order); 0] with top kt x kt column major (column step ktop).
enum { HH_X = 0, HH_IDENT = 1, HH_TOP = 2 };

// A panel's p <= 64 reflectors in W applied to ncols columns of X (m x
// ncols, any strides), first to last (FWD: H^T) or last to first (Q).  Each
// column stays with its lanes, so no barrier is needed.  From an identity
// start (column c the unit vector c) reflector j leaves the columns below j
// alone.
template <int LPC, int RP, int SL, bool FWD>
static __device__ __noinline__ void hh_columns(const double* W, i64 ld, int m, int p,
                                               const double* tau, Mat X, int ncols, int start,
                                               const double* top, int kt, i64 ktop,
                                               const int* order) {
  constexpr int G = 32 / LPC, STEP = G * TTB_WARPS * SL;
  const int warp = threadIdx.x >> 5;
  for (int g0 = 0; g0 < ncols; g0 += STEP) {
    if (g0 + G * warp >= ncols) break;
    double x[SL][RP];
#pragma unroll
    for (int s = 0; s < SL; ++s) {
      const int c = g0 + tile_col<LPC>(s);
      if (start == HH_TOP) {
        const bool in = c < ncols;
        tile_load<LPC, RP>(in ? top + (order ? order[c] : c) * ktop : top, in ? min(kt, m) : 0, x[s]);
      } else {
#pragma unroll
        for (int r = 0; r < RP; ++r) {
          const int i = tile_row<LPC>(r);
          x[s][r] = 0.0;
          if (start == HH_IDENT) x[s][r] = i == c ? 1.0 : 0.0;
          else if (c < ncols && i < m) x[s][r] = X(i, c);
        }
      }
    }
    const int last = start == HH_IDENT
                         ? min(p - 1, g0 + G * (TTB_WARPS * (SL - 1) + warp + 1) - 1)
                         : p - 1;
    for (int q = 0; q <= last; ++q) {
      const int j = FWD ? q : last - q;
      const double t = tau[j];
      if (t == 0.0) continue;
      double v[RP];
      hh_load<LPC, RP>(W, ld, m, j, v);
      hh_reflect<LPC, RP, SL>(x, v, t, 0);
    }
#pragma unroll
    for (int s = 0; s < SL; ++s) {
      const int c = g0 + tile_col<LPC>(s);
      if (c >= ncols) continue;
#pragma unroll
      for (int r = 0; r < RP; ++r) {
        const int i = tile_row<LPC>(r);
        if (i < m) X(i, c) = x[s][r];
      }
    }
  }
}

// Most rows the register tiles take.
constexpr int kHHRows = 2048;

// The tile for a panel of ``rows`` rows: eight lanes a column up to 256 rows
// (64 columns in a block), 16 up to 512 (32), the whole warp beyond (16 up to
// 1024 rows, then 8): 64 doubles of a thread's registers at most.
#define TTB_HH_TILE(rows, CALL)        \
  if ((rows) <= 32) { CALL(8, 4, 2); } \
  else if ((rows) <= 64) { CALL(8, 8, 2); }    \
  else if ((rows) <= 128) { CALL(8, 16, 2); }  \
  else if ((rows) <= 256) { CALL(8, 32, 2); }  \
  else if ((rows) <= 512) { CALL(16, 32, 2); } \
  else if ((rows) <= 1024) { CALL(32, 32, 2); } \
  else { CALL(32, 64, 1); }

static __device__ __forceinline__ int hh_width(int m) {
  return m <= 256 ? 64 : m <= 512 ? 32 : m <= 1024 ? 16 : 8;
}

// One panel's reflectors applied to columns (see hh_columns).
template <bool FWD>
static __device__ __noinline__ void cta_hh_panel_apply(const double* W, i64 ld, int m, int p,
                                                       const double* tau, Mat X, int ncols,
                                                       int start, const double* top, int kt,
                                                       i64 ktop, const int* order) {
#define TTB_HH_APPLY(L, R, S) \
  hh_columns<L, R, S, FWD>(W, ld, m, p, tau, X, ncols, start, top, kt, ktop, order)
  if (ncols <= 32 && m > 32 && m <= 256) {  // one slot holds them all
    if (m <= 64) TTB_HH_APPLY(8, 8, 1);
    else if (m <= 128) TTB_HH_APPLY(8, 16, 1);
    else TTB_HH_APPLY(8, 32, 1);
  } else {
    TTB_HH_TILE(m, TTB_HH_APPLY)
  }
#undef TTB_HH_APPLY
  __syncthreads();
}

// The p reflectors in W applied to X's ncols columns, last to first: Q X,
// Q [top(:, order); 0] or, from the identity, Q itself.  Up to kPanelMax
// reflectors at a time; only the last group can start from anything but X.
static __device__ void cta_hh_apply(const double* W, i64 ld, int m, int p, const double* tau,
                                    Mat X, int ncols, int start, const double* top = nullptr,
                                    int kt = 0, i64 ktop = 0, const int* order = nullptr) {
  if (p > kPanelMax && start != HH_X) {
    for (int e = threadIdx.x; e < m * ncols; e += TTB_THREADS) {
      const int i = e / ncols, c = e % ncols;
      X(i, c) = start == HH_IDENT ? (i == c ? 1.0 : 0.0)
                                  : (i < kt ? top[i + (order ? order[c] : c) * ktop] : 0.0);
    }
    __syncthreads();
  }
  for (int j0 = ((p - 1) / kPanelMax) * kPanelMax; j0 >= 0; j0 -= kPanelMax) {
    const bool whole = p <= kPanelMax;
    // from the identity, columns below j0 are still unit vectors there
    const int c0 = start == HH_IDENT ? j0 : 0;
    cta_hh_panel_apply<false>(W + j0 + j0 * ld, ld, m - j0, min(kPanelMax, p - j0), tau + j0,
                              Mat{X.p + j0 * X.rs + c0 * X.cs, X.rs, X.cs}, ncols - c0,
                              whole ? start : HH_X, top, kt, ktop, order);
  }
}

// cta_householder for m <= kHHRows: column panels as wide as the registers
// allow, each panel's reflectors applied to the columns right of it.
static __device__ __noinline__ void cta_hh(double* W, i64 ld, int m, int k, double* tau) {
  const int p = m < k ? m : k;
  const int width = hh_width(m);
  __shared__ double2 vb[3][128];  // hh_panel8's reflectors (here: one copy for its tiles)
  __shared__ double tb[3];
  for (int j0 = 0; j0 < p; j0 += width) {
    const int cols = min(width, k - j0), rows = m - j0;
    double* P = W + j0 + j0 * ld;
    if (rows <= 32) hh_panel8<4, 2>(P, ld, rows, cols, tau + j0, vb, tb);
    else if (rows <= 64) hh_panel8<8, 2>(P, ld, rows, cols, tau + j0, vb, tb);
    else if (rows <= 128) hh_panel8<16, 2>(P, ld, rows, cols, tau + j0, vb, tb);
    else if (rows <= 256) hh_panel8<32, 2>(P, ld, rows, cols, tau + j0, vb, tb);
    else if (rows <= 512) hh_panel<16, 32, 2>(P, ld, rows, cols, tau + j0);
    else if (rows <= 1024) hh_panel<32, 32, 2>(P, ld, rows, cols, tau + j0);
    else hh_panel<32, 64, 1>(P, ld, rows, cols, tau + j0);
    const int rest = k - j0 - cols;
    if (rest > 0)
      cta_hh_panel_apply<true>(P, ld, rows, min(cols, rows), tau + j0,
                               Mat{P + cols * ld, 1, ld}, rest, HH_X, nullptr, 0, 0, nullptr);
  }
}

// Rows up to which the register tiles alone factor a matrix in global memory
// (four columns a warp and step); taller ones take LNB-column panels with
// the trailing updates as GEMMs.
constexpr int kHHTall = 512;

// Whether the register tiles take a matrix: not beyond their rows, and not
// where a few columns leave most of a tile empty.  With Q, in tiles and column by
// column: 512 x 2 22 and 11 us, 256 x 4 21 and 17, 256 x 8 31 and 47; of four
// columns the shortest and the tallest stay in tiles (64 x 4 10.5 and 11.4,
// 1024 x 4 30 and 36).
constexpr int kNarrow = 4, kNarrowShort = 128, kNarrowTall = 640;
static __device__ __forceinline__ bool hh_tiled(int m, int k) {
  if (m > kHHRows || k < kNarrow) return false;
  return k > kNarrow || m <= kNarrowShort || m > kNarrowTall;
}

// A panel's reflectors: in registers, or column by column.
template <bool TILED>
static __device__ __forceinline__ void cta_hh_any(double* W, int m, int k, i64 ld, double* tau,
                                                  double* red) {
  if constexpr (TILED) {
    if (hh_tiled(m, k)) {
      cta_hh(W, ld, m, k, tau);
      return;
    }
  }
  cta_householder(W, m, k, ld, tau, red);
}

// Economic QR of the m x k matrix ``A`` (any strides): Q (m x p) and R
// (p x k), p = min(m, k).  ``W`` is a column-major work area (unit row step,
// column step ldw >= m; an odd one spreads a row over the shared-memory
// banks), ``tau`` p doubles; both may be shared or global memory.  Q and R
// may be NULL to skip them.
template <bool TILED>
__device__ __noinline__ void cta_qr(CMat A, int m, int k, double* W, i64 ldw, double* tau, Mat Q,
                                    Mat R, double* red) {
  const int p = m < k ? m : k;
  cta_load(A, W, ldw, m, k);
  __syncthreads();
  const bool tiles = TILED && hh_tiled(m, k);
  cta_hh_any<TILED>(W, m, k, ldw, tau, red);
  if (R.p) {
    for (int e = threadIdx.x; e < p * k; e += TTB_THREADS) {
      int i = e / k, j = e % k;
      R(i, j) = (i <= j) ? W[i + j * ldw] : 0.0;
    }
  }
  if (Q.p) {
    if (tiles) {
      if constexpr (TILED) cta_hh_apply(W, ldw, m, p, tau, Q, p, HH_IDENT);
    } else {
      for (int e = threadIdx.x; e < m * p; e += TTB_THREADS) {
        int i = e % m, j = e / m;
        Q(i, j) = (i == j) ? 1.0 : 0.0;
      }
      __syncthreads();
      cta_apply_q(W, m, p, ldw, tau, Q, p);
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// one-sided Jacobi SVD
// ---------------------------------------------------------------------------

// Hestenes one-sided Jacobi on the columns of the k x k matrix B (column
// major, leading dimension ldb): finds an orthogonal J with B J having
// orthogonal columns.  On return B holds B J and V (column major, ldv; may be
// NULL) V J.
// Pairs are visited in round-robin tournament order
// (k/2 disjoint pairs per round, one warp per pair).  A pair is rotated when
// |b_p . b_q| > tol sqrt(|b_p|^2 |b_q|^2); sweeps stop when one sweep
// rotates nothing, or after ``max_sweeps``.  Returns the sweeps used, or -1
// when the cap was hit.
static __device__ int cta_jacobi(double* B, int k, i64 ldb, double* V, i64 ldv, int max_sweeps,
                          double tol, int* flag) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (k < 2) {
    __syncthreads();
    return 0;
  }
  const int kk = (k + 1) & ~1;  // players, one dummy when k is odd
  const int half = kk / 2;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x == 0) *flag = 0;
    __syncthreads();
    int rotated = 0;
    for (int round = 0; round < kk - 1; ++round) {
      for (int pr = wid; pr < half; pr += TTB_WARPS) {
        int pa = (pr == 0) ? 0 : ((pr - 1 + round) % (kk - 1)) + 1;
        int pos = kk - 1 - pr;
        int pb = ((pos - 1 + round) % (kk - 1)) + 1;
        int p = pa < pb ? pa : pb, q = pa < pb ? pb : pa;
        if (q >= k) continue;  // paired with the dummy player
        double* bp = B + p * ldb;
        double* bq = B + q * ldb;
        double al = 0.0, be = 0.0, ga = 0.0;
        for (int i = lane; i < k; i += 32) {
          double x = bp[i], y = bq[i];
          al = fma(x, x, al);
          be = fma(y, y, be);
          ga = fma(x, y, ga);
        }
        al = warp_sum(al);
        be = warp_sum(be);
        ga = warp_sum(ga);
        if (ga != 0.0 && fabs(ga) > tol * sqrt(al) * sqrt(be)) {
          double zeta = (be - al) / (2.0 * ga);
          double t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
          double c = 1.0 / sqrt(1.0 + t * t);
          double s = c * t;
          for (int i = lane; i < k; i += 32) {
            double x = bp[i], y = bq[i];
            bp[i] = c * x - s * y;
            bq[i] = s * x + c * y;
          }
          double* vp = V + p * ldv;
          double* vq = V + q * ldv;
          for (int i = lane; V && i < k; i += 32) {
            double x = vp[i], y = vq[i];
            vp[i] = c * x - s * y;
            vq[i] = s * x + c * y;
          }
          rotated = 1;
        }
      }
      __syncthreads();
    }
    if (rotated) *flag = 1;  // benign race: every writer stores 1
    __syncthreads();
    int any = *flag;
    __syncthreads();
    if (!any) return sweep + 1;
  }
  return -1;
}

// Column-pivoted Householder QR of the upper-triangular k x k matrix R
// (column major, column step ld), k <= 8 RP and 32 SL: R P = Q R1, in place
// in LAPACK dgeqr2's layout; perm[j] is the column of R that came j-th, nrm
// (k) work.  Each step takes the remaining column of largest norm below the
// pivot row, the norms recomputed from the updated columns.
template <int RP, int SL>
static __device__ __noinline__ void hh_pivot(double* R, int k, i64 ld, int* perm, double* nrm,
                                             double* tau) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double x[SL][RP];
  unsigned done = 0;  // the slots whose column (this lane group's) is taken
#pragma unroll
  for (int s = 0; s < SL; ++s) {
    const int c = tile_col<8>(s);
    tile_load<8, RP>(R + c * ld, c < k ? k : 0, x[s]);
    if (c >= k) done |= 1u << s;
  }
  for (int j = -1; j < k; ++j) {
    if (j >= 0) {
      __syncthreads();  // the norms of this step
      // every warp finds the same pivot: the lowest column on ties, a NaN
      // before any number (a taken column, at -1, must never win)
      double best = -1.0;
      int at = -1;
#pragma unroll
      for (int s = 0; s < SL; ++s) {
        const int c = lane + 32 * s;
        double v = c < k ? nrm[c] : -1.0;
        if (v != v) v = INFINITY;
        if (c < k && (at < 0 || v > best)) {
          best = v;
          at = c;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double b2 = __shfl_xor_sync(0xffffffffu, best, o);
        const int a2 = __shfl_xor_sync(0xffffffffu, at, o);
        if (a2 >= 0 && (at < 0 || b2 > best || (b2 == best && a2 < at))) {
          best = b2;
          at = a2;
        }
      }
      at = __shfl_sync(0xffffffffu, at, 0);
      __syncthreads();  // every warp has read the norms
      if (warp == (at >> 2) % TTB_WARPS) {
        double col[RP];
        const int s = at >> 5;
        pick_slot<RP, SL>(x, s, col);
        const double t = hh_make<8, RP, 8 * RP>(col, j);
        if (tile_col<8>(s) == at) {
          done |= 1u << s;
          if ((lane & 7) == 0) {
            tau[j] = t;
            perm[j] = at;
            nrm[at] = -1.0;
          }
#pragma unroll
          for (int r = 0; r < RP; ++r) {
            const int i = tile_row<8>(r);
            if (i < k) R[i + j * ld] = col[r];
          }
        }
      }
      __syncthreads();  // reflector j is in R
      const double t = tau[j];
      if (t != 0.0) {
        double v[RP];
        hh_load<8, RP, 8 * RP>(R, ld, k, j, v);
        hh_reflect<8, RP, SL>(x, v, t, 0);
      }
    } else {
      __syncthreads();  // every warp has its columns of R
    }
    // squared norms of the remaining columns below row j
#pragma unroll
    for (int s = 0; s < SL; ++s) {
      double y[RP];
#pragma unroll
      for (int r = 0; r < RP; ++r) y[r] = tile_row<8>(r) > j ? x[s][r] : 0.0;
      const double n2 = group_sum<8>(lane_dot<RP>(y, y));
      if ((lane & 7) == 0 && !(done & (1u << s))) nrm[tile_col<8>(s)] = n2;
    }
  }
  __syncthreads();
}

// Cosine and sine of the Jacobi rotation of two columns with squared norms
// al and be and inner product ga, the rotation of smaller angle that makes
// them orthogonal, for squared norms whose products leave the exponent range.
static __device__ __noinline__ bool jacobi_angle_wide(double al, double be, double ga, double tol,
                                                      double& c, double& s) {
  if (!(fabs(ga) > tol * sqrt(al) * sqrt(be))) return false;
  const double zeta = (be - al) / (2.0 * ga);
  const double t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
  c = 1.0 / sqrt(1.0 + t * t);
  s = c * t;
  return true;
}

// 1e-100 < a < 1e100, by its exponent.
static __device__ __forceinline__ bool mid_range(double a) {
  return (unsigned)(__double2hiint(a) - 0x2b400000) < 0x54b00000u - 0x2b400000u;
}

// The same in the ordinary range; false (c = 1, s = 0) when
// |ga| <= tol sqrt(al be).  With d = be - al and h = hypot(d, 2 ga),
// c^2 = (1 + |d| / h) / 2 and |s| = |ga| / (h c): two reciprocal square roots
// in all, then one step towards c^2 + s^2 = 1.
static __device__ __forceinline__ bool jacobi_angle(double al, double be, double ga, double tol,
                                                    double tol2, double& c, double& s) {
  c = 1.0;
  s = 0.0;
  if (ga == 0.0) return false;
  if (!mid_range(al) || !mid_range(be)) return jacobi_angle_wide(al, be, ga, tol, c, s);
  const double g2 = ga * ga, d = be - al;
  if (g2 <= tol2 * (al * be)) return false;
  const double rh = rsqrt(fma(d, d, 4.0 * g2));
  const double c2 = fma(0.5 * fabs(d), rh, 0.5);
  const double ic = rsqrt(c2);
  c = c2 * ic;
  s = (d >= 0.0 ? ga : -ga) * rh * ic;
  const double e = 0.5 * fma(-s, s, fma(-c, c, 1.0));
  c = fma(c, e, c);
  s = fma(s, e, s);
  return true;
}

// Two column slots of a warp, x and y: G = 32 / LPC pairs, one per lane group.
template <int LPC, int RP, bool L2>
struct Pairs {
  static constexpr int G = 32 / LPC;
  double x[RP], y[RP];
  double nx, ny;  // their squared norms

  static __device__ __forceinline__ int group() { return (threadIdx.x & 31) / LPC; }

  __device__ __forceinline__ void norms() {
    nx = group_sum<LPC>(lane_dot<RP>(x, x));
    ny = group_sum<LPC>(lane_dot<RP>(y, y));
  }

  // x <- c x - s y, y <- s x + c y
  __device__ __forceinline__ void rotate(double c, double s) {
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      const double a = x[r], b = y[r];
      x[r] = c * a - s * b;
      y[r] = s * a + c * b;
    }
  }

  // The next pairing.  all: the circle method on the 2 G columns (the first x
  // fixed, the others moved round one place: 2 G - 1 steps meet all pairs);
  // else the y columns move round the groups (G steps meet the pairs
  // across).  Either way the last step returns every column to its place.
  static __device__ __forceinline__ void round_table(double& u, double& v) {
    const int lane = threadIdx.x & 31, g = group();
    const double up = __shfl_sync(0xffffffffu, g == 0 ? v : u, (lane + 32 - LPC) & 31);
    const double down = __shfl_sync(0xffffffffu, v, (lane + LPC) & 31);
    v = g == G - 1 ? u : down;
    if (g != 0) u = up;
  }
  __device__ __forceinline__ void next(bool all, bool with_norms) {
    if (all) {
#pragma unroll
      for (int r = 0; r < RP; ++r) round_table(x[r], y[r]);
      if (with_norms) round_table(nx, ny);
    } else {
      const int from = ((threadIdx.x & 31) + LPC) & 31;
#pragma unroll
      for (int r = 0; r < RP; ++r) y[r] = __shfl_sync(0xffffffffu, y[r], from);
      if (with_norms) ny = __shfl_sync(0xffffffffu, ny, from);
    }
  }

  // Columns ca + group and cb + group of the k x k matrix M (column step
  // ld), zeros beyond it; and back.
  __device__ __forceinline__ void load(const double* M, i64 ld, int k, int ca, int cb) {
    const int a = ca + group(), b = cb + group();
    tile_load<LPC, RP, L2>(M + a * ld, a < k ? k : 0, x);
    tile_load<LPC, RP, L2>(M + b * ld, b < k ? k : 0, y);
  }
  __device__ __forceinline__ void store(double* M, i64 ld, int k, int ca, int cb) const {
    const int a = ca + group(), b = cb + group();
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      const int i = tile_row<LPC>(r);
      if (i >= k) continue;
      if constexpr (L2) {
        if (a < k) __stcg(M + i + a * ld, x[r]);
        if (b < k) __stcg(M + i + b * ld, y[r]);
      } else {
        if (a < k) M[i + a * ld] = x[r];
        if (b < k) M[i + b * ld] = y[r];
      }
    }
  }
};

// One round of a Jacobi sweep over the block pairs first, first + step, ...:
// true if any of this warp's pairs was rotated.  See jacobi_blocks.
template <int LPC, int RP, bool VACC, bool L2>
static __device__ __forceinline__ bool jacobi_round(double* B, int k, i64 ld, double* V,
                                                    double tol, int nb, int round, int first,
                                                    int step) {
  constexpr bool kRide = VACC && RP <= 16, kReplay = VACC && !kRide;
  constexpr int G = 32 / LPC;
  const double tol2 = tol * tol;
  const bool all = round == 0;
  const int steps = all ? 2 * G - 1 : G;
  bool rotated = false;
  for (int pr = first; pr < nb / 2; pr += step) {
    const int pa = (pr == 0) ? 0 : ((pr - 1 + round) % (nb - 1)) + 1;
    const int pb = ((nb - 2 - pr + round) % (nb - 1)) + 1;
    const int ca = G * min(pa, pb), cb = G * max(pa, pb);
    Pairs<LPC, RP, L2> p;
    Pairs<LPC, kRide ? RP : 2, L2> q;
    double cs[kReplay ? 2 * G - 1 : 1], sn[kReplay ? 2 * G - 1 : 1];
    p.load(B, ld, k, ca, cb);
    if constexpr (kRide) q.load(V, ld, k, ca, cb);
    p.norms();
    bool turned = false;
#pragma unroll 1
    for (int t = 0; t < steps; ++t) {
      const double ga = group_sum<LPC>(lane_dot<RP>(p.x, p.y));
      double c, s;
      const bool rot = jacobi_angle(p.nx, p.ny, ga, tol, tol2, c, s);
      if (__any_sync(0xffffffffu, rot)) {
        turned = true;
        const double tg = ga * s * __drcp_rn(c);
        p.nx -= tg;
        p.ny += tg;
        p.rotate(c, s);
        if constexpr (kRide) q.rotate(c, s);
      }
      if constexpr (kReplay) {
        cs[t] = c;
        sn[t] = s;
      }
      p.next(all, true);
      if constexpr (kRide) q.next(all, false);
    }
    if (!turned) continue;
    rotated = true;
    p.store(B, ld, k, ca, cb);
    if constexpr (kRide) q.store(V, ld, k, ca, cb);
    if constexpr (kReplay) {
      p.load(V, ld, k, ca, cb);
#pragma unroll 1
      for (int t = 0; t < steps; ++t) {
        p.rotate(cs[t], sn[t]);
        p.next(all, false);
      }
      p.store(V, ld, k, ca, cb);
    }
  }
  return rotated;
}

// Hestenes' one-sided Jacobi on the columns of the k x k matrix B (column
// step ld; see cta_jacobi, which it replaces up to k = kPivotMax) and, with VACC,
// V (k x k, the same step) multiplied by the same rotations.  Columns go in
// blocks of four; a warp loads a pair of blocks into registers, eight lanes
// to a column, and rotates all their column pairs, four disjoint pairs at a
// time: each pair belongs to eight lanes, which reduce its inner product in
// three shuffle levels and compute its angle; squared norms are summed when
// the blocks are loaded and follow the rotations until they are stored (a
// sweep without rotations, which ends the iteration, has only summed ones).
// Between steps the second columns move on to the next lanes.  Blocks meet in
// round-robin order, one block barrier per meeting: a sweep of 64 columns has
// 15 barriers and moves the matrices through shared memory 15 times, where
// pairing single columns took 63.  What bounds a step is its chain (sums,
// two reciprocal square roots, rotation: about 900 cycles) and, with V, the
// issue of FP64 and shuffle instructions.  V rides along in registers up to
// RP = 16 and is rotated afterwards beyond.
template <int RP, bool VACC>
static __device__ __noinline__ int jacobi_blocks(double* B, int k, i64 ld, double* V,
                                                 int max_sweeps, double tol, int* flag) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = ((k + 7) >> 3) << 1;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    __syncthreads();
    if (threadIdx.x == 0) *flag = 0;
    __syncthreads();
    bool rotated = false;
    for (int round = 0; round < nb - 1; ++round) {
      rotated |= jacobi_round<8, RP, VACC, false>(B, k, ld, V, tol, nb, round, warp, TTB_WARPS);
      __syncthreads();
    }
    if (rotated && lane == 0) *flag = 1;  // benign race: every writer stores 1
    __syncthreads();
    if (!*flag) return sweep + 1;
  }
  return -1;
}

// The same iteration by a cluster of blocks on matrices in global memory: the
// block pairs of a round are dealt out to the cluster's warps, which meet at
// a cluster barrier after each round and read and write the columns past
// their first-level caches.  flags: three ints in global memory, the first
// zero.  A round of 192 columns is 24 pairs: one per warp of three blocks,
// where one block had taken them in three turns.  192 x 192 (left factor)
// took 12.2 ms in one block and takes 4.0 ms, 250 x 250 24.2 and 7.6 ms; up
// to 96 columns, which shared memory holds, one block is as fast.
template <int LPC, int RP, bool VACC>
static __device__ __noinline__ int jacobi_cluster(double* B, int k, i64 ld, double* V,
                                                  int max_sweeps, double tol, int* flags) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  constexpr int G = 32 / LPC;
  const int lane = threadIdx.x & 31;
  const int first = (int)cl.block_rank() * TTB_WARPS + (threadIdx.x >> 5);
  const int step = (int)cl.num_blocks() * TTB_WARPS;
  const int nb = 2 * ((k + 2 * G - 1) / (2 * G));
  auto meet = [&]() {
    __threadfence();
    cl.sync();
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
  };
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    // the flag of the next sweep is cleared before this one's last barrier
    if (cl.block_rank() == 0 && threadIdx.x == 0) __stcg(flags + (sweep + 1) % 3, 0);
    bool rotated = false;
    for (int round = 0; round < nb - 1; ++round) {
      rotated |= jacobi_round<LPC, RP, VACC, true>(B, k, ld, V, tol, nb, round, first, step);
      if (round == nb - 2 && rotated && lane == 0) __stcg(flags + sweep % 3, 1);
      meet();
    }
    if (!__ldcg(flags + sweep % 3)) return sweep + 1;
  }
  return -1;
}

template <bool VACC>
static __device__ __forceinline__ int cluster_iterate(double* B, int k, i64 ld, double* V,
                                                      double tol, int* flags) {
  if (k <= 128) return jacobi_cluster<8, 16, VACC>(B, k, ld, V, 60, tol, flags);
  if (k <= 192) return jacobi_cluster<8, 24, VACC>(B, k, ld, V, 60, tol, flags);
  if (k <= 256) return jacobi_cluster<8, 32, VACC>(B, k, ld, V, 60, tol, flags);
  if (k <= 384) return jacobi_cluster<16, 24, VACC>(B, k, ld, V, 60, tol, flags);
  return jacobi_cluster<16, 32, VACC>(B, k, ld, V, 60, tol, flags);
}

// Orthonormal rows for the singular values that are exactly zero (their rows
// of M are not defined by the iteration): each is the unit vector furthest
// from the rows so far, orthogonalised against them twice.  Singular value
// number order[r], the last ones the zeros, belongs to row order[r] of M
// (``rows`` given) or row r.
static __device__ __noinline__ void cta_complete_rows(int k, const double* sv, const int* rows,
                                                      const int* order, Mat M, double* red) {
  __shared__ int redi[TTB_WARPS];
  const int* ord = rows ? rows : order;
  auto row = [&](int r) { return rows ? rows[r] : r; };
  for (int r = 0; r < k; ++r) {
    if (sv[ord[r]] != 0.0) continue;
    const int rr = row(r);
    double best = -1.0;
    int at = -1;
    for (int i = threadIdx.x; i < k; i += TTB_THREADS) {
      double s = 0.0;
      for (int q = 0; q < r; ++q) s = fma(M(row(q), i), M(row(q), i), s);
      const double left = fmax(2.0 - s, 0.0);
      if (left > best) { best = left; at = i; }
    }
    at = max(block_argmax_abs(best, at, red, redi), 0);
    for (int i = threadIdx.x; i < k; i += TTB_THREADS) M(rr, i) = i == at ? 1.0 : 0.0;
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass)
      for (int q = 0; q < r; ++q) {
        double s = 0.0;
        for (int i = threadIdx.x; i < k; i += TTB_THREADS) s = fma(M(row(q), i), M(rr, i), s);
        s = block_sum(s, red);
        for (int i = threadIdx.x; i < k; i += TTB_THREADS) M(rr, i) -= s * M(row(q), i);
      }
    double n2 = 0.0;
    for (int i = threadIdx.x; i < k; i += TTB_THREADS) n2 = fma(M(rr, i), M(rr, i), n2);
    const double inv = 1.0 / sqrt(block_sum(n2, red));
    for (int i = threadIdx.x; i < k; i += TTB_THREADS) M(rr, i) *= inv;
    __syncthreads();
  }
}

// Largest k of the register-blocked Jacobi iteration in one block and of the
// pivoted preconditioner in registers (beyond, a cluster iterates up to
// kClusterMax, then the plain form).
constexpr int kPivotMax = 128;

template <bool VACC>
static __device__ int cta_jacobi_blocks(double* B, int k, i64 ld, double* V, int max_sweeps,
                                        double tol, int* flag) {
  if (k <= 16) return jacobi_blocks<2, VACC>(B, k, ld, V, max_sweeps, tol, flag);
  if (k <= 32) return jacobi_blocks<4, VACC>(B, k, ld, V, max_sweeps, tol, flag);
  if (k <= 64) return jacobi_blocks<8, VACC>(B, k, ld, V, max_sweeps, tol, flag);
  if (k <= 96) return jacobi_blocks<12, VACC>(B, k, ld, V, max_sweeps, tol, flag);
  return jacobi_blocks<16, VACC>(B, k, ld, V, max_sweeps, tol, flag);  // k <= kPivotMax
}

// M's upper triangle becomes its transpose in the lower one, the upper
// zeros (k x k, column step ld); with ``to`` another matrix instead of M.
static __device__ void cta_transpose_upper(const double* M, double* to, int k, i64 ld) {
  for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) {
    const int i = e / k, j = e % k;  // i <= j is done by one thread for (j, i) too
    if (i > j) continue;
    const double v = M[i + j * ld];
    to[j + i * ld] = v;
    if (i != j) to[i + j * ld] = 0.0;
  }
  __syncthreads();
}

// Column norms of the k x k matrix B (column step ld) into sv and their
// descending order; *flag tells whether one is zero.
static __device__ void cta_sort_columns(const double* B, int k, i64 ld, double* sv, int* order,
                                        int* flag) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = warp; j < k; j += TTB_WARPS) {
    double s = 0.0;
    for (int i = lane; i < k; i += 32) s = fma(B[i + j * ld], B[i + j * ld], s);
    s = warp_sum(s);
    if (lane == 0) {
      sv[j] = sqrt(s);
      order[j] = j;
    }
  }
  if (threadIdx.x == 0) *flag = 0;
  __syncthreads();
  for (int j = threadIdx.x; j < k; j += TTB_THREADS) {
    const double sj = sv[j];
    int rank = 0;
    for (int i = 0; i < k; ++i) {
      const double si = sv[i];
      rank += (si > sj) || (si == sj && i < j);
    }
    if (sj == sj) order[rank] = j;  // a NaN keeps the unsorted order
    if (sj == 0.0) *flag = 1;       // benign race: every writer stores 1
  }
  __syncthreads();
}

// Column-pivoted QR of the upper-triangular k x k matrix in *F (column step
// ld, zeros below), in place; ``other`` is a work area of the same size.
// Beyond the registers the columns are sorted by norm once and factored
// plainly: the factors are then in ``other``, and the two pointers change
// places.
static __device__ void cta_pivoted(double*& F, double*& other, int k, i64 ld, int* perm,
                                   double* sv, double* tau2, double* red) {
  if (k <= 32) {
    hh_pivot<4, 1>(F, k, ld, perm, sv, tau2);
  } else if (k <= 64) {
    hh_pivot<8, 2>(F, k, ld, perm, sv, tau2);
  } else if (k <= 96) {
    hh_pivot<12, 3>(F, k, ld, perm, sv, tau2);
  } else if (k <= kPivotMax) {
    hh_pivot<16, 4>(F, k, ld, perm, sv, tau2);
  } else {
    for (int j = threadIdx.x; j < k; j += TTB_THREADS) {
      double s = 0.0;
      for (int i = 0; i <= j; ++i) s = fma(F[i + j * ld], F[i + j * ld], s);
      sv[j] = s;
      perm[j] = j;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < k; j += TTB_THREADS) {
      int rank = 0;
      for (int i = 0; i < k; ++i) rank += (sv[i] > sv[j]) || (sv[i] == sv[j] && i < j);
      if (sv[j] == sv[j]) perm[rank] = j;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < k * k; e += TTB_THREADS)
      other[e % k + (e / k) * ld] = F[e % k + perm[e / k] * ld];
    __syncthreads();
    if (k <= kHHRows)
      cta_hh(other, ld, k, k, tau2);
    else
      cta_householder(other, k, k, ld, tau2, red);
    double* t = F;
    F = other;
    other = t;
  }
}

// X <- Q X for the k x k reflectors in F, X k x k (column step ld) or a view.
static __device__ void cta_apply_square(const double* F, int k, i64 ld, const double* tau, Mat X,
                                        int start) {
  if (k <= kHHRows) {
    cta_hh_apply(F, ld, k, k, tau, X, k, start);
    return;
  }
  if (start == HH_IDENT)
    for (int e = threadIdx.x; e < k * k; e += TTB_THREADS)
      X(e % k, e / k) = e % k == e / k ? 1.0 : 0.0;
  __syncthreads();
  cta_apply_q(F, k, k, ld, tau, X, k);
}

// SVD of the upper-triangular k x k matrix R in Bsq (column major, column
// step svd_step(k), zeros below the diagonal).  ``order`` has room for 2 k
// ints (the second half keeps the pivot order), tau2 k doubles; S gets the
// singular values, descending.
//
// Jacobi's sweeps depend on how near to orthogonal the columns start.  R's
// own columns are far from it where the spectrum is steep, as it is in
// rounding; those of L = R1^T, from the column-pivoted QR R P = Q2 R1, are
// much nearer, and those of R2^T, from L = Q3 R2, nearer still (Drmac and
// Veselic, "New fast and accurate Jacobi SVD algorithm", 2008): the 64-column
// matrices of rounding a sum of rank-32 trains to 1e-6 take 15, 8 and 7
// sweeps, a sampled field's 24, 9 and 7.  A 256 x 64 SVD took 4.3 ms with the
// plain iteration and takes 0.69 ms, its left factor alone 0.63 and its right
// one 0.47 ms.
//
// SQ_BOTH:  with L J = W S (J the rotations), R = (Q2 J) S (P W)^T: Vh is
//           written and the left factor left in V (Us: scratch, the top of
//           the caller's U).
// SQ_LEFT:  with R2^T J = W S, R = (Q2 W) S (...): the left factor in V; no
//           rotations are accumulated.
// SQ_RIGHT: with L J = W S, the right factor (P W)^T is written to Vh.
//
// In three parts, so that the iteration can be a cluster's: the matrix X it
// works on and the factors F (of Q2, or the accumulated rotations) are Bsq
// and V in the order square_roles gives.  At the end the left factor's column
// of singular value r is column order[r] of square_left.
enum { SQ_BOTH = 0, SQ_LEFT = 1, SQ_RIGHT = 2 };
static __device__ __forceinline__ void square_roles(int want, int k, double* Bsq, double* V,
                                                    double*& F, double*& X) {
  const bool first = (k <= kPivotMax) != (want == SQ_BOTH);
  F = first ? Bsq : V;
  X = first ? V : Bsq;
}
static __device__ __forceinline__ double square_tol(int k) {
  return 2.0 * sqrt((double)k) * 2.220446049250313e-16;
}

static __device__ __noinline__ void square_prepare(int want, int k, double* Bsq, double* V,
                                                   double* sv, int* order, double* tau2, Mat Us,
                                                   double* red) {
  const i64 ld = svd_step(k);
  double *F = Bsq, *X = V;
  cta_pivoted(F, X, k, ld, order + k, sv, tau2, red);
  if (want == SQ_BOTH) {
    cta_apply_square(F, k, ld, tau2, Us, HH_IDENT);  // Q2, explicit
    cta_transpose_upper(F, F, k, ld);                // L takes the factors' place
    for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) X[e % k + (e / k) * ld] = Us(e % k, e / k);
    __syncthreads();
    return;
  }
  cta_transpose_upper(F, X, k, ld);
  if (want != SQ_LEFT) return;
  // (sv is free until the columns are sorted: the second QR's scalars)
  if (k <= kHHRows)
    cta_hh(X, ld, k, k, sv);
  else
    cta_householder(X, k, k, ld, sv, red);
  cta_transpose_upper(X, X, k, ld);
}

static __device__ __noinline__ int square_iterate(int want, int k, double* Bsq, double* V,
                                                  int* flag) {
  const i64 ld = svd_step(k);
  double *F, *X;
  square_roles(want, k, Bsq, V, F, X);
  const double tol = square_tol(k);
  if (k > kPivotMax) return cta_jacobi(X, k, ld, want == SQ_BOTH ? F : nullptr, ld, 60, tol, flag);
  if (want == SQ_BOTH) return cta_jacobi_blocks<true>(X, k, ld, F, 60, tol, flag);
  return cta_jacobi_blocks<false>(X, k, ld, nullptr, 60, tol, flag);
}

static __device__ __noinline__ void square_finish(int want, int k, double* Bsq, double* V,
                                                  double* sv, int* order, double* tau2, int* flag,
                                                  double* S, Mat Vh, double* red) {
  const i64 ld = svd_step(k);
  const int* perm = order + k;
  double *F, *X;
  square_roles(want, k, Bsq, V, F, X);
  cta_sort_columns(X, k, ld, sv, order, flag);
  for (int r = threadIdx.x; r < k; r += TTB_THREADS) S[r] = sv[order[r]];
  if (want == SQ_LEFT) {
    // W's columns in place, those of zero singular values completed
    for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) {
      const int j = e / k, i = e % k;
      if (sv[j] != 0.0) X[i + j * ld] /= sv[j];
    }
    __syncthreads();
    if (*flag) cta_complete_rows(k, sv, order, order, Mat{X, ld, 1}, red);
    cta_apply_square(F, k, ld, tau2, Mat{X, 1, ld}, HH_X);
    return;
  }
  for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) {
    const int r = e / k, c = e % k, j = order[r];
    Vh(r, perm[c]) = sv[j] == 0.0 ? 0.0 : X[c + j * ld] / sv[j];
  }
  __syncthreads();
  if (*flag) cta_complete_rows(k, sv, nullptr, order, Vh, red);
}

static __device__ __forceinline__ double* square_left(int want, int k, double* Bsq, double* V) {
  double *F, *X;
  square_roles(want, k, Bsq, V, F, X);
  return want == SQ_LEFT ? X : F;
}

// The SVD of an upper-triangular B of up to kSmall columns (column step
// svd_step(k)): one-sided Jacobi on its own columns, B J = U S, without the
// pivoted QRs that pay from there on.  ``want``, ``order``, S and Vh as above;
// the left factor (columns in ``order``) takes B's place.  What the pivoted QR,
// its factors, a second QR and five block-wide steps cost does not depend on k:
// 64 x 1 takes 20 us with them and 9 us so, 64 x 4 42 and 25, 64 x 6 54 and 40,
// 64 x 8 59 and 58.
constexpr int kSmall = 6;
static __device__ __noinline__ int cta_svd_small(int want, int k, double* B, double* V, double* sv,
                                                 int* order, int* flag, double* S, Mat Vh,
                                                 double* red) {
  const i64 ld = svd_step(k);
  const int lane = threadIdx.x & 31;
  double* J = want == SQ_LEFT ? nullptr : V;
  if (J)
    for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) J[e % k + (e / k) * ld] = e % k == e / k;
  const int status = cta_jacobi(B, k, ld, J, ld, 60, square_tol(k), flag);
  // singular values and their order, a lane a column
  if (threadIdx.x < 32) {
    double s = 0.0;
    for (int i = 0; lane < k && i < k; ++i) s = fma(B[i + lane * ld], B[i + lane * ld], s);
    s = sqrt(s);
    int rank = 0;
    for (int i = 0; i < k; ++i) {
      const double si = __shfl_sync(0xffffffffu, s, i);
      rank += (si > s) || (si == s && i < lane);
    }
    if (lane < k) {
      sv[lane] = s;
      order[lane] = lane;
    }
    __syncwarp();
    if (lane < k && s == s) order[rank] = lane;  // a NaN keeps the unsorted order
  }
  __syncthreads();
  const int zero = __syncthreads_or(threadIdx.x < k && sv[threadIdx.x] == 0.0);
  // a NaN anywhere leaves no value or vector defined, as after the pivoted QRs
  if (__syncthreads_or(threadIdx.x < k && sv[threadIdx.x] != sv[threadIdx.x])) {
    if (threadIdx.x < k) S[threadIdx.x] = NAN;
    for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) {
      if (J) Vh(e / k, e % k) = NAN;
      B[e % k + (e / k) * ld] = NAN;
    }
    __syncthreads();
    return status;
  }
  if (threadIdx.x < k) S[threadIdx.x] = sv[order[threadIdx.x]];
  for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) {
    const int i = e % k, j = e / k;
    if (J) Vh(j, i) = J[i + order[j] * ld];
    if (want != SQ_RIGHT && sv[j] != 0.0) B[i + j * ld] /= sv[j];
  }
  __syncthreads();
  if (want != SQ_RIGHT && zero) cta_complete_rows(k, sv, order, order, Mat{B, ld, 1}, red);
  return status;
}

static __device__ __noinline__ int cta_svd_square(int want, int k, double* Bsq, double*& V,
                                                  double* sv, int* order, double* tau2, int* flag,
                                                  Mat Us, double* S, Mat Vh, double* red) {
  if (k <= kSmall) {
    const int status = cta_svd_small(want, k, Bsq, V, sv, order, flag, S, Vh, red);
    V = Bsq;
    return status;
  }
  square_prepare(want, k, Bsq, V, sv, order, tau2, Us, red);
  const int status = square_iterate(want, k, Bsq, V, flag);
  square_finish(want, k, Bsq, V, sv, order, tau2, flag, S, Vh, red);
  V = square_left(want, k, Bsq, V);
  return status;
}

// The SVD of R by the plain iteration on R's own columns (R V = B): S and Vh
// written, B's columns S times the left factor.
static __device__ __noinline__ int cta_svd_plain(int k, double* B, double* V, double* sv,
                                                 int* order, int* flag, double* S, Mat Vh) {
  const i64 ld = k;
  const double tol = 4.0 * k * 2.220446049250313e-16;
  for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) {
    const int i = e % k, j = e / k;
    V[i + j * ld] = (i == j) ? 1.0 : 0.0;
  }
  const int status = cta_jacobi(B, k, ld, V, ld, 60, tol, flag);
  for (int j = threadIdx.x; j < k; j += TTB_THREADS) {
    double s = 0.0;
    for (int i = 0; i < k; ++i) s = fma(B[i + j * ld], B[i + j * ld], s);
    sv[j] = sqrt(s);
    order[j] = j;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < k; j += TTB_THREADS) {
    const double sj = sv[j];
    int rank = 0;
    for (int i = 0; i < k; ++i) {
      const double si = sv[i];
      rank += (si > sj) || (si == sj && i < j);
    }
    if (sj == sj) order[rank] = j;  // a NaN keeps the unsorted order
  }
  __syncthreads();
  for (int r = threadIdx.x; r < k; r += TTB_THREADS) S[r] = sv[order[r]];
  for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) {
    const int r = e % k, c = e / k;
    Vh(r, c) = V[c + order[r] * ld];
  }
  __syncthreads();
  return status;
}

// U <- [B(:, order) / S; 0] after cta_svd_plain.
static __device__ void cta_top_u(int k, int m, const double* B, const double* sv,
                                 const int* order, Mat U) {
  const i64 ld = k;
  for (int e = threadIdx.x; e < m * k; e += TTB_THREADS) {
    const int i = e % m, r = e / m, j = order[r];
    double v = 0.0;
    if (i < k) v = (sv[j] > 0.0) ? B[i + j * ld] / sv[j] : (i == r ? 1.0 : 0.0);
    U(i, r) = v;
  }
  __syncthreads();
}

// Thin SVD of the m x k matrix A (any strides), m >= k required, as
// A = U diag(S) Vh with S descending: Householder QR A = Q R, the SVD of R
// (cta_svd_square), U = Q [U_R; 0].  A caller that needs one orthonormal
// factor only (the other times S is its product with A) passes the other as
// NULL and saves the accumulation of the rotations.  Work areas (shared or global): W (m x k,
// column major, column step ldw), tau (k), Bsq and V (k columns of svd_step(k) each, 16-byte
// aligned, or k x k when not tiled), sv (k),
// order (2 k ints), flag (1 int), tau2 (k).  U (m x k), S (k) and Vh (k x k)
// are strided outputs.  Returns the Jacobi sweeps used, or -1 if the sweep
// cap was hit.
template <bool TILED>
__device__ __noinline__ int cta_svd_tall(CMat A, int m, int k, double* W, i64 ldw, double* tau,
                                   double* Bsq, double* V, double* sv, int* order, int* flag,
                                   double* tau2, Mat U, double* S, Mat Vh, double* red) {
  cta_load(A, W, ldw, m, k);
  __syncthreads();
  const bool tiles = TILED && hh_tiled(m, k);
  cta_hh_any<TILED>(W, m, k, ldw, tau, red);
  const i64 ld = TILED ? svd_step(k) : k;
  for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) {
    int i = e % k, j = e / k;
    Bsq[i + j * ld] = (i <= j) ? W[i + j * ldw] : 0.0;
  }
  __syncthreads();
  const int want = !Vh.p ? SQ_LEFT : !U.p ? SQ_RIGHT : SQ_BOTH;
  int status;
  if constexpr (TILED)
    status = cta_svd_square(want, k, Bsq, V, sv, order, tau2, flag, U, S, Vh, red);
  else
    status = cta_svd_plain(k, Bsq, V, sv, order, flag, S, Vh);
  if (!U.p) return status;
  if constexpr (!TILED) {
    cta_top_u(k, m, Bsq, sv, order, U);
    cta_apply_q(W, m, k, ldw, tau, U, k);
    return status;
  }
  if (tiles) {
    if constexpr (TILED) cta_hh_apply(W, ldw, m, k, tau, U, k, HH_TOP, V, k, ld, order);
  } else {
    for (int e = threadIdx.x; e < m * k; e += TTB_THREADS) {
      int i = e % m, r = e / m;
      U(i, r) = i < k ? V[i + order[r] * ld] : 0.0;
    }
    __syncthreads();
    cta_apply_q(W, m, k, ldw, tau, U, k);
  }
  return status;
}

// ---------------------------------------------------------------------------
// register-tiled Gaussian elimination
// ---------------------------------------------------------------------------

// Steps 0 .. steps - 1 of Gaussian elimination with partial pivoting on a
// panel of rows x cols held in registers, warp w the columns w, w +
// TTB_WARPS, ..., lane l the rows l, l + 32, ....  Rows stay where they are:
// ``pos`` follows the position each would have had if the rows were swapped
// (the pivot of a step is the largest remaining entry, the one of lowest
// position on ties, as cta_gepp_solve takes it), and a row that has been
// pivot keeps its values.  Each step's multipliers go through ``lbuf`` (2 x
// 32 RPL doubles, shared; zeros in the finished rows), its pivot row through
// ``piv`` (2 ints, shared); ipiv[j], if given, gets the position swapped with
// j.  Every entry sees the updates of cta_gepp_solve in the same order: the
// same bits.  Returns 0 or the 1-based step whose pivot is exactly zero.
// The warp of the next pivot column takes it first and publishes it before
// its other updates, so that a step costs the chain of one column: a search,
// a reciprocal, a barrier; updating in memory took four barriers.
template <int RPL, int CPW>
static __device__ __forceinline__ int lu_steps(double (&x)[CPW][RPL], int (&pos)[RPL], int rows,
                                               int steps, double* lbuf, int* piv, int* ipiv) {
  constexpr int PW = ceil_pow2(RPL);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < RPL; ++r) pos[r] = lane + 32 * r;
  __syncthreads();  // every warp has its columns, and lbuf and piv are free
  for (int j = -1; j < steps; ++j) {
    double l[RPL];
    int slot = 0, from = 0;
    if (j >= 0) {
      if (warp != j % TTB_WARPS) step_wait(j);
      const int pr = piv[j & 1];
      if (pr < 0) return j + 1;
      const double* lb = lbuf + (j & 1) * 32 * RPL;
#pragma unroll
      for (int r = 0; r < RPL; ++r) l[r] = lb[lane + 32 * r];
      slot = pr >> 5;
      from = pr & 31;
      // the pivot row takes position j, the row that was there the pivot's
      int pp = pos[0];
#pragma unroll
      for (int r = 1; r < RPL; ++r) pp = r == slot ? pos[r] : pp;
      pp = __shfl_sync(0xffffffffu, pp, from);
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        if (lane + 32 * r == pr) pos[r] = j;
        else if (pos[r] == j) pos[r] = pp;
      }
      if (ipiv && threadIdx.x == 0) ipiv[j] = pp;
    } else {
#pragma unroll
      for (int r = 0; r < RPL; ++r) l[r] = 0.0;
    }
    const int n = j + 1;  // the next pivot column
    int mine = -1;
    if (n < steps && warp == n % TTB_WARPS) {  // this warp's, and done first
      mine = n / TTB_WARPS;
      double col[RPL];
      pick_slot<RPL, CPW>(x, mine, col);
      if (j >= 0) {
        const double u = __shfl_sync(0xffffffffu, pick_reg<PW, RPL>(col, slot), from);
#pragma unroll
        for (int r = 0; r < RPL; ++r) col[r] = fma(-l[r], u, col[r]);
      }
      // the largest entry, the lowest position on ties, a NaN only where no
      // number is left (at -0.5, below all of them): by the high word (one up,
      // so that a zero is not a NaN's 0), the low word, then position and row
      double best = -1.0;
      unsigned at = 0x7fffffffu;
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const int row = lane + 32 * r;
        const double a = col[r] == col[r] ? fabs(col[r]) : -0.5;
        const unsigned id = ((unsigned)pos[r] << 16) | row;
        const bool in = row < rows && pos[r] >= n;
        if (in && (a > best || (a == best && id < at))) {
          best = a;
          at = id;
        }
      }
      const unsigned hi = best < 0.0 ? 0u : (unsigned)__double2hiint(best) + 1u;
      const unsigned top = __reduce_max_sync(0xffffffffu, hi);
      const unsigned lo = hi == top && hi ? (unsigned)__double2loint(best) : 0u;
      const unsigned low = __reduce_max_sync(0xffffffffu, lo);
      at = __reduce_min_sync(0xffffffffu, hi == top && lo == low ? at : 0x7fffffffu);
      const int pr = (int)(at & 0xffff);
      const double d = __shfl_sync(0xffffffffu, pick_reg<PW, RPL>(col, pr >> 5), pr & 31);
      if (lane == 0) piv[n & 1] = d == 0.0 ? -1 : pr;
      const double rd = 1.0 / d;
      double* lb = lbuf + (n & 1) * 32 * RPL;
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const int row = lane + 32 * r;
        const bool below = pos[r] >= n && row != pr;
        const double q = col[r] * rd;
        lb[row] = below ? q : 0.0;
        col[r] = below ? q : col[r];
      }
      __syncwarp();
      step_arrive(n);
#pragma unroll
      for (int s = 0; s < CPW; ++s)
        if (s == mine) {
#pragma unroll
          for (int r = 0; r < RPL; ++r)
            asm volatile("mov.f64 %0, %1;" : "=d"(x[s][r]) : "d"(col[r]));
        }
    }
    if (j < 0) continue;
#pragma unroll
    for (int s = 0; s < CPW; ++s) {
      if (warp + TTB_WARPS * s <= j || s == mine) continue;
      const double u = __shfl_sync(0xffffffffu, pick_reg<PW, RPL>(x[s], slot), from);
#pragma unroll
      for (int r = 0; r < RPL; ++r) x[s][r] = fma(-l[r], u, x[s][r]);
    }
  }
  return 0;
}

// Solves U x = b for the upper triangle of W (column step ld), x over b, by
// blocks of 32 columns: one warp the diagonal block, every thread the rows
// above it.  Each row sees the columns last to first, one fma each, as a
// column-by-column substitution takes them.
__device__ __noinline__ void cta_back_substitute(const double* W, i64 ld, double* b,
                                                        int n) {
  const int lane = threadIdx.x & 31;
  for (int j0 = ((n - 1) / 32) * 32; j0 >= 0; j0 -= 32) {
    const int jn = min(32, n - j0);
    if (threadIdx.x < 32) {
      double x = lane < jn ? b[j0 + lane] : 0.0;
      const double diag = lane < jn ? W[(j0 + lane) + (j0 + lane) * ld] : 1.0;
      for (int j = jn - 1; j >= 0; --j) {
        const double w = lane < j ? W[(j0 + lane) + (j0 + j) * ld] : 0.0;
        if (lane == j) x = x / diag;
        const double xj = __shfl_sync(0xffffffffu, x, j);
        if (lane < j) x = fma(-w, xj, x);
      }
      if (lane < jn) b[j0 + lane] = x;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < j0; i += TTB_THREADS) {
      double acc = b[i];
      const double* row = W + i + j0 * ld;
#pragma unroll 8
      for (int j = jn - 1; j >= 0; --j) acc = fma(-row[j * ld], b[j0 + j], acc);
      b[i] = acc;
    }
    __syncthreads();
  }
}

// The whole matrix and b in registers: n <= 32 RPL, n + 1 <= TTB_WARPS CPW.
template <int RPL, int CPW>
static __device__ __noinline__ int lu_whole(double* W, i64 ld, double* b, int n, double* lbuf,
                                            int* piv) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double x[CPW][RPL];
  int pos[RPL];
#pragma unroll
  for (int s = 0; s < CPW; ++s) {
    const int c = warp + TTB_WARPS * s;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int i = lane + 32 * r;
      x[s][r] = (c <= n && i < n) ? (c < n ? W[i + c * ld] : b[i]) : 0.0;
    }
  }
  const int info = lu_steps<RPL, CPW>(x, pos, n, n, lbuf, piv, nullptr);
  if (info) return info;
#pragma unroll
  for (int s = 0; s < CPW; ++s) {
    const int c = warp + TTB_WARPS * s;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int i = lane + 32 * r;
      if (c > n || i >= n) continue;
      if (c < n) W[pos[r] + c * ld] = x[s][r];
      else b[pos[r]] = x[s][r];
    }
  }
  __syncthreads();
  cta_back_substitute(W, ld, b, n);
  return 0;
}

// Gaussian elimination with partial pivoting on [W | b] (LAPACK getrf/getrs
// semantics: largest |pivot|, first index on ties), W column major with
// leading dimension ld, then back substitution.  b is overwritten with the
// solution and W with the factors.  ``lbuf`` (shared) holds
// lu_buf_doubles(n).  Returns 0, or the 1-based index of the first exactly-zero pivot
// (the solve then stops, like gesv's info > 0).  Bound by the chain of a
// step (a pivot search, a reciprocal, one barrier): 128 unknowns took 522 us
// with the matrix updated in shared memory and take 193 us.
__device__ __noinline__ int cta_gepp_solve(double* W, i64 ld, double* b, int n, double* lbuf) {
  __shared__ int piv[2];
  int info;
  if (n <= 32) info = lu_whole<1, 5>(W, ld, b, n, lbuf, piv);
  else if (n <= 64) info = lu_whole<2, 9>(W, ld, b, n, lbuf, piv);
  else if (n <= 96) info = lu_whole<3, 13>(W, ld, b, n, lbuf, piv);
  else if (n <= 128) info = lu_whole<4, 17>(W, ld, b, n, lbuf, piv);
  else info = lu_whole<5, 21>(W, ld, b, n, lbuf, piv);
  __syncthreads();
  return info;
}

// One LNB-column panel of the blocked elimination: columns j0 .. of W's rows
// j0 .., factored in registers, written back in pivoted order and, transposed
// for the products, to P (pitch ``pp``): P[c * pp + i] is row i of column c.
template <int RPL>
static __device__ __noinline__ int lu_panel(double* W, i64 ld, int rows, int jb, double* P,
                                            int pp, double* lbuf, int* piv, int* ipiv) {
  constexpr int CPW = 2;
  static_assert(TTB_WARPS * CPW == LNB, "a panel fills the warps' columns");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double x[CPW][RPL];
  int pos[RPL];
#pragma unroll
  for (int s = 0; s < CPW; ++s) {
    const int c = warp + TTB_WARPS * s;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int i = lane + 32 * r;
      x[s][r] = (c < jb && i < rows) ? W[i + c * ld] : 0.0;
    }
  }
  const int info = lu_steps<RPL, CPW>(x, pos, rows, jb, lbuf, piv, ipiv);
  if (info) return info;
  __syncthreads();  // lbuf may share P's memory
#pragma unroll
  for (int s = 0; s < CPW; ++s) {
    const int c = warp + TTB_WARPS * s;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int i = lane + 32 * r;
      if (c >= jb || i >= rows) continue;
      W[pos[r] + c * ld] = x[s][r];
      P[c * pp + pos[r]] = x[s][r];
    }
  }
  __syncthreads();
  return 0;
}

// cta_gepp_solve for a matrix in global memory, kLuWhole < n <= kLuRows,
// panels of LNB columns; ``pool`` (shared) holds lu_panel_doubles(n).  Per
// panel: the panel in registers (cta_gepp_panel); then the trailing columns, a
// strip at a time (cta_gepp_update): row swaps as one permutation of the at
// most 32 rows they touch, the unit-lower solve with a thread per column, both
// into shared memory, and C -= L21 U12 on the FP64 tensor path with C loaded
// straight into the accumulator fragments' lanes, 32 x 16 entries a warp.
// Every entry sees the products and roundings of the plain blocked form
// (cta_gepp_blocked) in the same order, whatever the strips.  The floor on one
// SM is 2 n^3 / 3 flops at 128 a cycle (2.1 ms for 928 unknowns); 928 unknowns
// took 27.4 ms with one synchronised tile at a time and take 10.7 ms, half of
// it waiting for C, so a cluster deals out the strips.
//
// The panel at j0: factored in place, a copy in the pool for cta_gepp_update,
// its row swaps in ``ipiv`` (shared, LNB).  The tiles of 512 and 1024 rows do not
// quite fit the registers and spill 0.3 and 1.2 KB a thread.  Returns 0 or the
// first zero pivot.
__device__ __noinline__ int cta_gepp_panel(double* W, i64 ld, int n, int j0, double* pool,
                                           int* ipiv) {
  __shared__ int piv[2];
  const int jb = min(LNB, n - j0), rows = n - j0, pp = lu_pitch(rows);
  double* Wp = W + j0 + j0 * ld;
  int info;
  if (rows <= 128) info = lu_panel<4>(Wp, ld, rows, jb, pool, pp, pool, piv, ipiv);
  else if (rows <= 256) info = lu_panel<8>(Wp, ld, rows, jb, pool, pp, pool, piv, ipiv);
  else if (rows <= 512) info = lu_panel<16>(Wp, ld, rows, jb, pool, pp, pool, piv, ipiv);
  else info = lu_panel<32>(Wp, ld, rows, jb, pool, pp, pool, piv, ipiv);
  return info ? j0 + info : 0;
}

// The trailing columns and b under the panel at j0: the strips rank, rank +
// size, ...; ``fetch`` reads the panel from W first (a block that did not
// factor it).
__device__ __noinline__ void cta_gepp_update(double* W, i64 ld, double* b, int n, int j0,
                                             double* pool, const int* ipiv, bool fetch, int rank,
                                             int size) {
  __shared__ int nmove, src[2 * LNB], dst[2 * LNB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int jb = min(LNB, n - j0), rows = n - j0, pp = lu_pitch(rows);
  double* P = pool;                       // the panel, row pitch pp
  double* Us = pool + LNB * lu_pitch(n);  // U12's strip, LNB x kLuStripPitch
  double* Wp = W + j0 + j0 * ld;
  const int ncols = n - j0 - jb;  // trailing columns; b comes after them
  // a strip per block where there are that many columns, in tiles of 16
  const int strip = min(kLuStrip, ((ncols + size) / size + 15) & ~15);
  if (fetch)
    for (int e = tid; e < jb * rows; e += TTB_THREADS) {
      const int c = e / rows, i = e % rows;
      P[c * pp + i] = Wp[i + c * ld];
    }
  // the swaps as moves: position dst[e] gets the row that was at src[e]
  if (tid == 0) {
    int cnt = 0;
    for (int c = 0; c < jb; ++c) {
      const int q = ipiv[c];
      int ec = -1, eq = -1;
      for (int e = 0; e < cnt; ++e) {
        if (dst[e] == c) ec = e;
        if (dst[e] == q) eq = e;
      }
      if (ec < 0) { ec = cnt++; dst[ec] = src[ec] = c; }
      if (q == c) continue;
      if (eq < 0) { eq = cnt++; dst[eq] = src[eq] = q; }
      const int v = src[ec];
      src[ec] = src[eq];
      src[eq] = v;
    }
    nmove = cnt;
  }
  // zero rows below the panel, so that the products need no row test
  for (int e = tid; e < LNB * (pp - rows); e += TTB_THREADS) {
    const int c = e / (pp - rows), i = rows + e % (pp - rows);
    P[c * pp + i] = 0.0;
  }
  if (jb < LNB)
    for (int e = tid; e < (LNB - jb) * pp; e += TTB_THREADS) P[jb * pp + e] = 0.0;
  __syncthreads();
  const int cnt = nmove;
  for (int s0 = rank * strip; s0 <= ncols; s0 += size * strip) {
    const int sn = min(strip, ncols + 1 - s0);
    // swaps: four columns of a warp in flight
    for (int c4 = 4 * warp; c4 < sn; c4 += 4 * TTB_WARPS) {
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = s0 + c4 + u;
        const double* col = c < ncols ? Wp + (jb + c) * ld : b + j0;
        v[u] = (c4 + u < sn && lane < cnt) ? col[src[lane]] : 0.0;
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = s0 + c4 + u;
        double* col = c < ncols ? Wp + (jb + c) * ld : b + j0;
        if (c4 + u >= sn || lane >= cnt) continue;
        const int to = dst[lane];
        if (to < jb) Us[to * kLuStripPitch + c4 + u] = v[u];
        else col[to] = v[u];
      }
    }
    if (jb < LNB)
      for (int e = tid; e < (LNB - jb) * sn; e += TTB_THREADS)
        Us[(jb + e / sn) * kLuStripPitch + e % sn] = 0.0;
    __syncthreads();
    // the unit-lower solve, a thread per column
    for (int c = tid; c < sn; c += TTB_THREADS) {
      double y[LNB];
#pragma unroll
      for (int r = 0; r < LNB; ++r) {
        y[r] = Us[r * kLuStripPitch + c];
        double acc = y[r];
#pragma unroll
        for (int q = 0; q < r; ++q) acc = fma(-P[q * pp + r], y[q], acc);
        y[r] = r < jb ? acc : 0.0;
        Us[r * kLuStripPitch + c] = y[r];
      }
    }
    __syncthreads();
    for (int e = tid; e < sn * LNB; e += TTB_THREADS) {
      const int r = e % LNB, c = e / LNB;
      double* col = s0 + c < ncols ? Wp + (jb + s0 + c) * ld : b + j0;
      if (r < jb) col[r] = Us[r * kLuStripPitch + c];
    }
    // C -= L21 U12, b2 -= L21 u_b
    const int below = rows - jb, wide = min(sn, ncols - s0);
    const int tm = (below + 31) / 32, tn = (wide + 15) / 16;
    if (below > 0 && wide > 0) {
      for (int tile = warp; tile < tm * tn; tile += TTB_WARPS) {
        const int m0 = jb + (tile % tm) * 32, n0 = (tile / tm) * 16;
        double c0[4][2][2], acc[4][2][2];
        double* cp[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int cc = n0 + 8 * j + 2 * t + h;
            cp[j][h] = cc < wide ? Wp + (jb + s0 + cc) * ld : nullptr;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int r = m0 + 8 * i + g;
              acc[i][j][h] = 0.0;
              c0[i][j][h] = (cp[j][h] && r < rows) ? cp[j][h][r] : 0.0;
            }
          }
#pragma unroll
        for (int kk = 0; kk < LNB; kk += 4) {
          if (kk >= jb) break;
          double av[4], bv[2];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = m0 + 8 * i + g;
            av[i] = r < pp ? P[(kk + t) * pp + r] : 0.0;
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) bv[j] = Us[(kk + t) * kLuStripPitch + n0 + 8 * j + g];
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (!cp[j][h]) continue;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int r = m0 + 8 * i + g;
              if (r < rows) cp[j][h][r] = fma(1.0, c0[i][j][h], -1.0 * acc[i][j][h]);
            }
          }
      }
    }
    if (s0 + sn > ncols) {  // this strip holds b, in its last column
      for (int i = tid; i < below; i += TTB_THREADS) {
        double acc = b[j0 + jb + i];
        for (int q = 0; q < jb; ++q)
          acc = fma(-P[q * pp + jb + i], Us[q * kLuStripPitch + sn - 1], acc);
        b[j0 + jb + i] = acc;
      }
    }
    __syncthreads();  // the strip's reads are done
  }
}

static __device__ __noinline__ int cta_gepp_strips(double* W, i64 ld, double* b, int n,
                                                   double* pool) {
  __shared__ int ipiv[LNB];
  for (int j0 = 0; j0 < n; j0 += LNB) {
    if (const int info = cta_gepp_panel(W, ld, n, j0, pool, ipiv)) return info;
    cta_gepp_update(W, ld, b, n, j0, pool, ipiv, false, 0, 1);
  }
  cta_back_substitute(W, ld, b, n);
  return 0;
}

// ---------------------------------------------------------------------------
// blocked factorisations for matrices that do not fit in shared memory
// ---------------------------------------------------------------------------


// Blocked Gaussian elimination with partial pivoting on [W | b] (W column
// major, leading dimension ld), panels of LNB columns factored in ``panel``
// (rows x LNB doubles, shared or global memory), trailing updates as GEMMs.
// Same pivot rule and result as cta_gepp_solve; b becomes the solution.
__device__ __noinline__ int cta_gepp_blocked(double* W, i64 ld, double* b, int n, double* panel, double* redv,
                                int* redi, int* ipiv, GemmSmem& gsm, double* ring) {
  if (n <= kLuRows && __isShared(panel)) return cta_gepp_strips(W, ld, b, n, panel);
  const int tid = threadIdx.x;
  for (int j0 = 0; j0 < n; j0 += LNB) {
    const int jb = min(LNB, n - j0);
    const int rows = n - j0;
    double* P = panel;
    for (int e = tid; e < rows * jb; e += TTB_THREADS) {
      int i = e % rows, c = e / rows;
      P[i + (i64)c * rows] = W[(j0 + i) + (i64)(j0 + c) * ld];
    }
    __syncthreads();
    for (int c = 0; c < jb; ++c) {
      double best = -1.0;
      int bi = -1;
      for (int i = c + tid; i < rows; i += TTB_THREADS) {
        double a = fabs(P[i + (i64)c * rows]);
        if (a > best) { best = a; bi = i; }
      }
      // a column of NaN has no largest entry (-1): its own row
      const int piv = max(block_argmax_abs(best, bi, redv, redi), c);
      if (tid == 0) ipiv[c] = piv;
      if (piv != c) {
        for (int cc = tid; cc < jb; cc += TTB_THREADS) {
          double t = P[c + (i64)cc * rows];
          P[c + (i64)cc * rows] = P[piv + (i64)cc * rows];
          P[piv + (i64)cc * rows] = t;
        }
      }
      __syncthreads();
      const double d = P[c + (i64)c * rows];
      if (d == 0.0) return j0 + c + 1;
      const double rd = 1.0 / d;
      for (int i = c + 1 + tid; i < rows; i += TTB_THREADS) P[i + (i64)c * rows] *= rd;
      __syncthreads();
      const int rr = rows - c - 1, cw = jb - c - 1;
      for (int e = tid; e < rr * cw; e += TTB_THREADS) {
        int i = c + 1 + e % rr, cc = c + 1 + e / rr;
        P[i + (i64)cc * rows] = fma(-P[i + (i64)c * rows], P[c + (i64)cc * rows],
                                    P[i + (i64)cc * rows]);
      }
      __syncthreads();
    }
    for (int e = tid; e < rows * jb; e += TTB_THREADS) {
      int i = e % rows, c = e / rows;
      W[(j0 + i) + (i64)(j0 + c) * ld] = P[i + (i64)c * rows];
    }
    // row swaps and the unit-lower solve on the columns right of the panel
    // and on b; each thread owns whole columns, so no synchronisation
    const int ncols = n - j0 - jb;
    for (int col = tid; col <= ncols; col += TTB_THREADS) {
      double* x = (col < ncols) ? W + (i64)(j0 + jb + col) * ld + j0 : b + j0;
      for (int c = 0; c < jb; ++c) {
        const int piv = ipiv[c];
        if (piv != c) {
          double t = x[c];
          x[c] = x[piv];
          x[piv] = t;
        }
      }
      for (int r = 1; r < jb; ++r) {
        double acc = x[r];
        for (int q = 0; q < r; ++q) acc = fma(-P[r + (i64)q * rows], x[q], acc);
        x[r] = acc;
      }
    }
    __syncthreads();
    if (rows > jb) {
      // A22 -= L21 U12 ; b2 -= L21 u_b
      if (ncols > 0)
        gemm_sel(CMat{P + jb, 1, rows}, CMat{W + j0 + (i64)(j0 + jb) * ld, 1, ld},
                 Mat{W + (j0 + jb) + (i64)(j0 + jb) * ld, 1, ld}, rows - jb, ncols, jb, -1.0,
                 1.0, gsm, ring);
      for (int i = tid; i < rows - jb; i += TTB_THREADS) {
        double acc = b[j0 + jb + i];
        for (int q = 0; q < jb; ++q) acc = fma(-P[jb + i + (i64)q * rows], b[j0 + q], acc);
        b[j0 + jb + i] = acc;
      }
    }
    __syncthreads();
  }
  cta_back_substitute(W, ld, b, n);
  return 0;
}

// T factor (jb x jb, upper triangular, column major in Tm) of the block
// reflector H_0 ... H_{jb-1} = I - V T V^T, V the rows x jb explicit
// reflector block (unit diagonal, zeros above) in Wp with leading dim ldw
// (LAPACK dlarft, forward column-wise).  G is jb x jb scratch.
static __device__ void cta_block_t(const double* Wp, i64 ldw, int rows, int jb, const double* tau,
                            double* G, double* Tm, GemmSmem& gsm, double* ring) {
  gemm_sel(CMat{Wp, ldw, 1}, CMat{Wp, 1, ldw}, Mat{G, 1, LNB}, jb, jb, rows, 1.0, 0.0, gsm, ring);
  const int tid = threadIdx.x;
  for (int e = tid; e < LNB * LNB; e += TTB_THREADS) Tm[e] = 0.0;
  __syncthreads();
  for (int i = 0; i < jb; ++i) {  // column i, a thread per entry
    if (tid < i) {
      double acc = 0.0;
      for (int r = tid; r < i; ++r) acc = fma(Tm[tid + r * LNB], G[r + i * LNB], acc);
      Tm[tid + i * LNB] = -tau[i] * acc;
    }
    if (tid == i) Tm[i + i * LNB] = tau[i];
    __syncthreads();
  }
}

// X (m x nx, strided) <- H_0 ... H_{p-1} X for the block reflectors left in
// W by cta_qr_blocked (explicit reflector blocks, leading dimension m),
// applied last block first; only rows >= the block's first row change.
// Columns of X left of a block are untouched (as for an identity start).
static __device__ void cta_apply_q_blocked(const double* W, int m, int p, const double* tau, Mat X,
                                    int nx, double* Y, double* G, double* Tm, GemmSmem& gsm, double* ring) {
  const int tid = threadIdx.x;
  const int last = ((p - 1) / LNB) * LNB;
  for (int j0 = last; j0 >= 0; j0 -= LNB) {
    const int jb = min(LNB, p - j0);
    const int rows = m - j0;
    const double* Wp = W + j0 + (i64)j0 * m;
    cta_block_t(Wp, m, rows, jb, tau + j0, G, Tm, gsm, ring);
    for (int c0 = 0; c0 < nx; c0 += YCH) {
      const int nc = min(YCH, nx - c0);
      Mat Xs{X.p + j0 * X.rs + c0 * X.cs, X.rs, X.cs};
      gemm_sel(CMat{Wp, m, 1}, CMat{Xs.p, Xs.rs, Xs.cs}, Mat{Y, 1, LNB}, jb, nc, rows, 1.0, 0.0,
               gsm, ring);
      for (int col = tid; col < nc; col += TTB_THREADS) {
        double y[LNB];
        for (int i = 0; i < jb; ++i) y[i] = Y[i + (i64)col * LNB];
        for (int i = 0; i < jb; ++i) {
          double acc = 0.0;
          for (int q = i; q < jb; ++q) acc = fma(Tm[i + q * LNB], y[q], acc);
          Y[i + (i64)col * LNB] = acc;
        }
      }
      __syncthreads();
      gemm_sel(CMat{Wp, 1, m}, CMat{Y, 1, LNB}, Xs, rows, nc, jb, -1.0, 1.0, gsm, ring);
    }
  }
}

// Blocked (compact WY) economic QR of the m x k matrix A into the m x k
// column-major work area W (global), panels of LNB columns: Householder on
// the panel (cta_householder), the T factor, then the trailing update
// C -= V (T^T (V^T C)) as two GEMMs through Y (LNB x k, shared).  Q (m x p)
// and R (p x k) as in cta_qr; either may be NULL.  Same reflectors and R as
// the unblocked factorisation up to rounding.
template <bool TILED>
__device__ __noinline__ void cta_qr_blocked(CMat A, int m, int k, double* W, double* tau, Mat Q, Mat R,
                               double* Y, double* G, double* Tm, double* red, GemmSmem& gsm, double* ring) {
  if constexpr (TILED) {
    if (m <= kHHTall) {
      cta_qr<true>(A, m, k, W, m, tau, Q, R, red);
      return;
    }
  }
  const int p = m < k ? m : k;
  const int tid = threadIdx.x;
  cta_load(A, W, m, m, k);
  __syncthreads();
  for (int j0 = 0; j0 < p; j0 += LNB) {
    const int jb = min(LNB, p - j0);
    const int rows = m - j0;
    double* Wp = W + j0 + (i64)j0 * m;
    cta_hh_any<TILED>(Wp, rows, jb, m, tau + j0, red);
    // R's diagonal block, then the explicit reflector form in its place
    for (int e = tid; e < jb * jb; e += TTB_THREADS) {
      int r = e % jb, c = e / jb;
      if (r <= c) {
        if (R.p) R(j0 + r, j0 + c) = Wp[r + (i64)c * m];
        Wp[r + (i64)c * m] = (r == c) ? 1.0 : 0.0;
      }
    }
    __syncthreads();
    const int nt = k - j0 - jb;
    if (nt > 0) {
      cta_block_t(Wp, m, rows, jb, tau + j0, G, Tm, gsm, ring);
      for (int c0 = 0; c0 < nt; c0 += YCH) {
        const int nc = min(YCH, nt - c0);
        double* C = W + j0 + (i64)(j0 + jb + c0) * m;
        // Y = V^T C (jb x nc), then Y = T^T Y, then C -= V Y
        gemm_sel(CMat{Wp, m, 1}, CMat{C, 1, m}, Mat{Y, 1, LNB}, jb, nc, rows, 1.0, 0.0, gsm, ring);
        for (int col = tid; col < nc; col += TTB_THREADS) {
          double y[LNB];
          for (int i = 0; i < jb; ++i) y[i] = Y[i + (i64)col * LNB];
          for (int i = jb - 1; i >= 0; --i) {
            double acc = 0.0;
            for (int q = 0; q <= i; ++q) acc = fma(Tm[q + i * LNB], y[q], acc);
            Y[i + (i64)col * LNB] = acc;
          }
        }
        __syncthreads();
        gemm_sel(CMat{Wp, 1, m}, CMat{Y, 1, LNB}, Mat{C, 1, m}, rows, nc, jb, -1.0, 1.0, gsm, ring);
      }
    }
  }
  if (R.p) {
    for (int e = tid; e < p * k; e += TTB_THREADS) {
      int i = e % p, j = e / p;
      int jp = (i / LNB) * LNB;  // panel of row i
      bool in_diag_block = (j >= jp && j < jp + LNB && j < p);
      if (i > j) R(i, j) = 0.0;
      else if (!in_diag_block) R(i, j) = W[i + (i64)j * m];
    }
  }
  if (Q.p) {
    for (int e = tid; e < m * p; e += TTB_THREADS) {
      int i = e % m, j = e / m;
      Q(i, j) = (i == j) ? 1.0 : 0.0;
    }
    __syncthreads();
    cta_apply_q_blocked(W, m, p, tau, Q, p, Y, G, Tm, gsm, ring);
  }
  __syncthreads();
}

// Every block of a cluster of ``size`` at a point, its global writes visible
// to the others; one block: its threads.
static __device__ __forceinline__ void team_sync(int size) {
  if (size > 1) {
    cooperative_groups::this_cluster().sync();
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
  } else {
    __syncthreads();
  }
}

// cta_householder of a panel (k <= LNB) by the blocks of a cluster, every
// entry and sum as the lone block computes it: that block's warp ``vw`` takes
// the rows j + 1 + 32 vw + lane + TTB_THREADS i of a step, so block ``rank``
// takes the rows of the warps rank, rank + size, ..., its own warps two
// columns each, and the warps' partial sums go to every block.  Two cluster
// barriers a column.  A lone block reads and writes the panel through one
// multiprocessor's path to L2: 6400 x 16 is 13 us a column there.
static __device__ __noinline__ void team_householder(double* W, int m, int k, i64 ldw, double* tau,
                                                     int rank, int size) {
  static_assert(LNB <= 2 * TTB_WARPS, "two columns a warp");
  constexpr int U = 8;  // rows of a lane in flight
  __shared__ double hred[TTB_WARPS][LNB], nred[TTB_WARPS], hw[LNB];
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int p = min(m, k);
  for (int vw = rank; vw < TTB_WARPS; vw += size) {
    if (wid != vw / size) continue;
    double part = 0.0;
#pragma unroll 8
    for (int i = 1 + 32 * vw + lane; i < m; i += TTB_THREADS) part = fma(W[i], W[i], part);
    part = warp_sum(part);
    if (lane < size) *cl.map_shared_rank(&nred[vw], lane) = part;
  }
  team_sync(size);
  for (int j = 0; j < p; ++j) {
    double sigma = 0.0;
    for (int w = 0; w < TTB_WARPS; ++w) sigma += nred[w];
    double* col = W + j * ldw;
    double* cb = col + ldw;
    const int nc = k - j - 1;
    const double alpha = col[j];
    const double rowj = tid < nc ? cb[j + tid * ldw] : 0.0;
    double t = 0.0, beta = alpha, scale = 0.0;
    if (sigma != 0.0) {
      const double nrm = sqrt(alpha * alpha + sigma);
      beta = (alpha >= 0.0) ? -nrm : nrm;
      t = (beta - alpha) / beta;
      scale = 1.0 / (alpha - beta);
      for (int vw = rank; vw < TTB_WARPS; vw += size)
        for (int i = j + 1 + 32 * vw + lane + TTB_THREADS * wid; i < m;
             i += TTB_THREADS * TTB_WARPS)
          col[i] *= scale;
    }
    __syncthreads();
    const int q0 = wid, q1 = wid + TTB_WARPS;  // this warp's columns
    const double* c0 = cb + q0 * ldw;
    const double* c1 = cb + q1 * ldw;
    if (t != 0.0 && q0 < nc) {
      for (int vw = rank; vw < TTB_WARPS; vw += size) {
        double w0 = 0.0, w1 = 0.0;
#pragma unroll 8
        for (int i = j + 1 + 32 * vw + lane; i < m; i += TTB_THREADS) {
          const double v = col[i];
          w0 = fma(v, c0[i], w0);
          if (q1 < nc) w1 = fma(v, c1[i], w1);
        }
        w0 = warp_sum(w0);
        w1 = warp_sum(w1);
        if (lane < size) {
          double* to = cl.map_shared_rank(&hred[vw][0], lane);
          to[q0] = w0;
          if (q1 < nc) to[q1] = w1;
        }
      }
    }
    team_sync(size);  // the sums are in; alpha and row j are read
    if (rank == 0 && tid == 0) {
      col[j] = beta;
      tau[j] = t;
    }
    if (t != 0.0) {
      if (tid < nc) {
        double sw = 0.0;
        for (int w = 0; w < TTB_WARPS; ++w) sw += hred[w][tid];
        const double wv = t * (sw + rowj);
        hw[tid] = wv;
        if (rank == 0) cb[j + tid * ldw] = rowj - wv;
      }
      __syncthreads();
    }
    for (int vw = rank; vw < TTB_WARPS; vw += size) {
      double next = 0.0;  // of |column j + 1, rows > j + 1|^2, by warp 0
      if (t != 0.0 && q0 < nc) {
        const double h0 = -hw[q0], h1 = q1 < nc ? -hw[q1] : 0.0;
        for (int i0 = j + 1 + 32 * vw + lane; i0 < m; i0 += U * TTB_THREADS) {
          double v[U], x0[U], x1[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int i = i0 + u * TTB_THREADS;
            v[u] = i < m ? col[i] : 0.0;
            x0[u] = i < m ? c0[i] : 0.0;
            x1[u] = (i < m && q1 < nc) ? c1[i] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int i = i0 + u * TTB_THREADS;
            if (i >= m) continue;
            const double x = fma(h0, v[u], x0[u]);
            cb[i + q0 * ldw] = x;
            if (q1 < nc) cb[i + q1 * ldw] = fma(h1, v[u], x1[u]);
            if (q0 == 0 && i > j + 1) next = fma(x, x, next);
          }
        }
      } else if (nc > 0 && wid == 0) {
        for (int i = j + 2 + 32 * vw + lane; i < m; i += TTB_THREADS)
          next = fma(cb[i], cb[i], next);
      }
      if (wid == 0) {
        next = warp_sum(next);
        if (lane < size) *cl.map_shared_rank(&nred[vw], lane) = next;
      }
    }
    team_sync(size);  // the panel and the next norm are complete
  }
}

// R factor only of the economic QR of the m x k view A, two-level blocked
// for tall operands: outer panels of LNB2 columns are factorised by the
// LNB-blocked Householder code (trailing updates inside the panel only),
// then the panel's LNB2 reflectors update the rest of the matrix as one
// compact-WY block, C -= V (T^T (V^T C)), whose products have 64-wide tiles
// and long K.  Same reflectors as cta_qr_blocked.  W (m x k column major)
// and tau (min(m, k)) are global work; ``pool`` (shared) holds
// 2 LNB2^2 + LNB2^2 + LNB * LNB2 + 2 LNB^2 doubles.  The blocks of a cluster
// may call it together (A, W, tau in global memory, R the leader's): they
// share the inner panels' reflectors and take the outer updates a chunk of
// LNB2 columns each, with the lone block's bits.
__device__ __noinline__ void cta_qr_r_blocked2(CMat A, int m, int k, double* W, double* tau,
                                                      Mat R, double* pool, double* red,
                                                      double* ring, int rank, int size) {
  const int p = m < k ? m : k;
  const int tid = threadIdx.x;
  double* G2 = pool;                      // LNB2 x LNB2: V^T V, later T^T Y
  double* T2 = G2 + LNB2 * LNB2;          // LNB2 x LNB2 upper triangular
  double* Yo = T2 + LNB2 * LNB2;          // LNB2 x LNB2 chunk of V^T C
  double* Yi = Yo + LNB2 * LNB2;          // LNB x LNB2 (inner updates)
  double* Gi = Yi + LNB * LNB2;
  double* Ti = Gi + LNB * LNB;
  {
    const int l0 = (int)((i64)k * rank / size), l1 = (int)((i64)k * (rank + 1) / size);
    cta_load(CMat{A.p + l0 * A.cs, A.rs, A.cs}, W + (i64)l0 * m, m, m, l1 - l0);
  }
  team_sync(size);
  for (int o0 = 0; o0 < p; o0 += LNB2) {
    const int ob = min(LNB2, p - o0);
    const int orows = m - o0;
    double* Wo = W + o0 + (i64)o0 * m;
    // inner LNB-blocked factorisation of the panel's ob columns
    for (int j0 = o0; j0 < o0 + ob; j0 += LNB) {
      const int jb = min(LNB, o0 + ob - j0);
      const int rows = m - j0;
      double* Wp = W + j0 + (i64)j0 * m;
      if (size > 1) {
        team_householder(Wp, rows, jb, m, tau + j0, rank, size);
        if (rank > 0) {
          team_sync(size);  // the leader updates the outer panel
          continue;
        }
      } else {
        cta_householder(Wp, rows, jb, m, tau + j0, red);
      }
      for (int e = tid; e < jb * jb; e += TTB_THREADS) {
        int r = e % jb, c = e / jb;
        if (r <= c) {
          R(j0 + r, j0 + c) = Wp[r + (i64)c * m];
          Wp[r + (i64)c * m] = (r == c) ? 1.0 : 0.0;
        }
      }
      __syncthreads();
      const int nt = o0 + ob - j0 - jb;
      if (nt > 0) {
        // T of the block (as cta_block_t), column by column over the block
        cta_gemm_pipe(CMat{Wp, m, 1}, CMat{Wp, 1, m}, Mat{Gi, 1, LNB}, jb, jb, rows, 1.0, 0.0,
                      ring);
        for (int e = tid; e < LNB * LNB; e += TTB_THREADS) Ti[e] = 0.0;
        __syncthreads();
        for (int i = 0; i < jb; ++i) {
          if (tid < i) {
            double acc = 0.0;
            for (int r = tid; r < i; ++r) acc = fma(Ti[tid + r * LNB], Gi[r + i * LNB], acc);
            Ti[tid + i * LNB] = -tau[j0 + i] * acc;
          }
          if (tid == 0) Ti[i + i * LNB] = tau[j0 + i];
          __syncthreads();
        }
        double* C = W + j0 + (i64)(j0 + jb) * m;
        cta_gemm_pipe(CMat{Wp, m, 1}, CMat{C, 1, m}, Mat{Yi, 1, LNB}, jb, nt, rows, 1.0, 0.0,
                      ring);
        for (int col = tid; col < nt; col += TTB_THREADS) {
          double y[LNB];
          for (int i = 0; i < jb; ++i) y[i] = Yi[i + (i64)col * LNB];
          for (int i = jb - 1; i >= 0; --i) {
            double acc = 0.0;
            for (int q = 0; q <= i; ++q) acc = fma(Ti[q + i * LNB], y[q], acc);
            Yi[i + (i64)col * LNB] = acc;
          }
        }
        __syncthreads();
        cta_gemm_pipe(CMat{Wp, 1, m}, CMat{Yi, 1, LNB}, Mat{C, 1, m}, rows, nt, jb, -1.0, 1.0,
                      ring);
      }
      if (size > 1) team_sync(size);
    }
    // R entries above the inner diagonal blocks move out; V gets zeros there
    for (int e = tid; rank == 0 && e < ob * ob; e += TTB_THREADS) {
      int r = e % ob, c = e / ob;
      if (r < c && (r / LNB) != (c / LNB)) {
        R(o0 + r, o0 + c) = Wo[r + (i64)c * m];
        Wo[r + (i64)c * m] = 0.0;
      }
    }
    team_sync(size);
    const int nt = k - o0 - ob;
    if (nt <= 0) continue;
    // T of the panel: T[i, i] = tau_i, T[0:i, i] = -tau_i T[0:i, 0:i] (V^T V)[0:i, i]
    cta_gemm_pipe(CMat{Wo, m, 1}, CMat{Wo, 1, m}, Mat{G2, 1, LNB2}, ob, ob, orows, 1.0, 0.0, ring);
    for (int e = tid; e < LNB2 * LNB2; e += TTB_THREADS) T2[e] = 0.0;
    __syncthreads();
    for (int i = 0; i < ob; ++i) {
      const double ti = tau[o0 + i];
      for (int q = tid; q < i; q += TTB_THREADS) {
        double acc = 0.0;
        for (int r = q; r < i; ++r) acc = fma(T2[q + r * LNB2], G2[r + i * LNB2], acc);
        T2[q + i * LNB2] = -ti * acc;
      }
      if (tid == 0) T2[i + i * LNB2] = ti;
      __syncthreads();
    }
    for (int c0 = rank * LNB2; c0 < nt; c0 += size * LNB2) {
      const int nc = min(LNB2, nt - c0);
      double* C = W + o0 + (i64)(o0 + ob + c0) * m;
      // Yo = V^T C, G2 = T^T Yo, C -= V G2
      cta_gemm_pipe(CMat{Wo, m, 1}, CMat{C, 1, m}, Mat{Yo, 1, LNB2}, ob, nc, orows, 1.0, 0.0, ring);
      cta_gemm_pipe(CMat{T2, LNB2, 1}, CMat{Yo, 1, LNB2}, Mat{G2, 1, LNB2}, ob, nc, ob, 1.0, 0.0,
                    ring);
      cta_gemm_pipe(CMat{Wo, 1, m}, CMat{G2, 1, LNB2}, Mat{C, 1, m}, orows, nc, ob, -1.0, 1.0,
                    ring);
    }
    if (size > 1) team_sync(size);
  }
  // the rest of R: below the diagonal zero, right of each outer panel from W
  for (int e = tid; rank == 0 && e < p * k; e += TTB_THREADS) {
    int i = e % p, j = e / p;
    if (i > j) {
      R(i, j) = 0.0;
    } else if (j >= min((i / LNB2) * LNB2 + LNB2, p)) {
      R(i, j) = W[i + (i64)j * m];
    }
  }
  __syncthreads();
}

// cta_svd_tall for matrices that do not fit in shared memory: blocked QR
// into the global work area W, the SVD of R in Bsq/V (global or shared), U
// by the reflectors.  Y needs LNB * max(k, 1) doubles, G and Tm LNB * LNB
// each (shared).
template <bool TILED>
__device__ __noinline__ int cta_svd_tall_blocked(CMat A, int m, int k, double* W, double* tau,
                                           double* Bsq, double* V, double* sv, int* order,
                                           int* flag, double* tau2, Mat U, double* S, Mat Vh,
                                           double* Y, double* G, double* Tm, double* red,
                                           GemmSmem& gsm, double* ring) {
  const i64 ld = TILED ? svd_step(k) : k;
  cta_qr_blocked<TILED>(A, m, k, W, tau, Mat{nullptr, 0, 0}, Mat{Bsq, 1, ld}, Y, G, Tm, red, gsm,
                        ring);
  __syncthreads();
  const int want = !Vh.p ? SQ_LEFT : !U.p ? SQ_RIGHT : SQ_BOTH;
  int status;
  if constexpr (TILED)
    status = cta_svd_square(want, k, Bsq, V, sv, order, tau2, flag, U, S, Vh, red);
  else
    status = cta_svd_plain(k, Bsq, V, sv, order, flag, S, Vh);
  if (!U.p) return status;
  if constexpr (!TILED) {
    cta_top_u(k, m, Bsq, sv, order, U);
    cta_apply_q_blocked(W, m, k, tau, U, k, Y, G, Tm, gsm, ring);
    return status;
  }
  if (m <= kHHTall) {
    if constexpr (TILED) cta_hh_apply(W, m, m, k, tau, U, k, HH_TOP, V, k, ld, order);
    return status;
  }
  for (int e = threadIdx.x; e < m * k; e += TTB_THREADS) {
    int i = e % m, r = e / m;
    U(i, r) = i < k ? V[i + order[r] * ld] : 0.0;
  }
  __syncthreads();
  cta_apply_q_blocked(W, m, k, tau, U, k, Y, G, Tm, gsm, ring);
  return status;
}

// cta_svd_tall_blocked with the iteration left to a cluster in between:
// everything in global memory.
__device__ __noinline__ void cta_svd_before(CMat A, int m, int k, double* W, double* tau,
                                            double* Bsq, double* V, double* sv, int* order,
                                            int* flags, double* tau2, Mat U, Mat Vh, double* Y,
                                            double* G, double* Tm, double* red, GemmSmem& gsm) {
  cta_qr_blocked<true>(A, m, k, W, tau, Mat{nullptr, 0, 0}, Mat{Bsq, 1, svd_step(k)}, Y, G, Tm,
                       red, gsm, nullptr);
  __syncthreads();
  const int want = !Vh.p ? SQ_LEFT : !U.p ? SQ_RIGHT : SQ_BOTH;
  square_prepare(want, k, Bsq, V, sv, order, tau2, U, red);
  if (threadIdx.x == 0) flags[0] = 0;
}

__device__ __noinline__ int cluster_svd_iterate(bool left, bool right, int k, double* Bsq,
                                                double* V, int* flags) {
  const int want = !right ? SQ_LEFT : !left ? SQ_RIGHT : SQ_BOTH;
  const i64 ld = svd_step(k);
  double *F, *X;
  square_roles(want, k, Bsq, V, F, X);
  const double tol = square_tol(k);
  return want == SQ_BOTH ? cluster_iterate<true>(X, k, ld, F, tol, flags)
                         : cluster_iterate<false>(X, k, ld, nullptr, tol, flags);
}

__device__ __noinline__ void cta_svd_after(int m, int k, double* W, double* tau, double* Bsq,
                                           double* V, double* sv, int* order, double* tau2,
                                           int* flag, Mat U, double* S, Mat Vh, double* Y,
                                           double* G, double* Tm, double* red, GemmSmem& gsm) {
  const i64 ld = svd_step(k);
  const int want = !Vh.p ? SQ_LEFT : !U.p ? SQ_RIGHT : SQ_BOTH;
  square_finish(want, k, Bsq, V, sv, order, tau2, flag, S, Vh, red);
  if (!U.p) return;
  const double* top = square_left(want, k, Bsq, V);
  if (m <= kHHTall) {
    cta_hh_apply(W, m, m, k, tau, U, k, HH_TOP, top, k, ld, order);
    return;
  }
  for (int e = threadIdx.x; e < m * k; e += TTB_THREADS) {
    int i = e % m, r = e / m;
    U(i, r) = i < k ? top[i + order[r] * ld] : 0.0;
  }
  __syncthreads();
  cta_apply_q_blocked(W, m, k, tau, U, k, Y, G, Tm, gsm, nullptr);
}

// ---------------------------------------------------------------------------
// nodes of a tree of factorisations (ttb200.cu)
// ---------------------------------------------------------------------------

__device__ __noinline__ void cta_node_factor(CMat A, int rows, int k, double* W, i64 ld,
                                             double* tau, double* smem, Mat R) {
  double* F = smem ? smem : W;
  const i64 lf = smem ? ld + 2 : ld;
  if (F != A.p) cta_load(A, F, lf, rows, k);
  __syncthreads();
  cta_hh(F, lf, rows, k, tau);
  const int p = min(rows, k);
  for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) {
    const int i = e % k, j = e / k;
    R(i, j) = (i < p && i <= j) ? F[i + j * lf] : 0.0;
  }
  if (smem)
    for (int e = threadIdx.x; e < rows * k; e += TTB_THREADS) {
      const int i = e % rows, j = e / rows;
      W[i + j * ld] = F[i + j * lf];
    }
}

__device__ __noinline__ void cta_node_apply(const double* W, i64 ld, int rows, int k,
                                            const double* tau, double* smem, const double* top,
                                            i64 ktop, Mat X, int c0, int nc) {
  const double* F = W;
  i64 lf = ld;
  if (smem) {
    lf = ld + 2;
    for (int e = threadIdx.x; e < rows * k; e += TTB_THREADS) {
      const int i = e % rows, j = e / rows;
      smem[i + j * lf] = W[i + j * ld];
    }
    F = smem;
  }
  __syncthreads();
  const Mat Xc{X.p + c0 * X.cs, X.rs, X.cs};
  if (top) {
    cta_hh_apply(F, lf, rows, min(rows, k), tau, Xc, nc, HH_TOP, top + c0 * ktop, k, ktop);
    return;
  }
  for (int e = threadIdx.x; e < rows * nc; e += TTB_THREADS) {
    const int i = e % rows, c = e / rows;
    Xc(i, c) = i == c0 + c ? 1.0 : 0.0;
  }
  __syncthreads();
  cta_hh_apply(F, lf, rows, min(rows, k), tau, Xc, nc, HH_X);
}

__device__ __noinline__ int cta_triangle_svd(const double* R, int k, double* work, Mat Us,
                                             double* S, Mat Vh, double* top, double* red) {
  const i64 ld = svd_step(k);
  double* B = align2(work);
  double* V = B + ld * k;
  double* sv = V + ld * k;
  int* order = reinterpret_cast<int*>(sv + k);
  double* tau2 = sv + 2 * k;
  int* flag = reinterpret_cast<int*>(sv + 3 * k);
  for (int e = threadIdx.x; e < k * k; e += TTB_THREADS) B[e % k + (e / k) * ld] = R[e];
  __syncthreads();
  const int want = !Vh.p ? SQ_LEFT : !top ? SQ_RIGHT : SQ_BOTH;
  const int status = cta_svd_square(want, k, B, V, sv, order, tau2, flag, Us, S, Vh, red);
  if (top)
    for (int e = threadIdx.x; e < k * k; e += TTB_THREADS)
      top[e] = V[e % k + order[e / k] * ld];
  return status;
}

#define TTB_FACTOR_INSTANCE(T)                                                                    \
  template __device__ void cta_qr<T>(CMat, int, int, double*, i64, double*, Mat, Mat, double*);    \
  template __device__ void cta_qr_blocked<T>(CMat, int, int, double*, double*, Mat, Mat, double*,  \
                                             double*, double*, double*, GemmSmem&, double*);      \
  template __device__ int cta_svd_tall<T>(CMat, int, int, double*, i64, double*, double*, double*, \
                                          double*, int*, int*, double*, Mat, double*, Mat,        \
                                          double*);                                              \
  template __device__ int cta_svd_tall_blocked<T>(CMat, int, int, double*, double*, double*,      \
                                                  double*, double*, int*, int*, double*, Mat,     \
                                                  double*, Mat, double*, double*, double*,        \
                                                  double*, GemmSmem&, double*);
TTB_FACTOR_INSTANCE(true)
TTB_FACTOR_INSTANCE(false)

}  // namespace ttb
