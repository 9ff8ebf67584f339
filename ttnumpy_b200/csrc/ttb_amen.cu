// Whole AMEn solves on the device: one thread block per solve.
//
// The block runs the reference sweep (ttnumpy/solvers/amen.py:395-725) end
// to end with every rank decision taken on the device.  Cores and
// environments live in the solve's slab (global memory) in fixed-capacity
// slots sized for bonds up to rmax; per-step temporaries come from a stack
// at the top of the slab.  Dense factorisations run in a shared-memory pool
// when the matrix fits and fall back to the blocked global-memory variants
// otherwise.  All control flow is uniform across the block: every decision
// derives from block-wide reductions that all threads see identically.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>

#include "ttb200.h"
#include "ttb_device.cuh"
#include "ttb_factor.cuh"
#include "ttb_tc_block.cuh"

namespace ttb {
void count_launch();  // the library's launch counter (ttb200.cu)
}

namespace ttb_solve {

using namespace ttb;

constexpr int kD = 64;                 // most cores per train
// dynamic shared-memory pool (after the GEMM ring, whose size follows GBK)
constexpr int kPoolBytes = (GBK == 16 ? 160 : 114) * 1024;
constexpr int kRingBytes = GSTAGES * GSTAGE_D * 8;
constexpr i64 kPoolD = kPoolBytes / 8;
// fixed-size pool users: the two-level R-only QR's panel buffers and the
// blocked factorisations' reflector chunk
static_assert(kPoolD >= 3 * LNB2 * LNB2 + LNB * LNB2 + 2 * LNB * LNB, "pool too small");
static_assert(kPoolD >= (i64)LNB * YCH + 2 * LNB * LNB, "pool too small");
// direct solves held in the pool fit the registers, their multipliers the ring
static_assert(kPoolD < (kLuWhole + 1) * (kLuWhole + 2), "pool beyond lu_whole");
static_assert(lu_buf_doubles(kLuWhole) <= GSTAGES * GSTAGE_D, "ring too small");
// ring + pool + the kernel's static shared memory (about 9 KB) within 227 KB
static_assert(kRingBytes + kPoolBytes <= 216 * 1024, "dynamic shared memory over budget");
constexpr int kMaxRestarts = 4;        // common.py:230
constexpr double kShrink = 1e-2;       // common.py:233
constexpr int kMaxMinres = 2000;       // iteration cap of one MINRES call
constexpr double kEps = 2.220446049250313e-16;

enum { ST_OK = 0, ST_SINGULAR = -1, ST_SLAB = -3, ST_RANK = -4, ST_SETTINGS = -5, ST_TIME = -6,
       ST_TENSOR = -7 };
enum { F_A = 0, F_B, F_ZB, F_ZAX, F_XZ };

struct Sm {
  int n[kD], R[kD + 1], rb[kD + 1], xb[kD + 1], zb[kD + 1];
  i64 xo[kD], zo[kD];
  i64 eo[2][5][kD];
  double red[TTB_WARPS];
  int redi[TTB_WARPS];
  int ipiv[LNB];
  int flag;
  i64 stack0;
  uint64_t mbar[TC_STAGES];  // tensor-core pipeline (mixed precision)
  uint32_t tmem_slot;
};

struct Ctx {
  const ttb_amen_task_t* T;
  Sm* sm;
  double* slab;
  i64 cap, top;
  double* pool;
  double* ring;   // shared staging ring of the pipelined GEMM
  GemmSmem* gsm;  // its first stage, for the one-stage GEMM of the factorisations
  int d, rmax, K;
  int status;
  double flops;  // FP64 FLOPs of the block's GEMMs (2 m n k each)
  long long applies;      // one-site operator applications
  double check;           // debug: worst relative gap of the factorised term products
  double check_qr;        // debug: worst relative gap of the two-level R-only QR
  int n_qr2;              // debug: two-level R-only QRs checked
  long long cyc[8];       // SM cycles per phase (see PH_*)
  int mixed;              // 3xTF32 inner solves with float64 refinement
  TcState tc;             // the block's tensor-core pipeline (mixed only)
  int csize;              // blocks in the solve's cluster (1: the block alone)
  struct ClusterCmd* cmd; // the leader's command slot (csize > 1)
  double* vpart;          // this block's chunk sums of a shared vector pass
  double flops_tc;        // FLOPs of the tensor-core products
  long long refine;       // float64 refinement steps of the local solves
};

// the device-wide nanosecond timer (comparable across SMs)
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// phases timed with clock64 for the per-solve breakdown; PH_GEMM is not a
// phase of its own: it sums the cycles of every dense product (inside the
// other phases), to measure the block's GEMM rate
enum { PH_ENV = 0, PH_SOLVE, PH_ZCORE, PH_TRUNC, PH_GEMM, PH_RESID, PH_INIT, PH_N };

__device__ double* take(Ctx& c, i64 n) {
  n = (n + 31) & ~31LL;
  if (c.top + n > c.cap) {
    c.status = ST_SLAB;
    return nullptr;
  }
  double* p = c.slab + c.top;
  c.top += n;
  return p;
}

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------

__device__ void vfill(double* x, i64 n, double v) {
  for (i64 i = threadIdx.x; i < n; i += TTB_THREADS) x[i] = v;
}

__device__ void vcopy(double* y, const double* x, i64 n, double a = 1.0) {
  for (i64 i = threadIdx.x; i < n; i += TTB_THREADS) y[i] = a * x[i];
}

__device__ double vdot(const double* x, const double* y, i64 n, double* red) {
  double s = 0.0;
  for (i64 i = threadIdx.x; i < n; i += TTB_THREADS) s = fma(x[i], y[i], s);
  return block_sum(s, red);
}

__device__ double vnorm_diff(const double* x, const double* y, i64 n, double* red) {
  double s = 0.0;
  for (i64 i = threadIdx.x; i < n; i += TTB_THREADS) {
    double v = y ? x[i] - y[i] : x[i];
    s = fma(v, v, s);
  }
  return sqrt(block_sum(s, red));
}

// ---------------------------------------------------------------------------
// products shared out between the blocks of a cluster
// ---------------------------------------------------------------------------

// A solve may run on a cluster of blocks: block 0 (the leader) runs the
// whole solve as a lone block would, and posts each product large enough
// (a tiled GEMM of two or more output tiles, a sparse operator-core product)
// and the steps of an elimination (the local matrix, a panel's update) as a
// command in its shared memory; the other blocks read it over
// distributed shared memory and compute their share of the output tiles
// (tiles rank, rank + csize, ...) or rows, each exactly as the lone block
// computes it, so the solve's results do not depend on the cluster size.  A
// command is bracketed by two cluster barriers (posted; done); the leader
// ends every solve, normally or on an error, with the exit command.
enum { CL_EXIT = 0, CL_GEMM = 1, CL_SPMM = 2, CL_VEC = 3, CL_LOCAL = 4, CL_LU = 5,
       CL_QR = 6 };

// The element-wise passes of a MINRES iteration on long vectors run in
// kVecChunks fixed chunks, each reduced by one block-wide sum; the chunk
// partials are added in chunk order.  A lone block walks the chunks in turn,
// a cluster's blocks take chunks rank, rank + csize, ..., so the sums are
// the same bits either way.  Shorter vectors take one pass by one block.
constexpr int kVecChunks = 16;
constexpr i64 kVecChunkMin = 1 << 16;
enum { VP_SCALE = 0, VP_LANCZOS = 1, VP_RESID = 2, VP_UPDATE = 3 };
struct VecArgs {
  int op, first;
  double a0, a1, a2, a3;
  double *p0, *p1, *p2, *p3;
  i64 N;
};

// The pairs lo .. hi of a pass (and, with ``tail``, the odd last element);
// returns this thread's partial sum (its pairs in index order, then the
// tail).  Each thread loads kVecBatch pairs of every input before it stores
// any output, so that those loads are in flight together (a store may alias
// a later load, which keeps the compiler from reordering them itself).
//   VP_SCALE:   p0 = a0 p1                         (v = r2 / beta)
//   VP_LANCZOS: p0 -= a0 p1 unless first; sum p2 . p0   (y, r1, v)
//   VP_RESID:   p0 = p1 - a0 p2; sum p0 . p0        (r1 <- y - g r2)
//   VP_UPDATE:  p0 <- (p2 - a0 p0 - a1 p1) a2; p3 += a3 p0; sum p3 . p3
//               (w2 <- new w from v, w2, w; x += phi w)
constexpr int kVecBatch = 4;

template <int OP>
__device__ __forceinline__ double vpass_range(const VecArgs& q, i64 lo, i64 hi, bool tail) {
  double acc = 0.0;
  double2* P0 = reinterpret_cast<double2*>(q.p0);
  const double2* P1 = reinterpret_cast<const double2*>(q.p1);
  const double2* P2 = reinterpret_cast<const double2*>(q.p2);
  double2* P3 = reinterpret_cast<double2*>(q.p3);
  const bool upd = OP != VP_LANCZOS || !q.first;
  for (i64 i0 = lo + threadIdx.x; i0 < hi; i0 += kVecBatch * TTB_THREADS) {
    double2 u0[kVecBatch], u1[kVecBatch], u2[kVecBatch], u3[kVecBatch];
#pragma unroll
    for (int b = 0; b < kVecBatch; ++b) {
      const i64 i = i0 + (i64)b * TTB_THREADS;
      if (i >= hi) break;
      if (OP == VP_SCALE) {
        u1[b] = P1[i];
      } else if (OP == VP_LANCZOS) {
        u0[b] = P0[i];
        u2[b] = P2[i];
        if (upd) u1[b] = P1[i];
      } else if (OP == VP_RESID) {
        u1[b] = P1[i];
        u2[b] = P2[i];
      } else {
        u0[b] = P0[i];
        u1[b] = P1[i];
        u2[b] = P2[i];
        u3[b] = P3[i];
      }
    }
#pragma unroll
    for (int b = 0; b < kVecBatch; ++b) {
      const i64 i = i0 + (i64)b * TTB_THREADS;
      if (i >= hi) break;
      if (OP == VP_SCALE) {
        P0[i] = make_double2(q.a0 * u1[b].x, q.a0 * u1[b].y);
      } else if (OP == VP_LANCZOS) {
        double2 yy = u0[b];
        const double2 vv = u2[b];
        if (upd) {
          const double2 rr = u1[b];
          yy.x -= q.a0 * rr.x;
          yy.y -= q.a0 * rr.y;
          P0[i] = yy;
        }
        acc = fma(vv.x, yy.x, acc);
        acc = fma(vv.y, yy.y, acc);
      } else if (OP == VP_RESID) {
        const double2 yy = u1[b], rr = u2[b];
        const double2 nv = make_double2(yy.x - q.a0 * rr.x, yy.y - q.a0 * rr.y);
        P0[i] = nv;
        acc = fma(nv.x, nv.x, acc);
        acc = fma(nv.y, nv.y, acc);
      } else {
        const double2 a1 = u0[b], a2 = u1[b], vv = u2[b];
        double2 xx = u3[b];
        const double2 wn = make_double2((vv.x - q.a0 * a1.x - q.a1 * a2.x) * q.a2,
                                        (vv.y - q.a0 * a1.y - q.a1 * a2.y) * q.a2);
        P0[i] = wn;
        xx.x += q.a3 * wn.x;
        xx.y += q.a3 * wn.y;
        P3[i] = xx;
        acc = fma(xx.x, xx.x, acc);
        acc = fma(xx.y, xx.y, acc);
      }
    }
  }
  if (tail) {
    const i64 t = q.N - 1;
    if (OP == VP_SCALE) {
      q.p0[t] = q.a0 * q.p1[t];
    } else if (OP == VP_LANCZOS) {
      double yi = q.p0[t];
      if (upd) {
        yi -= q.a0 * q.p1[t];
        q.p0[t] = yi;
      }
      acc = fma(q.p2[t], yi, acc);
    } else if (OP == VP_RESID) {
      const double yi = q.p1[t] - q.a0 * q.p2[t];
      q.p0[t] = yi;
      acc = fma(yi, yi, acc);
    } else {
      const double wn = (q.p2[t] - q.a0 * q.p0[t] - q.a1 * q.p1[t]) * q.a2;
      q.p0[t] = wn;
      const double xi = q.p3[t] + q.a3 * wn;
      q.p3[t] = xi;
      acc = fma(xi, xi, acc);
    }
  }
  return acc;
}

// One chunk of a pass (pairs of doubles; the odd last element goes to the
// last chunk); returns the chunk's sum, the same on every thread.
__device__ __noinline__ double vpass_chunk(const VecArgs& q, int chunk, double* red) {
  const i64 N2 = q.N >> 1;
  const i64 cs = (N2 + kVecChunks - 1) / kVecChunks;
  const i64 lo = min((i64)chunk * cs, N2), hi = min(lo + cs, N2);
  const bool tail = (q.N & 1) && chunk == kVecChunks - 1 && threadIdx.x == 0;
  double acc;
  switch (q.op) {
    case VP_SCALE: acc = vpass_range<VP_SCALE>(q, lo, hi, tail); break;
    case VP_LANCZOS: acc = vpass_range<VP_LANCZOS>(q, lo, hi, tail); break;
    case VP_RESID: acc = vpass_range<VP_RESID>(q, lo, hi, tail); break;
    default: acc = vpass_range<VP_UPDATE>(q, lo, hi, tail); break;
  }
  return block_sum(acc, red);
}

struct LocalDims {  // of a local operator: bonds and modes
  int lt, lf, R, R2, n, m, rt, rf;
};

struct ClusterCmd {
  int op;
  VecArgs vec;
  const double* a;
  i64 a_rs, a_cs;
  const double* b;
  i64 b_rs, b_cs;
  double* c;
  i64 c_rs, c_cs, c_rs_hi, c_cs_hi;
  int c_rdiv, c_cdiv;
  int M, N, K;
  double alpha, beta;
  const int* sp_ptr;
  const int* sp_col;
  const double* sp_val;
  int sp_rows, sp_nnz, sp_cols;
  // CL_LOCAL: a, b, sp_val the left environment, core and right environment,
  // c the matrix; CL_LU: c the matrix, rhs, M unknowns, the panel at K; CL_QR:
  // a the M x N matrix, c its work area, rhs the reflectors' scalars
  LocalDims dim;
  double* rhs;
  int ipiv[LNB];
};
static_assert(sizeof(ClusterCmd) % 8 == 0 && sizeof(ClusterCmd) / 8 <= TTB_THREADS,
              "a command is read in one step");

__device__ __forceinline__ void cluster_barrier() {
  cooperative_groups::this_cluster().sync();  // arrive.release + wait.acquire
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
}

__device__ __forceinline__ OMat cmd_out(const ClusterCmd& q) {
  return OMat(q.c, q.c_rdiv, q.c_rs_hi, q.c_rs, q.c_cdiv, q.c_cs_hi, q.c_cs);
}

__device__ void cmd_set_out(ClusterCmd& q, const OMat& C) {
  q.c = C.p;
  q.c_rs = C.rs;
  q.c_cs = C.cs;
  q.c_rs_hi = C.rs_hi;
  q.c_cs_hi = C.cs_hi;
  q.c_rdiv = C.rdiv;
  q.c_cdiv = C.cdiv;
}

__device__ __noinline__ void gemm(Ctx& c, CMat A, CMat B, OMat C, int M, int N, int K,
                                  double alpha, double beta) {
  if (M <= 0 || N <= 0) return;
  c.flops += 2.0 * M * N * (double)K;
  const long long t0 = clock64();
  const int tiles = ((M + GBM - 1) / GBM) * ((N + GBN - 1) / GBN);
  // shared out only with every operand and the output in global memory (a
  // worker's shared-memory address names its own shared memory)
  if (c.csize > 1 && tiles >= 2 && !__isShared(C.p) && gemm_pipe_tiled(A, B, M, N, K)) {
    if (threadIdx.x == 0) {
      ClusterCmd& q = *c.cmd;
      q.op = CL_GEMM;
      q.a = A.p;
      q.a_rs = A.rs;
      q.a_cs = A.cs;
      q.b = B.p;
      q.b_rs = B.rs;
      q.b_cs = B.cs;
      cmd_set_out(q, C);
      q.M = M;
      q.N = N;
      q.K = K;
      q.alpha = alpha;
      q.beta = beta;
    }
    cluster_barrier();  // posted
    cta_gemm_pipe(A, B, C, M, N, K, alpha, beta, c.ring, 0, c.csize);
    cluster_barrier();  // every block's tiles are written
  } else {
    cta_gemm_pipe(A, B, C, M, N, K, alpha, beta, c.ring);
  }
  c.cyc[PH_GEMM] += clock64() - t0;
}

// The product on the tensor cores in 3xTF32 (``tc``) or in float64.
__device__ __forceinline__ void gemm_any(Ctx& c, bool tc, CMat A, CMat B, OMat C, int M, int N,
                                         int K, double alpha, double beta) {
  if (!tc || K <= 0) {
    gemm(c, A, B, C, M, N, K, alpha, beta);
    return;
  }
  if (M <= 0 || N <= 0) return;
  c.flops_tc += 2.0 * M * N * (double)K;
  const long long t0 = clock64();
  cta_gemm_tc(c.tc, A, B, C, M, N, K, alpha, beta);
  if (c.tc.failed) c.status = ST_TENSOR;
  c.cyc[PH_GEMM] += clock64() - t0;
}

// ---------------------------------------------------------------------------
// operator cores as sparse matrices
// ---------------------------------------------------------------------------

// A TTM core op (R, n, m, R2) viewed as a matrix over two of its index pairs
// and stored by rows in compressed form with its exact zeros dropped.  The
// cores of discretised operators are block-banded (identity, diagonal and
// tridiagonal n x m blocks, most (a, b) blocks zero), so a product with the
// core touches a few percent of the dense core's entries; the result is the
// dense product's up to the order in which the nonzero terms are summed.
//   SP_X: rows (k, b), columns (a, l) (the one-site operator's middle product)
//   SP_T: rows (l, b), columns (a, k) (left environment updates)
//   SP_P: rows (a, k), columns (l, b) (the core's own row-major layout)
enum { SP_X = 0, SP_T = 1, SP_P = 2 };
struct SpOp {
  const int* ptr;  // rows + 1 row starts
  const int* col;
  const double* val;
  int rows;  // 0: no sparse form (the dense product is used)
  int nnz;
  int cols;  // columns of the sparse form (rows of the dense operand)
};

// Cores below this many entries, or denser than one nonzero in kSpDensity,
// keep the dense product.
constexpr int kSpMinEntries = 4096;
constexpr int kSpDensity = 4;

// Stack doubles a sparse form of an R * n * m * R2 core may take.
__host__ __device__ constexpr i64 spop_doubles(i64 entries, i64 rows) {
  return (rows + 2) / 2 + 1 + 3 * (entries / kSpDensity + 1) / 2 + 96;
}

__device__ __forceinline__ i64 sp_index(int pairing, int row, int col, int R, int n, int m,
                                        int R2) {
  int a, k, l, b;
  if (pairing == SP_X) {
    k = row / R2, b = row % R2, a = col / m, l = col % m;
  } else if (pairing == SP_T) {
    l = row / R2, b = row % R2, a = col / n, k = col % n;
  } else {
    return (i64)row * m * R2 + col;
  }
  return (((i64)a * n + k) * m + l) * R2 + b;
}

// Builds the sparse form of ``op`` on the stack (left there for the caller's
// mark to release).  S.rows == 0 when the core is small or dense.
__device__ __noinline__ SpOp build_spop(Ctx& c, const double* op, int R, int n, int m, int R2,
                                        int pairing) {
  SpOp S{nullptr, nullptr, nullptr, 0, 0};
  const i64 entries = (i64)R * n * m * R2;
  if (entries < kSpMinEntries) return S;
  const int rows = pairing == SP_X ? n * R2 : pairing == SP_T ? m * R2 : R * n;
  const int cols = (int)(entries / rows);
  const i64 cap = entries / kSpDensity + 1;
  int* ptr = reinterpret_cast<int*>(take(c, (rows + 2) / 2 + 1));
  double* val = take(c, cap);
  int* col = reinterpret_cast<int*>(take(c, (cap + 1) / 2));
  if (c.status) return S;
  for (int r = threadIdx.x; r < rows; r += TTB_THREADS) {
    int cnt = 0;
    for (int q = 0; q < cols; ++q) cnt += (op[sp_index(pairing, r, q, R, n, m, R2)] != 0.0);
    ptr[r + 1] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ptr[0] = 0;
    for (int r = 0; r < rows; ++r) ptr[r + 1] += ptr[r];
  }
  __syncthreads();
  const int nnz = ptr[rows];
  if ((i64)nnz > cap - 1) return S;  // too dense: dense product
  for (int r = threadIdx.x; r < rows; r += TTB_THREADS) {
    int e = ptr[r];
    for (int q = 0; q < cols; ++q) {
      const double v = op[sp_index(pairing, r, q, R, n, m, R2)];
      if (v != 0.0) {
        val[e] = v;
        col[e] = q;
        ++e;
      }
    }
  }
  __syncthreads();
  S.ptr = ptr;
  S.col = col;
  S.val = val;
  S.rows = rows;
  S.nnz = nnz;
  S.cols = cols;
  return S;
}

// C[r, j] = alpha * sum_e val[e] B[col[e], j] + beta * C[r, j] for r < S.rows,
// j < N, with B[q, j] = B[q * b_rs + j * b_cs] and C addressed through an
// OMat.  Warps take rows, lanes take columns; each element sums its row's
// nonzero terms in column order, so the result does not depend on the
// schedule.  beta == 0 never reads C.
// The rows rank, rank + csize, ... of the product below (each row as the
// whole product computes it).
__device__ __noinline__ void spmm_rows(const int* ptr, const int* col, const double* val,
                                       int rows, const double* B, i64 b_rs, i64 b_cs, OMat C,
                                       int N, double alpha, double beta, int rank, int csize) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = rank + csize * warp; r < rows; r += csize * TTB_WARPS) {
    const int e0 = ptr[r], e1 = ptr[r + 1];
    double* crow = C.p + C.row(r);
    for (int j = lane; j < N; j += 32) {
      const double* bj = B + (i64)j * b_cs;
      double acc = 0.0;
      for (int e = e0; e < e1; ++e) acc = fma(val[e], bj[(i64)col[e] * b_rs], acc);
      double* cp = crow + C.col(j);
      double v = alpha * acc;
      if (beta != 0.0) v = fma(beta, *cp, v);
      *cp = v;
    }
  }
  __syncthreads();
}

// The product for an operand with unit column stride, staged through the
// block's shared pool: the sparse form (row starts, columns, values) is
// copied in once, then column tiles of B (all S.cols rows, 64 U columns)
// are copied in with cp.async and worked on from shared memory.  A warp
// takes one row at a time and walks its terms; each lane owns U pairs of
// adjacent columns (16-byte shared loads), so the term's value and column
// are loaded once for 2 U outputs.  Every output element sums its row's
// terms in column order, as spmm_rows does from global memory (the same
// bits).  Without the staging each term is a chain of dependent global
// loads (column index, then operand), which left the product bound by load
// latency.  The pool is free whenever a product runs: only the
// factorisations, the direct solves and the tensor-core stages use it, each
// within its own call (a cluster's other blocks use theirs for nothing
// else).
__device__ __forceinline__ int spmm_tile(int rows, int nnz, int cols) {
  const i64 meta = nnz + (nnz + 1) / 2 + (rows + 2) / 2;
  if (cols <= 0 || meta >= kPoolD) return 0;
  const i64 tw = (kPoolD - meta) / cols;
  return tw >= 128 ? 128 : tw >= 64 ? 64 : 0;
}

template <int U>
__device__ __forceinline__ void spmm_tile_rows(const double* tile, const double* val,
                                               const int* col, const int* ptr, int rows, int j0,
                                               int w, const OMat& C, double alpha, double beta) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  i64 coff[U][2];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int jj = 64 * u + 2 * lane + h;
      coff[u][h] = jj < w ? C.col(j0 + jj) : 0;
    }
  for (int r = warp; r < rows; r += TTB_WARPS) {
    const int e0 = ptr[r], e1 = ptr[r + 1];
    double2 acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) acc[u] = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int e = e0; e < e1; ++e) {
      const double v = val[e];
      const double* trow = tile + col[e] + 2 * lane;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        // columns at and beyond w hold stale values; their sums are dropped
        const double2 b = *reinterpret_cast<const double2*>(trow + 64 * u);
        acc[u].x = fma(v, b.x, acc[u].x);
        acc[u].y = fma(v, b.y, acc[u].y);
      }
    }
    double* crow = C.p + C.row(r);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (64 * u + 2 * lane + h >= w) continue;
        double* cp = crow + coff[u][h];
        double v = alpha * (h ? acc[u].y : acc[u].x);
        if (beta != 0.0) v = fma(beta, *cp, v);
        *cp = v;
      }
  }
}

// The column tiles rank, rank + csize, ... of the staged product (each of a
// cluster's blocks stages and computes its own tiles, all rows of each).
__device__ __noinline__ void spmm_staged(double* pool, const int* sptr, const int* scol,
                                         const double* sval, int rows, int nnz, int cols,
                                         const double* B, i64 b_rs, OMat C, int N, double alpha,
                                         double beta, int tw, int rank, int csize) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* tile = pool;  // cols x tw, rows 16-byte aligned
  double* val = tile + (i64)cols * tw;
  int* col = reinterpret_cast<int*>(val + nnz);
  int* ptr = reinterpret_cast<int*>(val + nnz + (nnz + 1) / 2);
  __syncthreads();  // the pool's previous user is done with it
  for (int e = threadIdx.x; e < nnz; e += TTB_THREADS) {
    val[e] = sval[e];
    col[e] = scol[e] * tw;
  }
  for (int r = threadIdx.x; r <= rows; r += TTB_THREADS) ptr[r] = sptr[r];
  for (int j0 = rank * tw; j0 < N; j0 += csize * tw) {
    const int w = min(tw, N - j0);
    for (int q = warp; q < cols; q += TTB_WARPS) {
      const double* src = B + (i64)q * b_rs + j0;
      double* dst = tile + (i64)q * tw;
      for (int jj = lane; jj < w; jj += 32) cp_async8(dst + jj, src + jj, true);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();  // the tile (and the sparse form) landed
    if (tw == 128)
      spmm_tile_rows<2>(tile, val, col, ptr, rows, j0, w, C, alpha, beta);
    else
      spmm_tile_rows<1>(tile, val, col, ptr, rows, j0, w, C, alpha, beta);
    __syncthreads();  // the tile's reads are done before the next copy
  }
  __syncthreads();  // (a block without tiles) the sparse form's copies are done
}

__device__ __noinline__ void spmm(Ctx& c, const SpOp& S, const double* B, i64 b_rs, i64 b_cs,
                                  OMat C, int N, double alpha, double beta) {
  c.flops += 2.0 * S.nnz * (double)N;
  const long long t0 = clock64();
  if (c.csize > 1 && S.rows >= 2 * TTB_WARPS && !__isShared(C.p) && !__isShared(B) &&
      !__isShared(S.val)) {
    if (threadIdx.x == 0) {
      ClusterCmd& q = *c.cmd;
      q.op = CL_SPMM;
      q.sp_ptr = S.ptr;
      q.sp_col = S.col;
      q.sp_val = S.val;
      q.sp_rows = S.rows;
      q.sp_nnz = S.nnz;
      q.sp_cols = S.cols;
      q.b = B;
      q.b_rs = b_rs;
      q.b_cs = b_cs;
      cmd_set_out(q, C);
      q.N = N;
      q.alpha = alpha;
      q.beta = beta;
    }
    cluster_barrier();
    const int tw = b_cs == 1 ? spmm_tile(S.rows, S.nnz, S.cols) : 0;
    if (tw > 0)
      spmm_staged(c.pool, S.ptr, S.col, S.val, S.rows, S.nnz, S.cols, B, b_rs, C, N, alpha, beta,
                  tw, 0, c.csize);
    else
      spmm_rows(S.ptr, S.col, S.val, S.rows, B, b_rs, b_cs, C, N, alpha, beta, 0, c.csize);
    cluster_barrier();
    c.cyc[PH_GEMM] += clock64() - t0;
    return;
  }
  const int tw = (b_cs == 1 && !__isShared(B) && !__isShared(C.p) && !__isShared(S.val))
                     ? spmm_tile(S.rows, S.nnz, S.cols)
                     : 0;
  if (tw > 0) {
    spmm_staged(c.pool, S.ptr, S.col, S.val, S.rows, S.nnz, S.cols, B, b_rs, C, N, alpha, beta,
                tw, 0, 1);
    c.cyc[PH_GEMM] += clock64() - t0;
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = warp; r < S.rows; r += TTB_WARPS) {
    const int e0 = S.ptr[r], e1 = S.ptr[r + 1];
    double* crow = C.p + C.row(r);
    for (int j = lane; j < N; j += 32) {
      const double* bj = B + (i64)j * b_cs;
      double acc = 0.0;
      for (int e = e0; e < e1; ++e) acc = fma(S.val[e], bj[(i64)S.col[e] * b_rs], acc);
      double* cp = crow + C.col(j);
      double v = alpha * acc;
      if (beta != 0.0) v = fma(beta, *cp, v);
      *cp = v;
    }
  }
  __syncthreads();
  c.cyc[PH_GEMM] += clock64() - t0;
}

// A chunked vector pass (see vpass_chunk); returns the sum, the same on
// every thread.  In a cluster the chunks are shared out and the leader
// reads the other blocks' chunk sums over distributed shared memory.
__device__ __noinline__ double vpass(Ctx& c, const VecArgs& q) {
  double* red = c.sm->red;
  if (c.csize <= 1) {
    double sum = 0.0;
    for (int k = 0; k < kVecChunks; ++k) sum += vpass_chunk(q, k, red);
    return sum;
  }
  if (threadIdx.x == 0) {
    c.cmd->op = CL_VEC;
    c.cmd->vec = q;
  }
  cluster_barrier();  // posted
  for (int k = 0; k < kVecChunks; k += c.csize) {
    const double v = vpass_chunk(q, k, red);
    if (threadIdx.x == 0) c.vpart[k] = v;
  }
  cluster_barrier();  // every chunk sum is written
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  double sum = 0.0;
  for (int k = 0; k < kVecChunks; ++k) {
    const double* part = cl.map_shared_rank(c.vpart, k % c.csize);
    sum += part[k];
  }
  return sum;
}

// ---------------------------------------------------------------------------
// environments (common.py:149-217), same GEMM chains as ttb_env_update
// ---------------------------------------------------------------------------

__device__ __noinline__ void env_step(Ctx& c, int side, const double* env, int t, int R, int f,
                         const double* frame, int n, int f2, const double* op, int m, int R2,
                         const double* target, int t2, double* out) {
  const i64 mark = c.top;
  if (op) {
    if (side == 0) {
      double* S1 = take(c, (i64)t * R * n * f2);
      double* S2 = take(c, (i64)t * m * R2 * f2);
      if (c.status) return;
      // S1[a, k, i, q] = sum_p env[i, a, p] frame[p, k, q]
      gemm(c, CMat{env, f, 1}, CMat{frame, (i64)n * f2, 1},
           OMat(S1, R, f2, (i64)n * t * f2, f2, (i64)t * f2, 1), t * R, n * f2, f, 1.0, 0.0);
      // S2[i, l, b, q] = sum_{a, k} op[a, k, l, b] S1[(a, k), (i, q)]
      const SpOp S = build_spop(c, op, R, n, m, R2, SP_T);
      if (c.status) return;
      const OMat o2(S2, kNoSplit, 0, f2, f2, (i64)m * R2 * f2, 1);
      if (S.rows)
        spmm(c, S, S1, (i64)t * f2, 1, o2, t * f2, 1.0, 0.0);
      else
        gemm(c, CMat{op, 1, (i64)m * R2}, CMat{S1, (i64)t * f2, 1}, o2, m * R2, t * f2, R * n,
             1.0, 0.0);
      gemm(c, CMat{target, 1, t2}, CMat{S2, (i64)R2 * f2, 1}, Mat{out, (i64)R2 * f2, 1}, t2,
           R2 * f2, t * m, 1.0, 0.0);
    } else {
      double* S1 = take(c, (i64)t2 * m * R * f);
      double* S2 = take(c, (i64)t2 * R2 * n * f);
      if (c.status) return;
      // S1[l, a, j, p] = sum_i target[j, l, i] env[i, a, p]
      gemm(c, CMat{target, t, 1}, CMat{env, (i64)R * f, 1},
           OMat(S1, m, f, (i64)R * t2 * f, f, (i64)t2 * f, 1), t2 * m, R * f, t, 1.0, 0.0);
      // S2[j, b, k, p] = sum_{l, a} op[b, k, l, a] S1[(l, a), (j, p)]
      const SpOp S = build_spop(c, op, R2, n, m, R, SP_P);
      if (c.status) return;
      const OMat o2(S2, kNoSplit, 0, f, f, (i64)R2 * n * f, 1);
      if (S.rows)
        spmm(c, S, S1, (i64)t2 * f, 1, o2, t2 * f, 1.0, 0.0);
      else
        gemm(c, CMat{op, (i64)m * R, 1}, CMat{S1, (i64)t2 * f, 1}, o2, R2 * n, t2 * f, m * R,
             1.0, 0.0);
      gemm(c, CMat{S2, (i64)n * f, 1}, CMat{frame, 1, (i64)n * f}, Mat{out, f2, 1}, t2 * R2, f2,
           n * f, 1.0, 0.0);
    }
  } else {
    if (side == 0) {
      double* S1 = take(c, (i64)t * n * f2);
      if (c.status) return;
      gemm(c, CMat{env, f, 1}, CMat{frame, (i64)n * f2, 1}, Mat{S1, (i64)n * f2, 1}, t, n * f2,
           f, 1.0, 0.0);
      gemm(c, CMat{target, 1, t2}, CMat{S1, f2, 1}, Mat{out, f2, 1}, t2, f2, t * n, 1.0, 0.0);
    } else {
      double* S1 = take(c, (i64)t2 * n * f);
      if (c.status) return;
      gemm(c, CMat{target, t, 1}, CMat{env, f, 1}, Mat{S1, f, 1}, t2 * n, f, t, 1.0, 0.0);
      gemm(c, CMat{S1, (i64)n * f, 1}, CMat{frame, 1, (i64)n * f}, Mat{out, f2, 1}, t2, f2,
           n * f, 1.0, 0.0);
    }
  }
  c.top = mark;
}

__device__ double* xcore(Ctx& c, int k) { return c.slab + c.sm->xo[k]; }
__device__ double* zcore(Ctx& c, int k) { return c.slab + c.sm->zo[k]; }
__device__ const double* acore(Ctx& c, int k) { return c.T->A + c.T->A_off[k]; }
__device__ const double* bcore(Ctx& c, int k) { return c.T->b + c.T->b_off[k]; }
__device__ double* envp(Ctx& c, int side, int fam, int k) { return c.slab + c.sm->eo[side][fam][k]; }

// Environment of family ``fam`` at site k from its neighbour (left: from
// k - 1, right: from k + 1); the boundary ones are ones.
__device__ __noinline__ void build_env(Ctx& c, int side, int fam, int k) {
  Sm* s = c.sm;
  const int d = c.d;
  double* out = envp(c, side, fam, k);
  if ((side == 0 && k == 0) || (side == 1 && k == d - 1)) {
    if (threadIdx.x == 0) out[0] = 1.0;
    __syncthreads();
    return;
  }
  const int src = side == 0 ? k - 1 : k + 1;     // core contracted
  const int pin = side == 0 ? k - 1 : k + 2;     // bond of the previous env
  const int pout = side == 0 ? k : k + 1;        // bond of the new env
  const int psrc = side == 0 ? k - 1 : k + 1;    // previous env index
  const double* prev = envp(c, side, fam, psrc);
  const int n = s->n[src];
  const double* xc = xcore(c, src);
  const double* zc = zcore(c, src);
  const double* bc = bcore(c, src);
  const double* ac = acore(c, src);
  switch (fam) {
    case F_A:
      env_step(c, side, prev, s->xb[pin], s->R[pin], s->xb[pin], xc, n, s->xb[pout], ac, n,
               s->R[pout], xc, s->xb[pout], out);
      break;
    case F_B:
      env_step(c, side, prev, s->rb[pin], 1, s->xb[pin], xc, n, s->xb[pout], nullptr, n, 1, bc,
               s->rb[pout], out);
      break;
    case F_ZB:
      env_step(c, side, prev, s->rb[pin], 1, s->zb[pin], zc, n, s->zb[pout], nullptr, n, 1, bc,
               s->rb[pout], out);
      break;
    case F_ZAX:
      env_step(c, side, prev, s->xb[pin], s->R[pin], s->zb[pin], zc, n, s->zb[pout], ac, n,
               s->R[pout], xc, s->xb[pout], out);
      break;
    default:
      env_step(c, side, prev, s->zb[pin], 1, s->xb[pin], xc, n, s->xb[pout], nullptr, n, 1, zc,
               s->zb[pout], out);
      break;
  }
}

// ---------------------------------------------------------------------------
// one-site local operator and projections
// ---------------------------------------------------------------------------

struct LocalOp {
  const double* left;
  const double* op;
  const double* right;
  const double* opP;     // op re-laid out as [a, l, k, b] (permute_op)
  const double* rightP;  // right re-laid out as [b, p, q] (permute_op)
  SpOp sx, sp;           // op's sparse forms SP_X and SP_P (permute_op), if any
  int lt, lf, R, R2, n, m, rt, rf;

  __device__ LocalDims dims() const { return LocalDims{lt, lf, R, R2, n, m, rt, rf}; }
};

__device__ LocalOp local_A(Ctx& c, int k) {
  Sm* s = c.sm;
  LocalOp L;
  L.left = envp(c, 0, F_A, k);
  L.right = envp(c, 1, F_A, k);
  L.op = acore(c, k);
  L.lt = L.lf = s->xb[k];
  L.rt = L.rf = s->xb[k + 1];
  L.R = s->R[k];
  L.R2 = s->R[k + 1];
  L.n = L.m = s->n[k];
  L.opP = L.rightP = nullptr;
  L.sx.rows = L.sp.rows = 0;
  return L;
}

// The operator core and the right environment re-laid out (on the stack,
// released with the caller's mark) so that every product of apply() and of
// the forward rank-one terms is one GEMM over plain strides:
// opP[a, l, k, b] = op[a, k, l, b] and rightP[b, p, q] = right[p, b, q].
__device__ __noinline__ void permute_op(Ctx& c, LocalOp& L) {
  const int R = L.R, R2 = L.R2, n = L.n, m = L.m, rt = L.rt, rf = L.rf;
  const i64 no = (i64)R * m * n * R2, nr = (i64)R2 * rt * rf;
  double* opP = take(c, no);
  double* rightP = take(c, nr);
  if (c.status) return;
  for (i64 e = threadIdx.x; e < no; e += TTB_THREADS) {
    const int b = (int)(e % R2);
    const int k = (int)((e / R2) % n);
    const int l = (int)((e / ((i64)R2 * n)) % m);
    const int a = (int)(e / ((i64)R2 * n * m));
    opP[e] = L.op[(((i64)a * n + k) * m + l) * R2 + b];
  }
  for (i64 e = threadIdx.x; e < nr; e += TTB_THREADS) {
    const int q = (int)(e % rf);
    const int pp = (int)((e / rf) % rt);
    const int b = (int)(e / ((i64)rf * rt));
    rightP[e] = L.right[((i64)pp * R2 + b) * rf + q];
  }
  __syncthreads();
  L.opP = opP;
  L.rightP = rightP;
  L.sx = build_spop(c, L.op, R, n, m, R2, SP_X);
  if (c.status) return;
  L.sp = L.sx.rows ? build_spop(c, L.op, R, n, m, R2, SP_P) : SpOp{nullptr, nullptr, nullptr, 0, 0};
}

// y = alpha * B x + beta * y for ``cols`` vectors (one_site.py:78-115) as
// three GEMMs per vector, contracting the left bond, then the operator's
// (bond, mode) pair, then the right bond; the first two write their results
// permuted (split-index outputs) so that each next product reads plain
// strides.  Needs permute_op(L).
__device__ __noinline__ void apply(Ctx& c, const LocalOp& L, const double* x, double* y, int cols,
                      double alpha, double beta, bool tc = false) {
  const int lt = L.lt, lf = L.lf, R = L.R, R2 = L.R2, n = L.n, m = L.m, rt = L.rt, rf = L.rf;
  const i64 mark = c.top;
  c.applies += cols;
  double* W1 = take(c, (i64)R * m * lf * rt);   // W1[a, l, j, p]
  double* W2 = take(c, (i64)lf * n * R2 * rt);  // W2[j, k, b, p]
  if (c.status) return;
  for (int cc = 0; cc < cols; ++cc) {
    const double* xc = x + (i64)cc * lt * m * rt;
    double* yc = y + (i64)cc * lf * n * rf;
    // W1[(a, j), (l, p)] = sum_i left[i, a, j] x[i, l, p]
    gemm_any(c, tc, CMat{L.left, 1, (i64)R * lf}, CMat{xc, (i64)m * rt, 1},
             OMat(W1, lf, (i64)m * lf * rt, rt, rt, (i64)lf * rt, 1), R * lf, m * rt, lt, 1.0,
             0.0);
    // W2[(k, b), (j, p)] = sum_{a, l} op[a, k, l, b] W1[(a, l), (j, p)]
    const OMat o2(W2, kNoSplit, 0, rt, rt, (i64)n * R2 * rt, 1);
    if (L.sx.rows)
      spmm(c, L.sx, W1, (i64)lf * rt, 1, o2, lf * rt, 1.0, 0.0);
    else
      gemm_any(c, tc, CMat{L.opP, 1, (i64)n * R2}, CMat{W1, (i64)lf * rt, 1}, o2, n * R2,
               lf * rt, R * m, 1.0, 0.0);
    // y[(j, k), q] = alpha * sum_{b, p} W2[(j, k), (b, p)] right[p, b, q] + beta * y
    gemm_any(c, tc, CMat{W2, (i64)R2 * rt, 1}, CMat{L.rightP, rf, 1}, Mat{yc, rf, 1}, lf * n, rf,
             R2 * rt, alpha, beta);
    if (c.status) break;
  }
  c.top = mark;
}

// out (i, n, l) = alpha * Lb^T core Rb + beta * out (local_rhs_one_site)
__device__ __noinline__ void project(Ctx& c, const double* left, int a, int i, const double* core, int n,
                        int cc, const double* right, int l, double* out, double alpha,
                        double beta) {
  const i64 mark = c.top;
  double* W = take(c, (i64)a * n * l);
  if (c.status) return;
  gemm(c, CMat{core, cc, 1}, CMat{right, l, 1}, Mat{W, l, 1}, a * n, l, cc, 1.0, 0.0);
  gemm(c, CMat{left, 1, i}, CMat{W, (i64)n * l, 1}, Mat{out, (i64)n * l, 1}, i, n * l, a, alpha,
       beta);
  c.top = mark;
}

// ---------------------------------------------------------------------------
// factorisations with the shared pool or the blocked global variants
// ---------------------------------------------------------------------------

// Rows from which a cluster shares the residual norm's factorisations; below,
// the two barriers a column cost as much as a lone block's pass over it.  On
// eight blocks each, from 256, 1024 and 2048 rows on, and never: eight mode-32
// diffusion solves (d = 4) 471, 471, 489 and 489 ms, one of d = 6 and mode 16
// 337, 338, 350 and 386, eight of d = 5 and mode 8 72, 74, 74 and 74.
constexpr int kQrShare = 1024;

// Economic QR of the m x k view A: Q (m x p) and R (p x k) strided outputs.
__device__ __noinline__ void qr(Ctx& c, CMat A, int m, int k, Mat Q, Mat R) {
  const int p = min(m, k);
  if ((i64)m * k + p <= kPoolD) {
    cta_qr<false>(A, m, k, c.pool, m, c.pool + (i64)m * k, Q, R, c.sm->red);
    return;
  }
  const i64 mark = c.top;
  double* W = take(c, (i64)m * k + p);
  if (c.status) return;
  if (!Q.p && p > LNB2 && m >= 4 * k) {
    // R only of a tall matrix (the residual norm sweep): two-level blocking
    const bool shared = c.csize > 1 && m >= kQrShare && !__isShared(A.p);
    if (shared) {
      if (threadIdx.x == 0) {
        ClusterCmd& q = *c.cmd;
        q.op = CL_QR;
        q.a = A.p;
        q.a_rs = A.rs;
        q.a_cs = A.cs;
        q.M = m;
        q.N = k;
        q.c = W;
        q.rhs = W + (i64)m * k;
      }
      cluster_barrier();
    }
    cta_qr_r_blocked2(A, m, k, W, W + (i64)m * k, R, c.pool, c.sm->red, c.ring, 0,
                      shared ? c.csize : 1);
    if (shared) cluster_barrier();
    if (c.T->debug & 1) {
      // the one-level blocked factorisation of the same matrix, compared
      double* R1 = take(c, (i64)p * k);
      if (c.status) return;
      cta_qr_blocked<false>(A, m, k, W, W + (i64)m * k, Mat{nullptr, 0, 0}, Mat{R1, k, 1}, c.pool,
                     c.pool + (i64)LNB * YCH, c.pool + (i64)LNB * YCH + LNB * LNB, c.sm->red,
                     *c.gsm, nullptr);
      double dsq = 0.0, rsq = 0.0;
      for (i64 e = threadIdx.x; e < (i64)p * k; e += TTB_THREADS) {
        const int i = (int)(e / k), j = (int)(e % k);
        const double a = R(i, j), b = R1[e];
        dsq = fma(a - b, a - b, dsq);
        rsq = fma(b, b, rsq);
      }
      dsq = block_sum(dsq, c.sm->red);
      rsq = block_sum(rsq, c.sm->red);
      c.check_qr = fmax(c.check_qr, rsq > 0.0 ? sqrt(dsq / rsq) : sqrt(dsq));
      c.n_qr2 += 1;
    }
    c.top = mark;
    return;
  }
  double* Y = c.pool;
  double* G = Y + (i64)LNB * YCH;
  double* Tm = G + LNB * LNB;
  cta_qr_blocked<false>(A, m, k, W, W + (i64)m * k, Q, R, Y, G, Tm, c.sm->red, *c.gsm,
                        c.ring);
  c.top = mark;
}

// Thin SVD of the m x k view A into U (m x p), S (p), Vh (p x k).
__device__ __noinline__ void svd(Ctx& c, CMat A, int m, int k, Mat U, double* S, Mat Vh) {
  const bool tall = m >= k;
  const int M = tall ? m : k, K = tall ? k : m;
  CMat At = tall ? A : CMat{A.p, A.cs, A.rs};
  Mat Ut = tall ? U : Mat{Vh.p, Vh.cs, Vh.rs};
  Mat Vt = tall ? Vh : Mat{U.p, U.cs, U.rs};
  const i64 need = (i64)M * K + 2 * (i64)K * K + 3 * (i64)K + 2;
  const i64 mark = c.top;
  double* base;
  const bool in_pool = need <= kPoolD;
  if (in_pool) {
    base = c.pool;
  } else {
    base = take(c, need);
    if (c.status) return;
  }
  double* W = base;
  double* tau = W + (i64)M * K;
  double* Bsq = tau + K;
  double* V = Bsq + (i64)K * K;
  double* sv = V + (i64)K * K;
  int* order = reinterpret_cast<int*>(sv + K);
  int* flag = reinterpret_cast<int*>(sv + 2 * K);
  if (in_pool) {
    cta_svd_tall<false>(At, M, K, W, M, tau, Bsq, V, sv, order, flag, nullptr, Ut, S, Vt, c.sm->red);
  } else {
    double* Y = c.pool;
    double* G = Y + (i64)LNB * YCH;
    double* Tm = G + LNB * LNB;
    cta_svd_tall_blocked<false>(At, M, K, W, tau, Bsq, V, sv, order, flag, nullptr, Ut, S, Vt, Y, G, Tm,
                         c.sm->red, *c.gsm, c.ring);
  }
  c.top = mark;
}

// ---------------------------------------------------------------------------
// local solves
// ---------------------------------------------------------------------------

// Explicit local matrix, column major: the items rank, rank + size, ... of
// the blocks of a cluster.  An item is a row (j, kr, nf) and the part (l, mt)
// of a column: the operator core times the right environment gives one number
// per left operator bond, kept in registers while the item's lt columns (i, l,
// mt) are formed.  Consecutive threads take consecutive rows.  (A thread
// walking a whole row re-read core and environment for every entry and left
// the threads past N idle: as long as the elimination itself on the QTT
// systems.)
__device__ __noinline__ void form_local(const double* lenv, const double* core, const double* renv,
                                        const LocalDims& L, double* W, int rank, int size) {
  const int Nn = L.lf * L.n * L.rf;
  constexpr int kRegs = 8;  // left operator bonds held in registers at a time
  for (TableWalk e(rank * TTB_THREADS + threadIdx.x, size * TTB_THREADS, Nn); e.row < L.m * L.rt;
       e.next()) {
    const int row = e.at, mt = e.row % L.rt, l = e.row / L.rt;
    const int nf = row % L.rf, kr = (row / L.rf) % L.n, j = row / (L.rf * L.n);
    for (int a0 = 0; a0 < L.R; a0 += kRegs) {
      double t[kRegs];
#pragma unroll
      for (int a = 0; a < kRegs; ++a) {
        t[a] = 0.0;
        if (a0 + a >= L.R) continue;
        const double* op = core + (((i64)(a0 + a) * L.n + kr) * L.m + l) * L.R2;
        const double* right = renv + (i64)mt * L.R2 * L.rf + nf;
        for (int bb = 0; bb < L.R2; ++bb) t[a] = fma(op[bb], right[(i64)bb * L.rf], t[a]);
      }
      const double* left = lenv + (i64)a0 * L.lf + j;
      double* w = W + row + ((i64)l * L.rt + mt) * Nn;
      for (int i = 0; i < L.lt; ++i) {
        double acc = a0 ? *w : 0.0;
#pragma unroll
        for (int a = 0; a < kRegs; ++a) {
          if (a0 + a >= L.R) continue;
          const double la = left[(i64)a * L.lf];
          if (la != 0.0) acc = fma(la, t[a], acc);
        }
        *w = acc;
        left += (i64)L.R * L.lf;
        w += (i64)L.m * L.rt * Nn;
      }
    }
  }
}

// Trailing columns from which a panel's update is worth two cluster barriers
// and a read of the panel by every block: from 32, 96, 192 and 384 on, eight
// mode-32 diffusion solves take 471, 471, 472 and 483 ms, eight of d = 5 and
// mode 8 74.3, 74.2, 74.6 and 76.8.
constexpr int kLuShare = 96;

// cta_gepp_blocked with the strips of each panel's update shared out; W and b
// in global memory, n <= kLuRows, every entry as a lone block computes it.
__device__ __noinline__ int cluster_gepp(Ctx& c, double* W, double* b, int n) {
  ClusterCmd& q = *c.cmd;
  for (int j0 = 0; j0 < n; j0 += LNB) {
    if (const int info = cta_gepp_panel(W, n, n, j0, c.pool, q.ipiv)) return info;
    if (n - j0 - LNB < kLuShare) {
      cta_gepp_update(W, n, b, n, j0, c.pool, q.ipiv, false, 0, 1);
      continue;
    }
    if (threadIdx.x == 0) {
      q.op = CL_LU;
      q.c = W;
      q.rhs = b;
      q.M = n;
      q.K = j0;
    }
    cluster_barrier();  // posted
    cta_gepp_update(W, n, b, n, j0, c.pool, q.ipiv, false, 0, c.csize);
    cluster_barrier();  // every strip is written
  }
  cta_back_substitute(W, n, b, n);
  return 0;
}

// Explicit local matrix (column major, n x n) and GEPP solve; u <- solution.
__device__ __noinline__ void direct_solve(Ctx& c, const LocalOp& L, const double* b, double* u) {
  const i64 N = (i64)L.lf * L.n * L.rf;
  const i64 mark = c.top;
  Sm* s = c.sm;
  double* W;
  double* panel = c.pool;  // the blocked elimination's panel (N x LNB)
  const bool small = N * N + N <= kPoolD;  // in the pool and in registers
  if (small) {
    W = c.pool;
  } else {
    W = take(c, N * N);
    if (lu_panel_doubles((int)N) > kPoolD) panel = take(c, N * LNB);  // in the slab
    if (c.status) return;
  }
  // A cluster forms and eliminates the matrices of the slab together (a
  // quarter of a mode-32 diffusion solve while the leader did it alone: eight
  // such solves on eight blocks each 739 -> 626 ms).
  const bool shared = c.csize > 1 && !small && N <= kLuRows && panel == c.pool;
  if (shared) {
    if (threadIdx.x == 0) {
      ClusterCmd& q = *c.cmd;
      q.op = CL_LOCAL;
      q.a = L.left;
      q.b = L.op;
      q.sp_val = L.right;
      q.c = W;
      q.dim = L.dims();
    }
    cluster_barrier();
  }
  form_local(L.left, L.op, L.right, L.dims(), W, 0, shared ? c.csize : 1);
  if (shared) cluster_barrier();
  vcopy(u, b, N);
  __syncthreads();
  int info;
  if (small)
    info = cta_gepp_solve(W, N, u, (int)N, c.ring);
  else if (shared)
    info = cluster_gepp(c, W, u, (int)N);
  else
    info = cta_gepp_blocked(W, N, u, (int)N, panel, s->red, s->redi, s->ipiv, *c.gsm, c.ring);
  __syncthreads();
  if (info != 0) c.status = ST_SINGULAR;
  c.top = mark;
}

// MINRES, SciPy 1.18.1's algorithm and stopping rules (Paige & Saunders);
// x holds the initial guess (warm) on entry and the iterate on exit.
__device__ __noinline__ void minres(Ctx& c, const LocalOp& L, const double* b, double* x, i64 N, double rtol,
                       int maxit, bool warm, bool tc = false) {
  double* red = c.sm->red;
  const i64 mark = c.top;
  // vectors padded to an even length, so that each starts 16-byte aligned
  // and the passes below read and write pairs of doubles
  const i64 Np = (N + 1) & ~1LL, N2 = N >> 1;
  const bool odd = (N & 1) != 0;
  double* buf = take(c, 6 * Np);
  if (c.status) return;
  // r1, r2 and w, w2 rotate by pointer (SciPy's r1 <- r2, r2 <- y and
  // w1 <- w2, w2 <- w copies); y is the operator's output, and after each
  // iteration its value is r2's
  double* r1 = buf;
  double* r2 = buf + Np;
  double* y = buf + 2 * Np;
  double* v = buf + 3 * Np;
  double* w = buf + 4 * Np;
  double* w2 = buf + 5 * Np;
  if (warm) {
    apply(c, L, x, y, 1, 1.0, 0.0, tc);
    for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) r1[i] = b[i] - y[i];
  } else {
    vfill(x, N, 0.0);
    vcopy(r1, b, N);
  }
  __syncthreads();
  const double beta1sq = vdot(r1, r1, N, red);
  const double bnorm = sqrt(vdot(b, b, N, red));
  if (beta1sq == 0.0 || bnorm == 0.0) {
    if (bnorm == 0.0) vcopy(x, b, N);
    __syncthreads();
    c.top = mark;
    return;
  }
  const double beta1 = sqrt(beta1sq);
  double oldb = 0.0, beta = beta1, dbar = 0.0, epsln = 0.0, phibar = beta1, rhs1 = beta1,
         rhs2 = 0.0, tnorm2 = 0.0, gmax = 0.0, gmin = DBL_MAX, cs = -1.0, sn = 0.0;
  vfill(w, N, 0.0);
  vfill(w2, N, 0.0);
  vcopy(r2, r1, N);
  vcopy(y, r1, N);
  __syncthreads();
  // the odd last element goes to thread 0, after its pairs
  const bool tail = odd && threadIdx.x == 0;
  // long vectors: the chunked passes a cluster shares out (vpass)
  const bool chunked = N >= kVecChunkMin;
  int istop = 0;
  for (int itn = 1; itn <= maxit; ++itn) {
    const double s = 1.0 / beta;
    if (chunked)
      vpass(c, VecArgs{VP_SCALE, 0, s, 0.0, 0.0, 0.0, v, r2, nullptr, nullptr, N});
    else
      vpass_range<VP_SCALE>(VecArgs{VP_SCALE, 0, s, 0.0, 0.0, 0.0, v, r2, nullptr, nullptr, N}, 0,
                            N2, tail);
    __syncthreads();
    apply(c, L, v, y, 1, 1.0, 0.0, tc);
    if (c.status) return;
    // y -= (beta / oldb) r1 and alfa = v . y in one pass
    const VecArgs lz{VP_LANCZOS, itn == 1, itn >= 2 ? beta / oldb : 0.0, 0.0, 0.0, 0.0,
                     y, r1, v, nullptr, N};
    const double alfa =
        chunked ? vpass(c, lz) : block_sum(vpass_range<VP_LANCZOS>(lz, 0, N2, tail), red);
    const double g = alfa / beta;
    // r1 <- y - g r2 (the new r2) and its squared norm
    const VecArgs rs{VP_RESID, 0, g, 0.0, 0.0, 0.0, r1, y, r2, nullptr, N};
    const double psum =
        chunked ? vpass(c, rs) : block_sum(vpass_range<VP_RESID>(rs, 0, N2, tail), red);
    {
      double* t = r1;
      r1 = r2;
      r2 = t;
    }
    oldb = beta;
    beta = sqrt(psum);
    tnorm2 += alfa * alfa + oldb * oldb + beta * beta;
    if (itn == 1 && beta / beta1 <= 10.0 * kEps) istop = -1;
    const double oldeps = epsln;
    const double delta = cs * dbar + sn * alfa;
    const double gbar = sn * dbar - cs * alfa;
    epsln = sn * beta;
    dbar = -cs * beta;
    const double root = hypot(gbar, dbar);
    double gamma = fmax(hypot(gbar, beta), kEps);
    cs = gbar / gamma;
    sn = beta / gamma;
    const double phi = cs * phibar;
    phibar = sn * phibar;
    const double denom = 1.0 / gamma;
    // the new w (into w2's buffer) and x += phi w, with x's squared norm
    const VecArgs up{VP_UPDATE, 0, oldeps, delta, denom, phi, w2, w, v, x, N};
    const double xsum =
        chunked ? vpass(c, up) : block_sum(vpass_range<VP_UPDATE>(up, 0, N2, tail), red);
    {
      double* t = w2;
      w2 = w;
      w = t;
    }
    gmax = fmax(gmax, gamma);
    gmin = fmin(gmin, gamma);
    const double z = rhs1 / gamma;
    rhs1 = rhs2 - delta * z;
    rhs2 = -epsln * z;
    const double Anorm = sqrt(tnorm2);
    const double ynorm = sqrt(xsum);
    const double epsx = Anorm * ynorm * kEps;
    const double rnorm = phibar;
    const double test1 = (ynorm == 0.0 || Anorm == 0.0) ? INFINITY : rnorm / (Anorm * ynorm);
    const double test2 = (Anorm == 0.0) ? INFINITY : root / Anorm;
    const double Acond = gmax / gmin;
    if (istop == 0) {
      if (1.0 + test2 <= 1.0) istop = 2;
      if (1.0 + test1 <= 1.0) istop = 1;
      if (itn >= maxit) istop = 6;
      if (Acond >= 0.1 / kEps) istop = 4;
      if (epsx >= beta1) istop = 3;
      if (test2 <= rtol) istop = 2;
      if (test1 <= rtol) istop = 1;
    }
    if (istop != 0) break;
  }
  __syncthreads();
  c.top = mark;
}

// Restarted GMRES with SciPy 1.18.1's gmres control flow (restart 20,
// modified Gram-Schmidt Arnoldi, LAPACK dlartg Givens rotations, the
// presid / ptol inner test and the pmf update of ptol between cycles), as
// ttb_gmres runs it in separate launches: x holds the initial guess (warm)
// on entry and the iterate on exit.  At most ``maxcycles`` restart cycles
// (SciPy's default is 10 N; a block solving alone on one SM is bounded
// tighter, as MINRES is).
constexpr int kRestart = 20;

__device__ __forceinline__ void givens(double f, double g, double& cs, double& sn, double& r) {
  if (g == 0.0) {
    cs = 1.0;
    sn = 0.0;
    r = f;
    return;
  }
  if (f == 0.0) {
    cs = 0.0;
    sn = (g >= 0.0) ? 1.0 : -1.0;
    r = fabs(g);
    return;
  }
  const double dd = sqrt(f * f + g * g);
  cs = fabs(f) / dd;
  r = copysign(dd, f);
  sn = g / r;
}

__device__ __noinline__ void gmres(Ctx& c, const LocalOp& L, const double* b, double* x, i64 N,
                                   double rtol, int maxcycles, bool warm) {
  double* red = c.sm->red;
  const i64 mark = c.top;
  const int rs = (int)min((i64)kRestart, N);
  const int R1 = rs + 1;
  const i64 Np = (N + 31) & ~31LL;
  double* V = take(c, (i64)R1 * Np);
  double* w = take(c, Np);
  double* r = take(c, Np);
  double* h = take(c, (i64)rs * R1);  // h[col * R1 + row]
  double* giv = take(c, 2 * rs);
  double* S = take(c, R1);
  double* st = take(c, R1 + 4);       // y of the update, then presid, flags
  if (c.status) return;
  const double eps = kEps;
  if (warm) {
    apply(c, L, x, w, 1, 1.0, 0.0);
    if (c.status) return;
  }
  double sb = 0.0, sr = 0.0;
  for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) {
    const double bv = b[i];
    const double rv = warm ? bv - w[i] : bv;
    if (!warm) x[i] = 0.0;
    r[i] = rv;
    sb = fma(bv, bv, sb);
    sr = fma(rv, rv, sr);
  }
  const double bnrm2 = sqrt(block_sum(sb, red));
  const double rn0 = sqrt(block_sum(sr, red));
  if (bnrm2 == 0.0) {
    vcopy(x, b, N);
    __syncthreads();
    c.top = mark;
    return;
  }
  const double atol = fmax(0.0, rtol * bnrm2);
  double pmf = 1.0, ptol = bnrm2 * fmin(1.0, atol / bnrm2);
  if (rn0 < atol) {
    c.top = mark;
    return;
  }
  for (int cycle = 0; cycle < maxcycles; ++cycle) {
    // v0 = r / ||r||, S = [||r||, 0, ...]
    const double rr = sqrt(vdot(r, r, N, red));
    vcopy(V, r, N, 1.0 / rr);
    for (int i = threadIdx.x; i <= rs; i += TTB_THREADS) S[i] = (i == 0) ? rr : 0.0;
    __syncthreads();
    int col_end = rs - 1;
    bool brk = false;
    double presid = 0.0;
    for (int col = 0; col < rs; ++col) {
      apply(c, L, V + (i64)col * Np, w, 1, 1.0, 0.0);
      if (c.status) return;
      double* hc = h + (i64)col * R1;
      const double h0 = sqrt(vdot(w, w, N, red));
      for (int k = 0; k <= col; ++k) {
        const double* vk = V + (i64)k * Np;
        const double dk = vdot(vk, w, N, red);
        if (threadIdx.x == 0) hc[k] = dk;
        for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) w[i] -= dk * vk[i];
        __syncthreads();
      }
      const double h1 = sqrt(vdot(w, w, N, red));
      brk = h1 <= eps * h0;
      vcopy(V + (i64)(col + 1) * Np, w, N, brk ? 1.0 : 1.0 / h1);
      if (threadIdx.x == 0) {
        hc[col + 1] = brk ? 0.0 : h1;
        for (int k = 0; k < col; ++k) {
          const double cs = giv[2 * k], sn = giv[2 * k + 1];
          const double n0 = hc[k], n1 = hc[k + 1];
          hc[k] = cs * n0 + sn * n1;
          hc[k + 1] = -sn * n0 + cs * n1;
        }
        double cs, sn, mag;
        givens(hc[col], hc[col + 1], cs, sn, mag);
        giv[2 * col] = cs;
        giv[2 * col + 1] = sn;
        hc[col] = mag;
        hc[col + 1] = 0.0;
        const double tmp = -sn * S[col];
        S[col] = cs * S[col];
        S[col + 1] = tmp;
        st[R1] = fabs(tmp);
      }
      __syncthreads();
      presid = st[R1];
      if (presid <= ptol || brk || col == rs - 1) {
        col_end = col;
        break;
      }
    }
    // back substitution on the rotated Hessenberg factor; x += y V
    if (threadIdx.x == 0) {
      double* y = st;
      const int cl = col_end;
      if (h[(i64)cl * R1 + cl] == 0.0) S[cl] = 0.0;
      for (int k = 0; k <= cl; ++k) y[k] = S[k];
      for (int k = cl; k > 0; --k) {
        if (y[k] != 0.0) {
          y[k] /= h[(i64)k * R1 + k];
          const double t = y[k];
          for (int i = 0; i < k; ++i) y[i] -= t * h[(i64)k * R1 + i];
        }
      }
      if (y[0] != 0.0) y[0] /= h[0];
    }
    __syncthreads();
    for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) {
      double acc = 0.0;
      for (int k = 0; k <= col_end; ++k) acc = fma(st[k], V[(i64)k * Np + i], acc);
      x[i] += acc;
    }
    __syncthreads();
    // r = b - A x; the outer convergence test and the ptol update
    apply(c, L, x, w, 1, 1.0, 0.0);
    if (c.status) return;
    double s2 = 0.0;
    for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) {
      const double rv = b[i] - w[i];
      r[i] = rv;
      s2 = fma(rv, rv, s2);
    }
    const double rnorm = sqrt(block_sum(s2, red));
    if (rnorm <= atol || brk) break;
    if (presid <= ptol)
      pmf = fmax(eps, 0.25 * pmf);
    else
      pmf = fmin(1.0, 1.5 * pmf);
    ptol = presid * fmin(pmf, atol / rnorm);
  }
  __syncthreads();
  c.top = mark;
}

// Mixed-precision iterative local solve: float64 iterative refinement
// around inner MINRES solves whose operator applications run on the tensor
// cores in 3xTF32.  u holds the warm start on entry.  Each step computes the
// residual r = b - B u with the float64 operator, solves B d = r with the
// 3xTF32 operator to kInnerRtol, and adds d to u.  The solve ends once
// ||r|| <= kRefineMargin * local_rtol ||b||, or after kMaxRefine steps or
// when a step gains less than a factor 2; it counts as inexact when the
// reference's own true-residual test (||r|| <= local_rtol ||b||,
// common.py:776-809) fails.  The margin matters: the float64 MINRES path
// usually ends far below local_rtol, and the residual-budget truncation
// that follows raises its threshold with the local residual
// (common.py:850-853), so local solves stopped just at local_rtol would
// truncate harder than the reference does.
constexpr int kMaxRefine = 10;
constexpr double kInnerRtol = 1e-5;
constexpr double kRefineMargin = 1e-2;

__device__ __noinline__ void solve_refined(Ctx& c, const LocalOp& L, const double* b_loc,
                                           double* u, i64 N, int maxit, int* nsolves,
                                           int* ninexact) {
  const ttb_amen_task_t* T = c.T;
  double* red = c.sm->red;
  const i64 mark = c.top;
  double* r = take(c, N);
  double* dlt = take(c, N);
  if (c.status) return;
  const double bn = vnorm_diff(b_loc, nullptr, N, red);
  double rn = 0.0, prev = INFINITY;
  for (int it = 0; it <= kMaxRefine; ++it) {
    // r = b - B u in float64
    apply(c, L, u, r, 1, -1.0, 0.0);
    if (c.status) return;
    double part = 0.0;
    for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) {
      const double v = r[i] + b_loc[i];
      r[i] = v;
      part = fma(v, v, part);
    }
    rn = sqrt(block_sum(part, red));
    if (rn <= kRefineMargin * T->local_rtol * bn || it == kMaxRefine || rn > 0.5 * prev) break;
    prev = rn;
    c.refine += 1;
    minres(c, L, r, dlt, N, kInnerRtol, maxit, false, true);
    if (c.status) return;
    for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) u[i] += dlt[i];
    __syncthreads();
  }
  *nsolves += 1;
  if (!(rn <= T->local_rtol * bn)) *ninexact += 1;
  c.top = mark;
}

// _solve_local_system (common.py:729-809): u <- solution of B u = b.
__device__ __noinline__ void solve_local(Ctx& c, int k, const double* b_loc, double* u, int* nsolves,
                            int* ninexact) {
  const ttb_amen_task_t* T = c.T;
  LocalOp L = local_A(c, k);
  const i64 N = (i64)L.lf * L.n * L.rf;
  if (N <= T->direct_solve_size) {
    direct_solve(c, L, b_loc, u);
    return;
  }
  if (T->local_rtol <= 0.0) {  // iterative solves need a tolerance
    c.status = ST_SETTINGS;
    return;
  }
  const i64 mark = c.top;
  permute_op(c, L);
  vcopy(u, xcore(c, k), N);  // warm start: the current centre core
  __syncthreads();
  double* tmp = take(c, N);
  if (c.status) return;
  const double bn = vnorm_diff(b_loc, nullptr, N, c.sm->red);
  double rtol = T->local_rtol;
  // SciPy's default cap is 5 N iterations; a block solving alone on one SM
  // is bounded tighter so that no launch runs unbounded on a shared GPU
  const int maxit = (int)min(5 * N, (i64)kMaxMinres);
  if (c.mixed && !T->local_gmres) {
    solve_refined(c, L, b_loc, u, N, maxit, nsolves, ninexact);
    if (!c.status) c.top = mark;
    return;
  }
  for (int attempt = 0; attempt < kMaxRestarts; ++attempt) {
    if (T->local_gmres)
      gmres(c, L, b_loc, u, N, rtol, max(1, kMaxMinres / kRestart), true);
    else
      minres(c, L, b_loc, u, N, rtol, maxit, true);
    if (c.status) return;
    apply(c, L, u, tmp, 1, 1.0, 0.0);
    const double rn = vnorm_diff(tmp, b_loc, N, c.sm->red);
    if (rn <= T->local_rtol * bn) {
      *nsolves += 1;
      c.top = mark;
      return;
    }
    rtol = fmax(rtol * kShrink, 1e-15);
  }
  *nsolves += 1;
  *ninexact += 1;
  c.top = mark;
}

// ---------------------------------------------------------------------------
// truncation rank (common.py:812-929)
// ---------------------------------------------------------------------------

// The operator applied to the r-th rank-one term of the solved core,
// C = B (s_r U[:, r] (x) Vh[r, :]), using the factorisation of B over the
// operator bond: for a forward (right-bond) split the term is u (lt, m) (x)
// v (rt) and C[j, k, q] = sum_{a,b} (L_a^T A_ab u)[j, k] (R_b v)[q]; for a
// backward split the term is u (lt) (x) v (m, rt) and
// C[j, k, q] = sum_{a,b} (L_a^T u)[j] (A_ab V R_b)[k, q].  Same values as a
// full application of B to the term (up to rounding) at O(R R2 n^2 r)
// instead of O(n R r^3 + n^2 R^2 r^2) work.
__device__ __noinline__ void rank1_apply(Ctx& c, const LocalOp& L, bool forward, const double* U,
                                         const double* S, const double* Vh, int p, int r,
                                         double* out) {
  const int lt = L.lt, lf = L.lf, R = L.R, R2 = L.R2, n = L.n, m = L.m, rt = L.rt, rf = L.rf;
  const double sr = S[r];
  const i64 mark = c.top;
  if (forward) {
    // u_r[i, l] = s_r U[(i, l), r]; v_r[p'] = Vh[r, p']
    double* P = take(c, (i64)lf * R * m);  // P[j, a, l]
    double* Y = take(c, (i64)lf * n * R2);
    double* W = take(c, (i64)R2 * rf);
    if (c.status) return;
    // P[j, (a, l)] = s_r sum_i left[i, a, j] U[(i, l), r]
    gemm(c, CMat{L.left, 1, (i64)R * lf}, CMat{U + r, (i64)m * p, p},
         OMat(P, lf, m, (i64)R * m, kNoSplit, 0, 1), R * lf, m, lt, sr, 0.0);
    // Y[j, (k, b)] = sum_{a, l} P[j, (a, l)] op[a, k, l, b]
    gemm(c, CMat{P, (i64)R * m, 1}, CMat{L.opP, (i64)n * R2, 1}, Mat{Y, (i64)n * R2, 1}, lf,
         n * R2, R * m, 1.0, 0.0);
    gemm(c, CMat{Vh + (i64)r * rt, 0, 1}, CMat{L.right, (i64)R2 * rf, 1}, Mat{W, 0, 1}, 1,
         R2 * rf, rt, 1.0, 0.0);
    gemm(c, CMat{Y, R2, 1}, CMat{W, rf, 1}, Mat{out, rf, 1}, lf * n, rf, R2, 1.0, 0.0);
  } else {
    // u_r[i] = s_r U[i, r]; v_r[l, p'] = Vh[r, (l, p')]
    double* yv = take(c, (i64)R * lf);
    double* Q = take(c, (i64)m * R2 * rf);
    double* Z = take(c, (i64)R * n * rf);
    if (c.status) return;
    gemm(c, CMat{U + r, 0, p}, CMat{L.left, (i64)R * lf, 1}, Mat{yv, 0, 1}, 1, R * lf, lt, sr,
         0.0);
    gemm(c, CMat{Vh + (i64)r * m * rt, rt, 1}, CMat{L.right, (i64)R2 * rf, 1},
         Mat{Q, (i64)R2 * rf, 1}, m, R2 * rf, rt, 1.0, 0.0);
    // Z[(a, k), q] = sum_{l, b} op[(a, k), (l, b)] Q[(l, b), q]
    gemm(c, CMat{L.op, (i64)m * R2, 1}, CMat{Q, rf, 1}, Mat{Z, rf, 1}, R * n, rf, m * R2, 1.0,
         0.0);
    gemm(c, CMat{yv, 1, lf}, CMat{Z, (i64)n * rf, 1}, Mat{out, (i64)n * rf, 1}, lf, n * rf, R,
         1.0, 0.0);
  }
  c.top = mark;
}

// Ranks whose applied rank-one terms are formed together in choose_rank.
constexpr int kRankChunk = 8;

// The operator applied to the rank-one terms c0 .. c0+nc-1 of the solved
// core at once (rank1_apply for a chunk): the per-term products become three
// GEMMs over the whole chunk, and the last, rank-R contraction is left to the
// caller's accumulation loop.  Forward split: Yc[(r, j), (k, b)] =
// sum_{a, l} (sum_i left[i, a, j] U[(i, l), c0 + r]) op[a, k, l, b], to be
// combined with Wall[c0 + r, (b, q)] = s sum_p' Vh[., p'] right[p', b, q].
// Backward split: Zc[(a, k), (r, q)] = sum_{l, b} op[a, k, l, b]
// (sum_p' Vh[c0 + r, (l, p')] right[p', b, q]), to be combined with
// YV[c0 + r, (a, j)] = sum_i U[i, .] left[i, a, j].
__device__ __noinline__ void rank_chunk(Ctx& c, const LocalOp& L, bool forward, const double* Up,
                                        const double* Vh, int p, int c0, int nc, double* Y,
                                        double* out) {
  const int lt = L.lt, lf = L.lf, R = L.R, R2 = L.R2, n = L.n, m = L.m, rt = L.rt, rf = L.rf;
  if (forward) {
    // Y (PP2[r][j][a][l]) = left^T Up[:, c0:c0+nc, :], written permuted
    gemm(c, CMat{L.left, 1, (i64)R * lf}, CMat{Up + (i64)c0 * m, (i64)p * m, 1},
         OMat(Y, lf, m, (i64)R * m, m, (i64)lf * R * m, 1), R * lf, nc * m, lt, 1.0, 0.0);
    // out[(r, j), (k, b)] = PP2[(r, j), (a, l)] opP[(a, l), (k, b)]
    if (L.sx.rows)  // as out^T = op_X PP2^T
      spmm(c, L.sx, Y, 1, (i64)R * m, OMat(Mat{out, 1, (i64)n * R2}), nc * lf, 1.0, 0.0);
    else
      gemm(c, CMat{Y, (i64)R * m, 1}, CMat{L.opP, (i64)n * R2, 1}, Mat{out, (i64)n * R2, 1},
           nc * lf, n * R2, R * m, 1.0, 0.0);
  } else {
    // Y (Qt[(l, b)][(r, q)]) = Vh[c0:c0+nc, (l, p')] right[p', (b, q)], written permuted
    gemm(c, CMat{Vh + (i64)c0 * m * rt, rt, 1}, CMat{L.right, (i64)R2 * rf, 1},
         OMat(Y, m, rf, (i64)R2 * nc * rf, rf, (i64)nc * rf, 1), nc * m, R2 * rf, rt, 1.0, 0.0);
    // out[(a, k), (r, q)] = op[(a, k), (l, b)] Qt[(l, b), (r, q)]
    if (L.sp.rows)
      spmm(c, L.sp, Y, (i64)nc * rf, 1, OMat(Mat{out, (i64)nc * rf, 1}), nc * rf, 1.0, 0.0);
    else
      gemm(c, CMat{L.op, (i64)m * R2, 1}, CMat{Y, (i64)nc * rf, 1}, Mat{out, (i64)nc * rf, 1},
           R * n, nc * rf, m * R2, 1.0, 0.0);
  }
}

// U (M x p row major), S (p), Vh (p x Kc row major): the solved core
// u = U diag(S) Vh as a vector of length M * Kc.
__device__ __noinline__ int choose_rank(Ctx& c, int k, const double* u, const double* b_loc, const double* U,
                           const double* S, const double* Vh, int M, int Kc, int p) {
  const ttb_amen_task_t* T = c.T;
  double* red = c.sm->red;
  if (!T->residual_mode) {
    if (p <= 0 || S[0] == 0.0) return 1;
    int cnt = 0;
    for (int i = 0; i < p; ++i) cnt += (S[i] / S[0] > T->error_threshold);
    int r = max(cnt, 1);
    if (T->max_rank > 0 && r > T->max_rank) r = T->max_rank;
    return r;
  }
  if (S[0] == 0.0) return 1;
  int limit = p;
  if (T->max_rank > 0) limit = min(limit, T->max_rank);
  LocalOp L = local_A(c, k);
  const i64 N = (i64)M * Kc;
  const i64 mark = c.top;
  permute_op(c, L);
  double* tmp = take(c, N);
  double* part = take(c, N);
  if (c.status) return 1;
  apply(c, L, u, tmp, 1, 1.0, 0.0);
  const double exact = vnorm_diff(tmp, b_loc, N, red);
  const double bn = vnorm_diff(b_loc, nullptr, N, red);
  const double thr = fmax(T->residual_damp * exact, 0.5 * T->truncation_tol * bn);
  for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) part[i] = -b_loc[i];
  __syncthreads();
  int rank = limit;
  const bool forward = (M == L.lt * L.m);
  if (T->debug & 1) {
    // one term at a time, each also applied in full for the self-check
    double* term = take(c, N);
    if (c.status) return 1;
    for (int r = 0; r < limit; ++r) {
      rank1_apply(c, L, forward, U, S, Vh, p, r, tmp);
      if (c.status) return 1;
      const double sr = S[r];
      for (i64 e = threadIdx.x; e < N; e += TTB_THREADS) {
        i64 i = e / Kc, j = e % Kc;
        term[e] = (U[i * p + r] * sr) * Vh[(i64)r * Kc + j];
      }
      __syncthreads();
      double* full = take(c, N);
      if (c.status) return 1;
      apply(c, L, term, full, 1, 1.0, 0.0);
      double dmax = 0.0, fmax_ = 0.0;
      for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) {
        dmax = fmax(dmax, fabs(full[i] - tmp[i]));
        fmax_ = fmax(fmax_, fabs(full[i]));
      }
      // block max via the sum slots: one warp value per warp, then serial
      for (int o = 16; o > 0; o >>= 1) {
        dmax = fmax(dmax, __shfl_down_sync(0xffffffffu, dmax, o));
        fmax_ = fmax(fmax_, __shfl_down_sync(0xffffffffu, fmax_, o));
      }
      __syncthreads();
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = fmax_ > 0.0 ? dmax / fmax_ : dmax;
      __syncthreads();
      double worst = 0.0;
      for (int w = 0; w < TTB_WARPS; ++w) worst = fmax(worst, red[w]);
      c.check = fmax(c.check, worst);
      __syncthreads();
      c.top -= ((N + 31) & ~31LL);
      double s = 0.0;
      for (i64 i = threadIdx.x; i < N; i += TTB_THREADS) {
        double v = part[i] + tmp[i];
        part[i] = v;
        s = fma(v, v, s);
      }
      if (sqrt(block_sum(s, red)) <= thr) {
        rank = r + 1;
        break;
      }
    }
    c.top = mark;
    return rank;
  }
  // Chunks of kRankChunk terms: their applications by rank_chunk, then the
  // running sum -b + C_0 + ... + C_r and its norm term by term, in order, so
  // the first rank within the budget is the one a term-by-term search finds.
  const int lt = L.lt, lf = L.lf, R = L.R, R2 = L.R2, n = L.n, m = L.m, rf = L.rf, rt = L.rt;
  const int CH = kRankChunk;
  double* Up = nullptr;    // forward: Up[i][r][l] = U[(i, l), r]
  double* side = nullptr;  // forward: Wall (limit x R2*rf); backward: YV (limit x R*lf)
  double* Y = take(c, forward ? (i64)CH * lf * R * m : (i64)CH * m * R2 * rf);
  double* Cc = take(c, forward ? (i64)CH * lf * n * R2 : (i64)R * n * CH * rf);
  if (forward) {
    Up = take(c, (i64)lt * p * m);
    side = take(c, (i64)limit * R2 * rf);
    double* svh = take(c, (i64)limit * rt);
    if (c.status) return 1;
    for (i64 e = threadIdx.x; e < (i64)lt * p * m; e += TTB_THREADS) {
      const int l = (int)(e % m);
      const int r = (int)((e / m) % p);
      const i64 i = e / ((i64)m * p);
      Up[e] = U[(i * m + l) * p + r];
    }
    for (i64 e = threadIdx.x; e < (i64)limit * rt; e += TTB_THREADS) svh[e] = S[e / rt] * Vh[e];
    __syncthreads();
    gemm(c, CMat{svh, rt, 1}, CMat{L.right, (i64)R2 * rf, 1}, Mat{side, (i64)R2 * rf, 1}, limit,
         R2 * rf, rt, 1.0, 0.0);
  } else {
    side = take(c, (i64)limit * R * lf);
    if (c.status) return 1;
    gemm(c, CMat{U, 1, p}, CMat{L.left, (i64)R * lf, 1}, Mat{side, (i64)R * lf, 1}, limit,
         R * lf, lt, 1.0, 0.0);
  }
  if (c.status) return 1;
  for (int c0 = 0; c0 < limit; c0 += CH) {
    const int nc = min(CH, limit - c0);
    rank_chunk(c, L, forward, Up, Vh, p, c0, nc, Y, Cc);
    if (c.status) return 1;
    for (int rr = 0; rr < nc; ++rr) {
      const int r = c0 + rr;
      double s = 0.0;
      if (forward) {
        // part[(j, k), q] += sum_b Cc[(rr, j, k), b] Wall[r, (b, q)]
        const double* Yr = Cc + (i64)rr * lf * n * R2;
        const double* Wr = side + (i64)r * R2 * rf;
        for (unsigned e = threadIdx.x; e < (unsigned)N; e += TTB_THREADS) {
          const unsigned jk = e / (unsigned)rf, q = e % (unsigned)rf;
          const double* y = Yr + (i64)jk * R2;
          double v = part[e];
          for (int b = 0; b < R2; ++b) v = fma(y[b], Wr[(i64)b * rf + q], v);
          part[e] = v;
          s = fma(v, v, s);
        }
      } else {
        // part[j, (k, q)] += s_r sum_a YV[r, (a, j)] Cc[(a, k), (rr, q)]
        const double sr = S[r];
        const double* yv = side + (i64)r * R * lf;
        const unsigned nq = (unsigned)(n * rf);
        for (unsigned e = threadIdx.x; e < (unsigned)N; e += TTB_THREADS) {
          const unsigned j = e / nq;
          const unsigned kq = e % nq;
          const unsigned kk = kq / (unsigned)rf, q = kq % (unsigned)rf;
          double acc = 0.0;
          for (int a = 0; a < R; ++a)
            acc = fma(yv[(i64)a * lf + j], Cc[((i64)a * n + kk) * ((i64)nc * rf) + (i64)rr * rf + q],
                      acc);
          const double v = fma(sr, acc, part[e]);
          part[e] = v;
          s = fma(v, v, s);
        }
      }
      if (sqrt(block_sum(s, red)) <= thr) {
        c.top = mark;
        return r + 1;
      }
    }
  }
  c.top = mark;
  return rank;
}

// ---------------------------------------------------------------------------
// centre shifts and enrichment
// ---------------------------------------------------------------------------

// z core k <- Q of core (zl, n, zr); z core k+1 <- R z core k+1 (in place
// through a temporary), zb[k+1] = p.
__device__ __noinline__ void z_shift_right(Ctx& c, int k, const double* core, int zl, int n, int zr) {
  Sm* s = c.sm;
  const int p = min(zl * n, zr);
  const i64 mark = c.top;
  double* R = take(c, (i64)p * zr);
  const int n2 = s->n[k + 1], zr2 = s->zb[k + 2];
  double* nxt = take(c, (i64)p * n2 * zr2);
  if (c.status) return;
  qr(c, CMat{core, zr, 1}, zl * n, zr, Mat{zcore(c, k), p, 1}, Mat{R, zr, 1});
  gemm(c, CMat{R, zr, 1}, CMat{zcore(c, k + 1), (i64)n2 * zr2, 1}, Mat{nxt, (i64)n2 * zr2, 1}, p,
       n2 * zr2, zr, 1.0, 0.0);
  vcopy(zcore(c, k + 1), nxt, (i64)p * n2 * zr2);
  __syncthreads();
  if (threadIdx.x == 0) s->zb[k + 1] = p;
  __syncthreads();
  c.top = mark;
}

__device__ __noinline__ void z_shift_left(Ctx& c, int k, const double* core, int zl, int n, int zr) {
  Sm* s = c.sm;
  const int p = min(zl, n * zr);
  const i64 mark = c.top;
  double* R = take(c, (i64)p * zl);
  const int zpp = s->zb[k - 1], n0 = s->n[k - 1];
  double* prv = take(c, (i64)zpp * n0 * p);
  if (c.status) return;
  // Q^T of core^T goes straight into the slot as (p, n, zr)
  qr(c, CMat{core, 1, (i64)n * zr}, n * zr, zl, Mat{zcore(c, k), 1, (i64)n * zr},
     Mat{R, zl, 1});
  gemm(c, CMat{zcore(c, k - 1), zl, 1}, CMat{R, 1, zl}, Mat{prv, p, 1}, zpp * n0, p, zl, 1.0, 0.0);
  vcopy(zcore(c, k - 1), prv, (i64)zpp * n0 * p);
  __syncthreads();
  if (threadIdx.x == 0) s->zb[k] = p;
  __syncthreads();
  c.top = mark;
}

// generic right-orthonormalisation of the x or z train from ``start`` to 1
__device__ __noinline__ void orth_right(Ctx& c, bool isx, int start) {
  Sm* s = c.sm;
  int* bonds = isx ? s->xb : s->zb;
  for (int i = start; i >= 1; --i) {
    const int rl = bonds[i], n = s->n[i], rr = bonds[i + 1];
    const int p = min(rl, n * rr);
    const i64 mark = c.top;
    double* core = take(c, (i64)rl * n * rr);
    double* R = take(c, (i64)p * rl);
    const int rpp = bonds[i - 1], n0 = s->n[i - 1];
    double* prv = take(c, (i64)rpp * n0 * p);
    if (c.status) return;
    double* slot = isx ? xcore(c, i) : zcore(c, i);
    double* pslot = isx ? xcore(c, i - 1) : zcore(c, i - 1);
    vcopy(core, slot, (i64)rl * n * rr);
    __syncthreads();
    qr(c, CMat{core, 1, (i64)n * rr}, n * rr, rl, Mat{slot, 1, (i64)n * rr}, Mat{R, rl, 1});
    gemm(c, CMat{pslot, rl, 1}, CMat{R, 1, rl}, Mat{prv, p, 1}, rpp * n0, p, rl, 1.0, 0.0);
    if (isx && p > c.rmax) {
      c.status = ST_RANK;
      return;
    }
    vcopy(pslot, prv, (i64)rpp * n0 * p);
    __syncthreads();
    if (threadIdx.x == 0) bonds[i] = p;
    __syncthreads();
    c.top = mark;
  }
}

__device__ __noinline__ void orth_left(Ctx& c, int end) {
  Sm* s = c.sm;
  for (int i = 0; i < end; ++i) {
    const int rl = s->xb[i], n = s->n[i], rr = s->xb[i + 1];
    const int p = min(rl * n, rr);
    const i64 mark = c.top;
    double* core = take(c, (i64)rl * n * rr);
    double* R = take(c, (i64)p * rr);
    const int n2 = s->n[i + 1], r2 = s->xb[i + 2];
    double* nxt = take(c, (i64)p * n2 * r2);
    if (c.status) return;
    vcopy(core, xcore(c, i), (i64)rl * n * rr);
    __syncthreads();
    qr(c, CMat{core, rr, 1}, rl * n, rr, Mat{xcore(c, i), p, 1}, Mat{R, rr, 1});
    gemm(c, CMat{R, rr, 1}, CMat{xcore(c, i + 1), (i64)n2 * r2, 1}, Mat{nxt, (i64)n2 * r2, 1}, p,
         n2 * r2, rr, 1.0, 0.0);
    vcopy(xcore(c, i + 1), nxt, (i64)p * n2 * r2);
    __syncthreads();
    if (threadIdx.x == 0) s->xb[i + 1] = p;
    __syncthreads();
    c.top = mark;
  }
}

// residual core z (amen.py:109-159) of the solved core u at site k
__device__ __noinline__ void residual_core(Ctx& c, int k, const double* u, double* out) {
  Sm* s = c.sm;
  const int zl = s->zb[k], zr = s->zb[k + 1], n = s->n[k];
  project(c, envp(c, 0, F_ZB, k), s->rb[k], zl, bcore(c, k), n, s->rb[k + 1],
          envp(c, 1, F_ZB, k), zr, out, 1.0, 0.0);
  LocalOp L;
  L.left = envp(c, 0, F_ZAX, k);
  L.right = envp(c, 1, F_ZAX, k);
  L.op = acore(c, k);
  L.lt = s->xb[k];
  L.lf = zl;
  L.rt = s->xb[k + 1];
  L.rf = zr;
  L.R = s->R[k];
  L.R2 = s->R[k + 1];
  L.n = L.m = n;
  const i64 mark = c.top;
  permute_op(c, L);
  apply(c, L, u, out, 1, -1.0, 1.0);
  c.top = mark;
}

// forward step after the solve: truncate, enrich, shift x and z
__device__ __noinline__ void forward_update(Ctx& c, int k, const double* u, const double* b_loc,
                               const double* znew) {
  Sm* s = c.sm;
  const int rl = s->xb[k], n = s->n[k], rr = s->xb[k + 1];
  const int zl = s->zb[k], zr = s->zb[k + 1];
  const int M = rl * n, p = min(M, rr);
  const i64 mark = c.top;
  double* U = take(c, (i64)M * p);
  double* S = take(c, p);
  double* Vh = take(c, (i64)p * rr);
  if (c.status) return;
  svd(c, CMat{u, rr, 1}, M, rr, Mat{U, p, 1}, S, Mat{Vh, rr, 1});
  __syncthreads();
  const int rank = choose_rank(c, k, u, b_loc, U, S, Vh, M, rr, p);
  if (c.status) return;
  const int cols = rank + zr;
  const int n2 = s->n[k + 1], r2 = s->xb[k + 2];
  double* enr = take(c, (i64)M * cols);
  double* padded = take(c, (i64)cols * n2 * r2);
  if (c.status) return;
  // enriched = [U[:, :rank] | block], block (rl, n, zr) = lxz^T z_new
  double* block = take(c, (i64)rl * n * zr);
  if (c.status) return;
  gemm(c, CMat{envp(c, 0, F_XZ, k), 1, rl}, CMat{znew, (i64)n * zr, 1},
       Mat{block, (i64)n * zr, 1}, rl, n * zr, zl, 1.0, 0.0);
  for (i64 e = threadIdx.x; e < (i64)M * cols; e += TTB_THREADS) {
    const i64 i = e / cols;
    const int j = (int)(e % cols);
    enr[e] = (j < rank) ? U[i * p + j] : block[i * zr + (j - rank)];
  }
  // padded next core: [S Vh[:rank] @ x_{k+1} ; 0]
  vfill(padded + (i64)rank * n2 * r2, (i64)zr * n2 * r2, 0.0);
  double* svh = take(c, (i64)rank * rr);
  if (c.status) return;
  for (i64 e = threadIdx.x; e < (i64)rank * rr; e += TTB_THREADS) svh[e] = S[e / rr] * Vh[e];
  __syncthreads();
  gemm(c, CMat{svh, rr, 1}, CMat{xcore(c, k + 1), (i64)n2 * r2, 1}, Mat{padded, (i64)n2 * r2, 1},
       rank, n2 * r2, rr, 1.0, 0.0);
  const int q = min(M, cols);
  double* Qb = take(c, (i64)M * q);
  double* R = take(c, (i64)q * cols);
  double* nxt = take(c, (i64)q * n2 * r2);
  if (c.status) return;
  qr(c, CMat{enr, cols, 1}, M, cols, Mat{Qb, q, 1}, Mat{R, cols, 1});
  gemm(c, CMat{R, cols, 1}, CMat{padded, (i64)n2 * r2, 1}, Mat{nxt, (i64)n2 * r2, 1}, q, n2 * r2,
       cols, 1.0, 0.0);
  int nb = q;
  const ttb_amen_task_t* T = c.T;
  if (T->max_rank > 0 && nb > T->max_rank) nb = T->max_rank;  // amen.py:354-358
  if (nb > c.rmax) {
    c.status = ST_RANK;
    return;
  }
  double* xk = xcore(c, k);
  for (i64 e = threadIdx.x; e < (i64)M * nb; e += TTB_THREADS) xk[e] = Qb[(e / nb) * q + e % nb];
  vcopy(xcore(c, k + 1), nxt, (i64)nb * n2 * r2);
  __syncthreads();
  if (threadIdx.x == 0) s->xb[k + 1] = nb;
  __syncthreads();
  c.top = mark;
}

__device__ __noinline__ void backward_update(Ctx& c, int k, const double* u, const double* b_loc,
                                const double* znew) {
  Sm* s = c.sm;
  const int rl = s->xb[k], n = s->n[k], rr = s->xb[k + 1];
  const int zl = s->zb[k], zr = s->zb[k + 1];
  const int Kc = n * rr, p = min(rl, Kc);
  const i64 mark = c.top;
  double* U = take(c, (i64)rl * p);
  double* S = take(c, p);
  double* Vh = take(c, (i64)p * Kc);
  if (c.status) return;
  svd(c, CMat{u, Kc, 1}, rl, Kc, Mat{U, p, 1}, S, Mat{Vh, Kc, 1});
  __syncthreads();
  const int rank = choose_rank(c, k, u, b_loc, U, S, Vh, rl, Kc, p);
  if (c.status) return;
  const int rows = rank + zl;
  const int rpp = s->xb[k - 1], n0 = s->n[k - 1];
  double* enr = take(c, (i64)rows * Kc);
  double* padded = take(c, (i64)rpp * n0 * rows);
  if (c.status) return;
  // enriched rows 0..rank-1: Vh[:rank]; rows rank..: z_new (zl*n, zr) @ rxz (zr, rr)
  vcopy(enr, Vh, (i64)rank * Kc);
  gemm(c, CMat{znew, zr, 1}, CMat{envp(c, 1, F_XZ, k), rr, 1}, Mat{enr + (i64)rank * Kc, rr, 1},
       zl * n, rr, zr, 1.0, 0.0);
  // padded previous core: [x_{k-1} @ (U[:, :rank] S) , 0]
  {
    double* us = take(c, (i64)rl * rank);
    if (c.status) return;
    for (i64 e = threadIdx.x; e < (i64)rl * rank; e += TTB_THREADS) {
      i64 i = e / rank, j = e % rank;
      us[e] = U[i * p + j] * S[j];
    }
    for (i64 e = threadIdx.x; e < (i64)rpp * n0; e += TTB_THREADS)
      for (int j = rank; j < rows; ++j) padded[e * rows + j] = 0.0;
    __syncthreads();
    gemm(c, CMat{xcore(c, k - 1), rl, 1}, CMat{us, rank, 1}, Mat{padded, rows, 1}, rpp * n0, rank,
         rl, 1.0, 0.0);
  }
  const int q = min(rows, Kc);
  double* Qt = take(c, (i64)q * Kc);
  double* R = take(c, (i64)q * rows);
  double* prv = take(c, (i64)rpp * n0 * q);
  if (c.status) return;
  // QR of enriched^T (Kc x rows): x_k <- Q^T (q, n, rr), x_{k-1} <- padded R^T
  qr(c, CMat{enr, 1, Kc}, Kc, rows, Mat{Qt, 1, Kc}, Mat{R, rows, 1});
  gemm(c, CMat{padded, rows, 1}, CMat{R, 1, rows}, Mat{prv, q, 1}, rpp * n0, q, rows, 1.0, 0.0);
  int nb = q;
  const ttb_amen_task_t* T = c.T;
  if (T->max_rank > 0 && nb > T->max_rank) nb = T->max_rank;  // leading rows of x_k stay
  if (nb > c.rmax) {
    c.status = ST_RANK;
    return;
  }
  vcopy(xcore(c, k), Qt, (i64)nb * Kc);
  // x_{k-1} <- prv[:, :nb]
  double* xp = xcore(c, k - 1);
  for (i64 e = threadIdx.x; e < (i64)rpp * n0 * nb; e += TTB_THREADS) {
    i64 i = e / nb, j = e % nb;
    xp[e] = prv[i * q + j];
  }
  __syncthreads();
  if (threadIdx.x == 0) s->xb[k] = nb;
  __syncthreads();
  c.top = mark;
}

// ---------------------------------------------------------------------------
// norms of trains: ||A x - b|| (common.py:118-146) and ||b||
// ---------------------------------------------------------------------------

// Core i of the residual train A x - b (block sum of the Kronecker core
// of A x and of -b at b's centre), as (rows, n, cols) row major.
__device__ __noinline__ void residual_train_core(Ctx& c, int i, double* out, int& rows, int& cols) {
  Sm* s = c.sm;
  const int d = c.d;
  const int n = s->n[i];
  const int x1 = s->xb[i], x2 = s->xb[i + 1], R2 = s->R[i + 1], rb2 = s->rb[i + 1];
  const int ra = s->R[i] * x1, ra2 = R2 * x2;  // 1 on the boundaries
  rows = (i == 0) ? 1 : ra + s->rb[i];
  cols = (i == d - 1) ? 1 : ra2 + rb2;
  const int kb = c.T->b_orth_center >= 0 ? c.T->b_orth_center : 0;
  const double bs = (i == kb) ? -1.0 : 1.0;
  const double* A = acore(c, i);
  const double* x = xcore(c, i);
  const double* b = bcore(c, i);
  const bool first = (i == 0), last = (i == d - 1);
  const i64 total = (i64)rows * n * cols;
  for (i64 e = threadIdx.x; e < total; e += TTB_THREADS) {
    const int cc = (int)(e % cols);
    const int j = (int)((e / cols) % n);
    const int rr = (int)(e / ((i64)cols * n));
    const bool inA = (first || rr < ra) && (last || cc < ra2);
    const bool inB = (first || rr >= ra) && (last || cc >= ra2);
    double v = 0.0;
    if (inA) {
      // Kronecker block of A x: rows (a, xr), columns (bb, xc)
      const int a = rr / x1, xr = rr % x1, bb = cc / x2, xc = cc % x2;
      for (int l = 0; l < n; ++l)
        v = fma(A[(((i64)a * n + j) * n + l) * R2 + bb], x[((i64)xr * n + l) * x2 + xc], v);
    }
    if (inB) {
      const int br = first ? 0 : rr - ra, bc = last ? 0 : cc - ra2;
      v += bs * b[((i64)br * n + j) * rb2 + bc];
    }
    out[e] = v;
  }
  __syncthreads();
}

// Frobenius norm of a train given core by core (right QR sweep keeping R).
// ``which``: 0 = the residual train, 1 = b.
__device__ __noinline__ double train_norm(Ctx& c, int which) {
  Sm* s = c.sm;
  const int d = c.d;
  const i64 mark = c.top;
  // largest bond of the train, for the two carry buffers
  int bmax = 1;
  for (int i = 0; i <= d; ++i) {
    const int bnd = which == 0 ? s->R[i] * s->xb[i] + s->rb[i] : s->rb[i];
    bmax = max(bmax, bnd);
  }
  double* carry_a = take(c, (i64)bmax * bmax);
  double* carry_b = take(c, (i64)bmax * bmax);
  if (c.status) return 0.0;
  double* carry = nullptr;
  int cp = 1;  // columns of the carry
  for (int i = d - 1; i >= 0; --i) {
    const i64 imark = c.top;
    int rows, cols;
    const int n = s->n[i];
    const double* core;
    const double* m = nullptr;
    if (which == 0 && carry) {
      // core i of A x - b times the carry without forming the core: the
      // A x block as (x then A) contractions, the b block as one product
      const int x1 = s->xb[i], x2 = s->xb[i + 1], R1 = s->R[i], R2 = s->R[i + 1];
      const int rb1 = s->rb[i], rb2 = s->rb[i + 1];
      const int ra = R1 * x1, ra2 = R2 * x2;
      const bool first = (i == 0);
      rows = first ? 1 : ra + rb1;
      cols = ra2 + rb2;
      double* mm = take(c, (i64)rows * n * cp);
      double* T = take(c, (i64)n * R2 * x1 * cp);  // T[l, b, xr, q]
      if (c.status) return 0.0;
      const double* xc = xcore(c, i);
      // T[(xr, l), q] = sum_xc x[xr, l, xc] carry[(b, xc), q] for each b
      for (int bb = 0; bb < R2; ++bb)
        gemm(c, CMat{xc, x2, 1}, CMat{carry + (i64)bb * x2 * cp, cp, 1},
             OMat(T + (i64)bb * x1 * cp, n, cp, (i64)R2 * x1 * cp, kNoSplit, 0, 1), x1 * n, cp,
             x2, 1.0, 0.0);
      // mm[(a, xr), j, q] = sum_{l, b} A[a, j, l, b] T[(l, b), (xr, q)]
      {
        const OMat om(mm, n, (i64)x1 * n * cp, cp, cp, (i64)n * cp, 1);
        const SpOp S = build_spop(c, acore(c, i), R1, n, n, R2, SP_P);
        if (c.status) return 0.0;
        if (S.rows)
          spmm(c, S, T, (i64)x1 * cp, 1, om, x1 * cp, 1.0, 0.0);
        else
          gemm(c, CMat{acore(c, i), (i64)n * R2, 1}, CMat{T, (i64)x1 * cp, 1}, om, R1 * n,
               x1 * cp, n * R2, 1.0, 0.0);
      }
      // b rows (the first core: the same row, accumulated), sign as in
      // residual_train_core
      const int kb = c.T->b_orth_center >= 0 ? c.T->b_orth_center : 0;
      gemm(c, CMat{bcore(c, i), rb2, 1}, CMat{carry + (i64)ra2 * cp, cp, 1},
           Mat{mm + (first ? 0 : (i64)ra * n * cp), cp, 1}, rb1 * n, cp, rb2,
           (i == kb) ? -1.0 : 1.0, first ? 1.0 : 0.0);
      m = mm;
      core = nullptr;
    } else if (which == 0) {
      const int ra = s->R[i] * s->xb[i], ra2 = s->R[i + 1] * s->xb[i + 1];
      const int rr = (i == 0) ? 1 : ra + s->rb[i];
      const int cc = (i == d - 1) ? 1 : ra2 + s->rb[i + 1];
      double* buf = take(c, (i64)rr * n * cc);
      if (c.status) return 0.0;
      residual_train_core(c, i, buf, rows, cols);
      core = buf;
    } else {
      rows = s->rb[i];
      cols = s->rb[i + 1];
      core = bcore(c, i);
    }
    if (m) {
      // formed above
    } else if (carry) {
      double* mm = take(c, (i64)rows * n * cp);
      if (c.status) return 0.0;
      gemm(c, CMat{core, cols, 1}, CMat{carry, cp, 1}, Mat{mm, cp, 1}, rows * n, cp, cols, 1.0,
           0.0);
      m = mm;
    } else {
      m = core;
      cp = cols;
    }
    if (i == 0) {
      const double nr = vnorm_diff(m, nullptr, (i64)rows * n * cp, s->red);
      c.top = mark;
      return nr;
    }
    // QR of m^T (n*cp x rows), keep R^T (rows x p) as the next carry
    const int p = min(n * cp, rows);
    double* R = take(c, (i64)p * rows);
    if (c.status) return 0.0;
    qr(c, CMat{m, 1, (i64)n * cp}, n * cp, rows, Mat{nullptr, 0, 0}, Mat{R, rows, 1});
    double* nc = (carry == carry_a) ? carry_b : carry_a;
    for (i64 e = threadIdx.x; e < (i64)rows * p; e += TTB_THREADS) {
      const i64 a = e / p, q = e % p;
      nc[e] = R[q * rows + a];
    }
    __syncthreads();
    carry = nc;
    cp = p;
    c.top = imark;
  }
  c.top = mark;
  return 0.0;
}

// True on every thread once the solve has run past its time limit: thread 0
// reads the device timer and the block follows its decision.
__device__ __noinline__ bool over_time(Ctx& c, unsigned long long t_start) {
  if (c.T->time_limit_ns <= 0) return false;
  __syncthreads();
  if (threadIdx.x == 0)
    c.sm->flag = (global_ns() - t_start > (unsigned long long)c.T->time_limit_ns) ? 1 : 0;
  __syncthreads();
  return c.sm->flag != 0;
}

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------

// The whole solve of one task (everything but the tensor-memory set-up).
__device__ __noinline__ void amen_run(Ctx& c, int rmax) {
  Sm& sm = *c.sm;
  const ttb_amen_task_t* T = c.T;
  const unsigned long long t_start = global_ns();
  long long t_ph = clock64();
#define PHASE(ph)                         \
  {                                       \
    const long long t_now = clock64();    \
    c.cyc[ph] += t_now - t_ph;            \
    t_ph = t_now;                         \
  }
  const int d = c.d;
  const int* dims = T->dims;
  if (d < 2 || d > kD) {
    if (threadIdx.x == 0) T->result[0] = ST_SETTINGS;
    return;
  }
  // shapes
  for (int i = threadIdx.x; i <= d; i += TTB_THREADS) {
    if (i < d) sm.n[i] = dims[i];
    sm.R[i] = dims[d + i];
    sm.rb[i] = dims[2 * d + 1 + i];
    sm.xb[i] = dims[3 * d + 2 + i];
    sm.zb[i] = dims[4 * d + 3 + i];
  }
  __syncthreads();
  // slots: x cores, z cores, environments
  if (threadIdx.x == 0) {
    i64 off = 0;
    const i64 K = c.K;
    for (int k = 0; k < d; ++k) {
      sm.xo[k] = off;
      off += ((i64)rmax * sm.n[k] * rmax + 31) & ~31LL;
    }
    for (int k = 0; k < d; ++k) {
      sm.zo[k] = off;
      off += (K * sm.n[k] * K + 31) & ~31LL;
    }
    for (int side = 0; side < 2; ++side)
      for (int k = 0; k < d; ++k) {
        const int pb = side == 0 ? k : k + 1;
        const i64 R = sm.R[pb], rb = sm.rb[pb];
        const i64 sizes[5] = {(i64)rmax * R * rmax, rb * rmax, rb * K, (i64)rmax * R * K,
                              K * rmax};
        for (int f = 0; f < 5; ++f) {
          sm.eo[side][f][k] = off;
          off += (sizes[f] + 31) & ~31LL;
        }
      }
    sm.flag = (off <= c.cap) ? 1 : 0;
    sm.stack0 = off;  // the stack starts after the slots
  }
  __syncthreads();
  if (!sm.flag) {
    if (threadIdx.x == 0) T->result[0] = ST_SLAB;
    return;
  }
  c.top = sm.stack0;
  __syncthreads();
  for (int k = 0; k <= d; ++k)
    if (sm.xb[k] > rmax) {
      if (threadIdx.x == 0) T->result[0] = ST_RANK;
      return;
    }
  // x0 and z0 into their slots
  for (int k = 0; k < d; ++k) {
    vcopy(xcore(c, k), T->x0 + T->x0_off[k], (i64)sm.xb[k] * sm.n[k] * sm.xb[k + 1]);
    vcopy(zcore(c, k), T->z0 + T->z0_off[k], (i64)sm.zb[k] * sm.n[k] * sm.zb[k + 1]);
  }
  __syncthreads();
  int nsolves = 0, ninexact = 0, sweeps = 0, stop = 2;
#define CHECK                                                      \
  if (c.status) {                                                  \
    if (threadIdx.x == 0) {                                        \
      T->result[0] = c.status;                                     \
      T->result[1] = sweeps;                                       \
      T->residuals[2 * T->max_sweeps] = c.flops;                   \
      T->residuals[2 * T->max_sweeps + 1] = (double)c.applies;     \
      T->residuals[2 * T->max_sweeps + 10] = (double)t_start;      \
      T->residuals[2 * T->max_sweeps + 11] = (double)global_ns();  \
    }                                                              \
    return;                                                        \
  }
  if (T->x0_orth_center != 0) orth_right(c, true, d - 1);
  CHECK;
  orth_right(c, false, d - 1);
  CHECK;
  // fit z to b - A x (amen.py:162-224)
  for (int i = d - 1; i >= 0; --i) {
    build_env(c, 1, F_ZB, i);
    build_env(c, 1, F_ZAX, i);
    CHECK;
  }
  const i64 base = c.top;
  for (int k = 0; k < d - 1; ++k) {
    build_env(c, 0, F_ZB, k);
    build_env(c, 0, F_ZAX, k);
    CHECK;
    double* core = take(c, (i64)sm.zb[k] * sm.n[k] * sm.zb[k + 1]);
    CHECK;
    residual_core(c, k, xcore(c, k), core);
    z_shift_right(c, k, core, sm.zb[k], sm.n[k], sm.zb[k + 1]);
    CHECK;
    c.top = base;
  }
  build_env(c, 0, F_ZB, d - 1);
  build_env(c, 0, F_ZAX, d - 1);
  for (int k = d - 1; k >= 0; --k) {
    build_env(c, 1, F_ZB, k);
    build_env(c, 1, F_ZAX, k);
    CHECK;
    double* core = take(c, (i64)sm.zb[k] * sm.n[k] * sm.zb[k + 1]);
    CHECK;
    residual_core(c, k, xcore(c, k), core);
    if (k > 0) {
      z_shift_left(c, k, core, sm.zb[k], sm.n[k], sm.zb[k + 1]);
    } else {
      vcopy(zcore(c, 0), core, (i64)sm.n[0] * sm.zb[1]);
      __syncthreads();
    }
    CHECK;
    c.top = base;
  }
  for (int i = d - 1; i >= 0; --i) {
    for (int f = 0; f < 5; ++f) build_env(c, 1, f, i);
    CHECK;
  }
  double b_norm = 0.0;
  if (T->track_residual) {
    if (T->b_orth_center >= 0) {
      const int kb = T->b_orth_center;
      b_norm = vnorm_diff(bcore(c, kb), nullptr, (i64)sm.rb[kb] * sm.n[kb] * sm.rb[kb + 1], sm.red);
    } else {
      b_norm = train_norm(c, 1);
    }
    CHECK;
  }
  double prev_res = 0.0;
  PHASE(PH_INIT);
  for (int sweep = 0; sweep < T->max_sweeps; ++sweep) {
    for (int k = 0; k < d - 1; ++k) {
      for (int f = 0; f < 5; ++f) build_env(c, 0, f, k);
      CHECK;
      PHASE(PH_ENV);
      const i64 N = (i64)sm.xb[k] * sm.n[k] * sm.xb[k + 1];
      double* b_loc = take(c, N);
      double* u = take(c, N);
      double* znew = take(c, (i64)sm.zb[k] * sm.n[k] * sm.zb[k + 1]);
      CHECK;
      project(c, envp(c, 0, F_B, k), sm.rb[k], sm.xb[k], bcore(c, k), sm.n[k], sm.rb[k + 1],
              envp(c, 1, F_B, k), sm.xb[k + 1], b_loc, 1.0, 0.0);
      solve_local(c, k, b_loc, u, &nsolves, &ninexact);
      CHECK;
      PHASE(PH_SOLVE);
      residual_core(c, k, u, znew);
      PHASE(PH_ZCORE);
      forward_update(c, k, u, b_loc, znew);
      CHECK;
      z_shift_right(c, k, znew, sm.zb[k], sm.n[k], sm.zb[k + 1]);
      CHECK;
      PHASE(PH_TRUNC);
      c.top = base;
      if (over_time(c, t_start)) c.status = ST_TIME;
      CHECK;
    }
    for (int f = 0; f < 5; ++f) build_env(c, 0, f, d - 1);
    CHECK;
    for (int k = d - 1; k >= 0; --k) {
      for (int f = 0; f < 5; ++f) build_env(c, 1, f, k);
      CHECK;
      PHASE(PH_ENV);
      const i64 N = (i64)sm.xb[k] * sm.n[k] * sm.xb[k + 1];
      double* b_loc = take(c, N);
      double* u = take(c, N);
      double* znew = take(c, (i64)sm.zb[k] * sm.n[k] * sm.zb[k + 1]);
      CHECK;
      project(c, envp(c, 0, F_B, k), sm.rb[k], sm.xb[k], bcore(c, k), sm.n[k], sm.rb[k + 1],
              envp(c, 1, F_B, k), sm.xb[k + 1], b_loc, 1.0, 0.0);
      solve_local(c, k, b_loc, u, &nsolves, &ninexact);
      CHECK;
      PHASE(PH_SOLVE);
      residual_core(c, k, u, znew);
      PHASE(PH_ZCORE);
      if (k == 0) {
        vcopy(xcore(c, 0), u, N);
        vcopy(zcore(c, 0), znew, (i64)sm.n[0] * sm.zb[1]);
        __syncthreads();
      } else {
        backward_update(c, k, u, b_loc, znew);
        CHECK;
        z_shift_left(c, k, znew, sm.zb[k], sm.n[k], sm.zb[k + 1]);
        CHECK;
      }
      PHASE(PH_TRUNC);
      c.top = base;
      if (over_time(c, t_start)) c.status = ST_TIME;
      CHECK;
    }
    sweeps = sweep + 1;
    {
      int mb = 1;
      for (int k = 0; k <= d; ++k) mb = max(mb, sm.xb[k]);
      if (threadIdx.x == 0) T->residuals[T->max_sweeps + sweep] = (double)mb;
    }
    if (!T->track_residual) continue;
    const double rn = train_norm(c, 0);
    CHECK;
    PHASE(PH_RESID);
    const double res = (b_norm == 0.0) ? rn : rn / b_norm;
    if (threadIdx.x == 0) T->residuals[sweep] = res;
    if (T->residual_mode && res <= T->residual_tol) {
      stop = 0;
      break;
    }
    if (T->stagnation_on && sweep >= 1 && res > T->stagnation_factor * prev_res) {
      stop = 1;
      break;
    }
    prev_res = res;
  }
  // amen.py:710-720: bonds above the product of the modes on their left
  {
    int last = 0;
    double prod = 1.0;
    for (int k = 1; k < d; ++k) {
      prod *= sm.n[k - 1];
      if ((double)sm.xb[k] > prod) last = k;
    }
    if (last > 0) {
      orth_left(c, last);
      CHECK;
      orth_right(c, true, last);
      CHECK;
    }
  }
  if (threadIdx.x == 0) {
    T->result[0] = ST_OK;
    T->result[1] = sweeps;
    T->result[2] = stop;
    T->result[3] = nsolves;
    T->result[4] = ninexact;
    for (int k = 0; k <= d; ++k) T->result[5 + k] = sm.xb[k];
    for (int k = 0; k < d; ++k) T->x_offsets[k] = sm.xo[k];
    T->residuals[2 * T->max_sweeps] = c.flops;
    T->residuals[2 * T->max_sweeps + 1] = (double)c.applies;
    for (int i = 0; i < PH_N; ++i) T->residuals[2 * T->max_sweeps + 2 + i] = (double)c.cyc[i];
    T->residuals[2 * T->max_sweeps + 2 + PH_N] = c.check;
    T->residuals[2 * T->max_sweeps + 12] = c.check_qr;
    T->residuals[2 * T->max_sweeps + 13] = (double)c.n_qr2;
    T->residuals[2 * T->max_sweeps + 10] = (double)t_start;
    T->residuals[2 * T->max_sweeps + 11] = (double)global_ns();
  }
#undef PHASE
#undef CHECK
}

// The tensor pipeline's shared-memory stages take the start of the pool,
// which the factorisations use only outside the mixed-precision solves.
static_assert(TC_RING_BYTES <= kPoolBytes, "tensor-core stages must fit the pool");

// Per-block context of a task (both kernels).
__device__ void init_ctx(Ctx& c, const ttb_amen_task_t* T, Sm* sm, double* dyn, int rmax) {
  c.T = T;
  c.sm = sm;
  c.slab = T->slab;
  c.cap = T->slab_doubles;
  c.top = 0;
  c.pool = dyn + GSTAGES * GSTAGE_D;
  c.ring = dyn;
  c.gsm = reinterpret_cast<GemmSmem*>(dyn);
  c.d = T->d;
  c.rmax = rmax;
  c.K = T->kickrank;
  c.status = ST_OK;
  c.flops = 0.0;
  c.applies = 0;
  c.check = 0.0;
  c.check_qr = 0.0;
  c.n_qr2 = 0;
  for (int i = 0; i < PH_N; ++i) c.cyc[i] = 0;
  c.mixed = (T->precision == 1);
  c.flops_tc = 0.0;
  c.refine = 0;
  c.csize = 1;
  c.cmd = nullptr;
  c.vpart = nullptr;
}

// The solve of task T by this block (the lone block or a cluster's leader),
// with the tensor-core pipeline around it in mixed precision.
__device__ void lead_solve(Ctx& c, Sm& sm, int rmax) {
  const ttb_amen_task_t* T = c.T;
  if (c.mixed) {
    c.tc.ring = reinterpret_cast<float*>(c.pool);
    c.tc.mbar = sm.mbar;
    c.tc.slot = &sm.tmem_slot;
    tc_init(c.tc);
  }
  amen_run(c, rmax);
  if (c.mixed) {
    tc_release(c.tc);
    if (threadIdx.x == 0) {
      T->residuals[2 * T->max_sweeps + 14] = c.flops_tc;
      T->residuals[2 * T->max_sweeps + 15] = (double)c.refine;
    }
  }
}

__global__ void __launch_bounds__(TTB_THREADS, 1)
    k_amen(const ttb_amen_task_t* __restrict__ tasks, int rmax) {
  extern __shared__ __align__(16) double dyn[];
  __shared__ Sm sm;
  Ctx c;
  init_ctx(c, tasks + blockIdx.x, &sm, dyn, rmax);
  lead_solve(c, sm, rmax);
}

// A cluster's worker block: run the leader's commands until the exit one.
// ``lead`` is the leader's command slot (distributed shared memory).
__device__ __noinline__ void cluster_worker(Ctx& c, const ClusterCmd* lead, int rank) {
  __shared__ ClusterCmd q;
  for (;;) {
    cluster_barrier();  // a command is posted
    if (threadIdx.x < sizeof(ClusterCmd) / 8)
      reinterpret_cast<unsigned long long*>(&q)[threadIdx.x] =
          reinterpret_cast<const unsigned long long*>(lead)[threadIdx.x];
    __syncthreads();
    if (q.op == CL_EXIT) {
      cluster_barrier();  // the leader's shared memory stays until every block has read
      return;
    }
    if (q.op == CL_GEMM) {
      cta_gemm_pipe(CMat{q.a, q.a_rs, q.a_cs}, CMat{q.b, q.b_rs, q.b_cs}, cmd_out(q), q.M, q.N,
                    q.K, q.alpha, q.beta, c.ring, rank, c.csize);
    } else if (q.op == CL_VEC) {
      for (int k = rank; k < kVecChunks; k += c.csize) {
        const double v = vpass_chunk(q.vec, k, c.sm->red);
        if (threadIdx.x == 0) c.vpart[k] = v;
      }
    } else if (q.op == CL_LOCAL) {
      form_local(q.a, q.b, q.sp_val, q.dim, q.c, rank, c.csize);
    } else if (q.op == CL_LU) {
      cta_gepp_update(q.c, q.M, q.rhs, q.M, q.K, c.pool, q.ipiv, true, rank, c.csize);
    } else if (q.op == CL_QR) {
      cta_qr_r_blocked2(CMat{q.a, q.a_rs, q.a_cs}, q.M, q.N, q.c, q.rhs, Mat{nullptr, 0, 0},
                        c.pool, c.sm->red, c.ring, rank, c.csize);
    } else {
      const int tw = q.b_cs == 1 ? spmm_tile(q.sp_rows, q.sp_nnz, q.sp_cols) : 0;
      if (tw > 0)
        spmm_staged(c.pool, q.sp_ptr, q.sp_col, q.sp_val, q.sp_rows, q.sp_nnz, q.sp_cols, q.b,
                    q.b_rs, cmd_out(q), q.N, q.alpha, q.beta, tw, rank, c.csize);
      else
        spmm_rows(q.sp_ptr, q.sp_col, q.sp_val, q.sp_rows, q.b, q.b_rs, q.b_cs, cmd_out(q), q.N,
                  q.alpha, q.beta, rank, c.csize);
    }
    cluster_barrier();  // this block's share is written
  }
}

// One solve per cluster of blocks (launched with a cluster dimension): the
// leader (rank 0) runs it, the other blocks take shares of its products.
__global__ void __launch_bounds__(TTB_THREADS, 1)
    k_amen_cl(const ttb_amen_task_t* __restrict__ tasks, int rmax) {
  extern __shared__ __align__(16) double dyn[];
  __shared__ Sm sm;
  __shared__ ClusterCmd cmd;
  __shared__ double vpart[kVecChunks];
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int rank = (int)cl.block_rank();
  const int csize = (int)cl.num_blocks();
  Ctx c;
  init_ctx(c, tasks + blockIdx.x / csize, &sm, dyn, rmax);
  c.csize = csize;
  c.cmd = &cmd;
  c.vpart = vpart;
  if (rank == 0) {
    lead_solve(c, sm, rmax);
    if (threadIdx.x == 0) cmd.op = CL_EXIT;
    cluster_barrier();
    cluster_barrier();
  } else {
    cluster_worker(c, cl.map_shared_rank(&cmd, 0), rank);
  }
}

}  // namespace ttb_solve
using namespace ttb_solve;

extern "C" {

long long ttb_amen_slab_doubles(int d, const int* dims, int kickrank, int rmax,
                                int direct_solve_size) {
  if (d < 2 || d > kD) return -1;
  const long long K = kickrank;
  long long slots = 0, nmax = 1, Rmax = 1, rbmax = 1;
  for (int k = 0; k < d; ++k) {
    const long long n = dims[k];
    nmax = std::max(nmax, n);
    slots += ((long long)rmax * n * rmax + 31) & ~31LL;
    slots += (K * n * K + 31) & ~31LL;
  }
  for (int k = 0; k <= d; ++k) {
    Rmax = std::max<long long>(Rmax, dims[d + k]);
    rbmax = std::max<long long>(rbmax, dims[2 * d + 1 + k]);
  }
  for (int side = 0; side < 2; ++side)
    for (int k = 0; k < d; ++k) {
      const int pb = side == 0 ? k : k + 1;
      const long long R = dims[d + pb], rb = dims[2 * d + 1 + pb];
      const long long sizes[5] = {(long long)rmax * R * rmax, rb * rmax, rb * K,
                                  (long long)rmax * R * K, K * rmax};
      for (int f = 0; f < 5; ++f) slots += (sizes[f] + 31) & ~31LL;
    }
  // stack bound of one sweep step: b_loc, u and z_new, then the largest of
  // the sub-steps, each term rounded up generously
  const long long r = rmax, n = nmax, R = Rmax, N = r * n * r, cols = r + K;
  // sparse forms of an operator core (two in permute_op, one elsewhere)
  const long long sp = spop_doubles(R * n * n * R, R * n);
  const long long env = 2 * r * R * n * r + r * n * r + sp;
  const long long apply = 2 * r * n * R * r + R * n * n * R + R * r * r + 2 * sp;  // + permute_op
  const long long dn = std::min<long long>(direct_solve_size, N);
  const long long direct = dn * dn + dn + dn * LNB;
  // MINRES: six vectors; GMRES: restart + 3 vectors and the Hessenberg data
  const long long iter = N + std::max(6 * N, (kRestart + 3) * (N + 32) + 2048) + apply;
  const long long rank = 4 * N + 2LL * kRankChunk * R * n * r + R * r * r + r * r + apply;
  const long long fact = r * n * r + r + r * n * r        // U S Vh
                         + (r * n) * r + 2 * r * r + 4 * r  // svd work
                         + (r * n) * cols + 2 * cols * n * r + r * r  // enriched, padded, svh
                         + r * n * cols + cols * cols + cols * n * r  // Q, R, next
                         + r * n * cols + cols + r * n * K;            // qr work, block
  const long long bb = R * r + rbmax;
  const long long resid = 2 * bb * bb + bb * n * bb + bb * n * bb + bb * bb + sp;
  const long long step = 3 * N + K * n * K +
                         std::max({env, direct, iter, rank + fact, resid, 2 * rbmax * n * r});
  return slots + 2 * step + (1 << 16);
}

int ttb_amen_persistent_cluster(const ttb_amen_task_t* tasks, int count, int rmax, int cluster,
                                void* stream) {
  if (cluster <= 1) return ttb_amen_persistent(tasks, count, rmax, stream);
  if (count <= 0) return 0;
  if (cluster > 8) return (int)cudaErrorInvalidValue;
  static int configured[kMaxDevices];
  const size_t smem = kRingBytes + kPoolBytes;
  if (int e = smem_limit_once((const void*)k_amen_cl, (int)smem, configured)) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(count * cluster), 1, 1);
  cfg.blockDim = dim3(TTB_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = reinterpret_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_amen_cl, tasks, rmax);
  ttb::count_launch();
  if (e != cudaSuccess) return (int)e;
  return (int)cudaGetLastError();
}

int ttb_amen_persistent(const ttb_amen_task_t* tasks, int count, int rmax, void* stream) {
  if (count <= 0) return 0;
  static int configured[kMaxDevices];
  const size_t smem = kRingBytes + kPoolBytes;
  if (int e = smem_limit_once((const void*)k_amen, (int)smem, configured)) return e;
  k_amen<<<count, TTB_THREADS, smem, reinterpret_cast<cudaStream_t>(stream)>>>(tasks, rmax);
  ttb::count_launch();
  return (int)cudaGetLastError();
}

}  // extern "C"
