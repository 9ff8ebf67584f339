// CTA-level float64 building blocks shared by every kernel of libttb200.
//
// All routines here are executed cooperatively by one thread block of
// TTB_THREADS threads.  Matrices are addressed through generic pointers and
// explicit (row, column) element strides, so the same code runs on shared
// memory, on global memory and on transposed views.  Reductions are done in a
// fixed order (per-thread strided partials, a warp tree, then the warp sums
// in warp order), so a result never depends on scheduling and every thread
// of the block sees the same value.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#ifndef TTB_THREADS
#define TTB_THREADS 256
#endif
#define TTB_WARPS (TTB_THREADS / 32)

namespace ttb {

typedef long long i64;

// Host side (ttb200.cu): raise ``func``'s dynamic shared-memory limit to
// ``bytes`` on the current device the first time a launch there needs it.
// ``done`` holds one flag per device index (kMaxDevices); a flag is set only
// after cudaFuncSetAttribute succeeded, and its error is returned otherwise.
constexpr int kMaxDevices = 64;
int smem_limit_once(const void* func, int bytes, int* done);

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------

static __device__ __forceinline__ double warp_sum(double v) {
  // tree towards lane 0, then broadcast lane 0 so all lanes agree bitwise
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return __shfl_sync(0xffffffffu, v, 0);
}

// Sum over the block; every thread returns the same value.  ``red`` must
// hold TTB_WARPS doubles of shared memory.  Contains two __syncthreads.
static __device__ __forceinline__ double block_sum(double v, double* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int i = 0; i < TTB_WARPS; ++i) t += red[i];
  return t;
}

// Index of the entry of largest absolute value, first index on ties (the
// LAPACK idamax convention).  ``redv``/``redi`` hold TTB_WARPS entries.
static __device__ __forceinline__ int block_argmax_abs(double v, int idx, double* redv, int* redi) {
  double a = (idx >= 0) ? fabs(v) : -1.0;
  int i = idx;
  for (int o = 16; o > 0; o >>= 1) {
    double a2 = __shfl_down_sync(0xffffffffu, a, o);
    int i2 = __shfl_down_sync(0xffffffffu, i, o);
    if (a2 > a || (a2 == a && i2 >= 0 && (i < 0 || i2 < i))) { a = a2; i = i2; }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) { redv[wid] = a; redi[wid] = i; }
  __syncthreads();
  double best = -1.0;
  int bi = -1;
  for (int w = 0; w < TTB_WARPS; ++w) {
    double a2 = redv[w];
    int i2 = redi[w];
    if (a2 > best || (a2 == best && i2 >= 0 && (bi < 0 || i2 < bi))) { best = a2; bi = i2; }
  }
  return bi;
}

// ---------------------------------------------------------------------------
// strided matrix view
// ---------------------------------------------------------------------------

struct Mat {
  double* p;
  i64 rs, cs;  // element strides of a row step and a column step
  __device__ __forceinline__ double& operator()(int i, int j) const { return p[i * rs + j * cs]; }
};

// Column step of an m-row matrix in shared memory: odd, so that the entries
// of a row fall on different banks.
__host__ __device__ constexpr int odd_step(int m) { return m | 1; }

// Column step of the SVD's k-row square matrices: eight lanes read eight
// row pairs of each of four neighbouring columns, 16 bytes a lane, so columns
// start on 16-byte boundaries and two neighbours cover all the banks.
__host__ __device__ constexpr int svd_step(int k) { return k + ((8 - k) & 15); }

// A thread's walk over a table of rows of ``width`` entries: the entries first,
// first + stride, ... (first < 2^31) as row and place in it, advanced without a
// division and without a count of entries, which may pass 32 bits.
struct TableWalk {
  int row, at;
  __host__ __device__ TableWalk(int first, int stride, int width_)
      : row(first / width_), at(first % width_), rows(stride / width_), rest(stride % width_),
        width(width_) {}
  __host__ __device__ __forceinline__ void next() {
    row += rows;
    at += rest;
    if (at >= width) {
      at -= width;
      ++row;
    }
  }

 private:
  int rows, rest, width;
};

// The first 16-byte boundary at or after p.
__device__ __forceinline__ double* align2(double* p) {
  return reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15);
}

struct CMat {
  const double* p;
  i64 rs, cs;
  __device__ __forceinline__ double operator()(int i, int j) const { return p[i * rs + j * cs]; }
};

// ---------------------------------------------------------------------------
// GEMM: one GBM x 64 output tile per call, K staged through shared memory,
// products on the FP64 tensor-core path (mma.sync m8n8k4 .f64)
// ---------------------------------------------------------------------------

// Tile rows: 32 per four warps (64 for 8 warps, 96 for 12), 64 columns.
// K depth of a staged slab (16, or 32 for half the block barriers per K)
#ifndef TTB_GBK
#define TTB_GBK 16
#endif
constexpr int GBM = 8 * TTB_WARPS, GBN = 64, GBK = TTB_GBK;
// Row pitches of the staged tiles: 4 more than a multiple of 16 doubles puts
// the four k-rows a fragment load touches on disjoint bank groups, so each
// load takes two wavefronts.
constexpr int GPITCH_A = GBM + 4, GPITCH_B = GBN + 4;
// loads per thread of one k-step's A and B tiles
constexpr int GNA = (GBM * GBK) / TTB_THREADS;
constexpr int GNB = (GBK * GBN + TTB_THREADS - 1) / TTB_THREADS;
static_assert(GNA * TTB_THREADS == GBM * GBK, "A tile loads must divide evenly");

struct GemmSmem {
  double a[GBK][GPITCH_A];  // a[k][m]
  double b[GBK][GPITCH_B];  // b[k][n]
};

// D += A(8x4, row) * B(4x8, col) in FP64; lane l holds A[l/4][l%4],
// B[l%4][l/4] and D[l/4][2(l%4) + {0,1}].
static __device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// GEMM output view whose row and column indices may each be split in two:
// (i, j) -> p + (i / rdiv) * rs_hi + (i % rdiv) * rs
//             + (j / cdiv) * cs_hi + (j % cdiv) * cs.
// A plain Mat converts to the unsplit form.  The split lets one product write
// a result whose two index groups interleave in memory (a tensor
// contraction's output permuted for the next contraction).
constexpr int kNoSplit = 1 << 30;

// Division of 0 <= n < 2^31 by an invariant d >= 1 as a multiply and a
// shift (Granlund and Montgomery, "Division by invariant integers using
// multiplication", 1994, theorem 4.2 with N = 32): with l = ceil(log2 d)
// and m = floor(2^32 (2^l - d) / d) + 1 (below 2^32),
// n / d = (mulhi(m, n) + n) >> l, the sum staying below 2^32 for n < 2^31.
// The split-index outputs divide every output index by their split sizes.
struct FastDiv {
  uint32_t m;
  int l, d;
  __device__ FastDiv() : m(1), l(0), d(1) {}
  __device__ explicit FastDiv(int d_) : d(d_) {
    l = 32 - __clz(d_ - 1);
    m = (uint32_t)(((1ull << 32) * ((1ull << l) - (unsigned long long)d_)) / (unsigned)d_ + 1);
  }
  __device__ __forceinline__ int div(int n) const {
    return (int)((__umulhi(m, (uint32_t)n) + (uint32_t)n) >> l);
  }
};

struct OMat {
  double* p;
  i64 rs, cs, rs_hi, cs_hi;
  int rdiv, cdiv;
  FastDiv rq, cq;  // rdiv and cdiv (when split)
  __device__ OMat(Mat m)
      : p(m.p), rs(m.rs), cs(m.cs), rs_hi(0), cs_hi(0), rdiv(kNoSplit), cdiv(kNoSplit) {}
  __device__ OMat(double* p_, int rdiv_, i64 rs_hi_, i64 rs_, int cdiv_, i64 cs_hi_, i64 cs_)
      : p(p_), rs(rs_), cs(cs_), rs_hi(rs_hi_), cs_hi(cs_hi_), rdiv(rdiv_), cdiv(cdiv_) {
    if (rdiv != kNoSplit) rq = FastDiv(rdiv);
    if (cdiv != kNoSplit) cq = FastDiv(cdiv);
  }
  __device__ __forceinline__ i64 row(int i) const {
    if (rdiv == kNoSplit) return i * rs;
    const int q = rq.div(i);
    return q * rs_hi + (i - q * rdiv) * rs;
  }
  __device__ __forceinline__ i64 col(int j) const {
    if (cdiv == kNoSplit) return j * cs;
    const int q = cq.div(j);
    return q * cs_hi + (j - q * cdiv) * cs;
  }
};

// C[m0:m0+GBM, n0:n0+64] = alpha * A * B + beta * C over the full K range.
// A is M x K, B is K x N.  beta == 0 never reads C.  The warps form a
// (TTB_WARPS / 4) x 4 grid of 32 x 16 warp tiles, each 4 x 2 MMA tiles of
// 8 x 8 (the tile is GBM = 8 * TTB_WARPS rows by 64 columns).  C_FIRST reads
// all of a thread's C before it writes any (16 registers more): the compiler
// cannot move a load past a store that may alias it, and a tile of small K waits
// for one entry after the other.
template <bool C_FIRST>
static __device__ __forceinline__ void cta_gemm_tile(CMat A, CMat B, const OMat& C, int M, int N, int K, int m0,
                                     int n0, double alpha, double beta, GemmSmem& sm) {
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
  const int g = lane >> 2, t = lane & 3;
  double acc[4][2][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  // loads walk the unit-stride direction of each operand when there is one
  const bool a_kfast = (A.cs == 1);
  const bool b_nfast = (B.cs == 1) || (B.rs != 1);
  double ra[GNA], rb[GNB];
  auto load = [&](int k0) {
#pragma unroll
    for (int e = 0; e < GNA; ++e) {
      int idx = tid + e * TTB_THREADS;
      int mm, kk;
      if (a_kfast) { kk = idx % GBK; mm = idx / GBK; } else { mm = idx % GBM; kk = idx / GBM; }
      int gm = m0 + mm, gk = k0 + kk;
      ra[e] = (gm < M && gk < K) ? A(gm, gk) : 0.0;
    }
#pragma unroll
    for (int e = 0; e < GNB; ++e) {
      int idx = tid + e * TTB_THREADS;
      if (idx >= GBK * GBN) break;
      int nn, kb;
      if (b_nfast) { nn = idx % GBN; kb = idx / GBN; } else { kb = idx % GBK; nn = idx / GBK; }
      int gn = n0 + nn, gk2 = k0 + kb;
      rb[e] = (gn < N && gk2 < K) ? B(gk2, gn) : 0.0;
    }
  };
  auto store = [&]() {
#pragma unroll
    for (int e = 0; e < GNA; ++e) {
      int idx = tid + e * TTB_THREADS;
      int mm, kk;
      if (a_kfast) { kk = idx % GBK; mm = idx / GBK; } else { mm = idx % GBM; kk = idx / GBM; }
      sm.a[kk][mm] = ra[e];
    }
#pragma unroll
    for (int e = 0; e < GNB; ++e) {
      int idx = tid + e * TTB_THREADS;
      if (idx >= GBK * GBN) break;
      int nn, kb;
      if (b_nfast) { nn = idx % GBN; kb = idx / GBN; } else { kb = idx % GBK; nn = idx / GBK; }
      sm.b[kb][nn] = rb[e];
    }
  };

  if (K > 0) load(0);
  for (int k0 = 0; k0 < K; k0 += GBK) {
    __syncthreads();  // previous compute finished with the tile
    store();
    __syncthreads();
    if (k0 + GBK < K) load(k0 + GBK);  // prefetch overlaps the MMAs below
#pragma unroll
    for (int kk = 0; kk < GBK; kk += 4) {
      double av[4], bv[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = sm.a[kk + t][wm + 8 * i + g];
#pragma unroll
      for (int j = 0; j < 2; ++j) bv[j] = sm.b[kk + t][wn + 8 * j + g];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
    }
  }
  i64 coff[2][2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) coff[j][h] = C.col(n0 + wn + 8 * j + 2 * t + h);
  double old[C_FIRST ? 4 : 1][2][2];
  if constexpr (C_FIRST) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int gm = m0 + wm + 8 * i + g;
      const double* crow = C.p + C.row(gm);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          old[i][j][h] = beta != 0.0 && gm < M && n0 + wn + 8 * j + 2 * t + h < N
                             ? crow[coff[j][h]] : 0.0;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + wm + 8 * i + g;
    if (gm >= M) continue;
    double* crow = C.p + C.row(gm);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gn = n0 + wn + 8 * j + 2 * t + h;
        if (gn >= N) continue;
        double v = alpha * acc[i][j][h];
        if (beta != 0.0) {
          if constexpr (C_FIRST) v = fma(beta, old[i][j][h], v);
          else v = fma(beta, crow[coff[j][h]], v);
        }
        crow[coff[j][h]] = v;
      }
  }
  __syncthreads();  // callers may reuse the staging buffers right away
}

// Whole product, looping over all output tiles with the one block.
static __device__ __noinline__ void cta_gemm(CMat A, CMat B, OMat C, int M, int N, int K, double alpha, double beta,
                         GemmSmem& sm) {
  for (int m0 = 0; m0 < M; m0 += GBM)
    for (int n0 = 0; n0 < N; n0 += GBN)
      cta_gemm_tile<true>(A, B, C, M, N, K, m0, n0, alpha, beta, sm);
}

// ---------------------------------------------------------------------------
// Pipelined GEMM: the same 64x64 tiles and MMA fragments as cta_gemm_tile,
// with operands copied by cp.async into a ring of GSTAGES shared-memory
// stages.  The (output tile, k-tile) steps of the whole product form one
// sequence, so loads run GSTAGES - 1 steps ahead across tile boundaries and
// a tile's first operands arrive while the previous tile is finishing.
// ``ring`` holds GSTAGES * GSTAGE_D doubles of shared memory; its
// first stage has the layout of GemmSmem.  A and B may be anywhere (shared
// operands take the one-stage path); C must not overlap the ring.
// ---------------------------------------------------------------------------

constexpr int GSTAGES = 3;
constexpr int GSTAGE_D = GBK * (GPITCH_A + GPITCH_B);

static __device__ __forceinline__ void cp_async8(double* dst, const double* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int sz = ok ? 8 : 0;  // 0 bytes read: the destination is zero-filled
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(sz)
               : "memory");
}
static __device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
static __device__ __forceinline__ void cp_async_wait_ahead() {
  asm volatile("cp.async.wait_group %0;" ::"n"(GSTAGES - 2) : "memory");
}
static __device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Split-K product for a small output and a long K range (the V^T V and
// V^T C products of the blocked factorisations: M, N <= 48, one of them <= 16,
// K in the thousands), where the tiled pipeline would spend one
// synchronised k-step per 16 of K on a mostly empty 64 x 64 tile.  Each warp
// takes a contiguous K slice and accumulates the whole MI*8 x NJ*8 product
// in DMMA fragments from direct global loads (32-byte runs along K), with no
// block barrier in the loop; the eight partial products are then added in
// warp order through ``scratch`` (TTB_WARPS * M * N doubles of shared
// memory), so the result does not depend on scheduling.
template <int MI, int NJ>
static __device__ __noinline__ void cta_gemm_skinny(CMat A, CMat B, OMat C, int M, int N, int K,
                                                    double alpha, double beta, double* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int mi = (M + 7) >> 3, nj = (N + 7) >> 3;
  double acc[MI][NJ][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int kper = (((K + TTB_WARPS - 1) / TTB_WARPS) + 3) & ~3;
  const int kb = warp * kper, ke = min(K, kb + kper);
  const double* ap[MI];
  const double* bp[NJ];
  bool aok[MI], bok[NJ];
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    aok[i] = 8 * i + g < M;
    ap[i] = A.p + (aok[i] ? (i64)(8 * i + g) * A.rs : 0);
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    bok[j] = 8 * j + g < N;
    bp[j] = B.p + (bok[j] ? (i64)(8 * j + g) * B.cs : 0);
  }
#pragma unroll 4
  for (int k0 = kb; k0 < ke; k0 += 4) {
    const int kk = k0 + t;
    const bool okk = kk < ke;
    double av[MI], bv[NJ];
#pragma unroll
    for (int i = 0; i < MI; ++i) av[i] = (okk && aok[i]) ? ap[i][(i64)kk * A.cs] : 0.0;
#pragma unroll
    for (int j = 0; j < NJ; ++j) bv[j] = (okk && bok[j]) ? bp[j][(i64)kk * B.rs] : 0.0;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        if (i < mi && j < nj) dmma_8x8x4(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
  }
  const int mn = M * N;
  double* mine = scratch + (i64)warp * mn;
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = 8 * i + g, col = 8 * j + 2 * t + h;
        if (r < M && col < N) mine[r * N + col] = acc[i][j][h];
      }
  __syncthreads();
  for (int e = threadIdx.x; e < mn; e += TTB_THREADS) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < TTB_WARPS; ++w) v += scratch[(i64)w * mn + e];
    const int r = e / N, col = e % N;
    double* cp = C.p + C.row(r) + C.col(col);
    v *= alpha;
    if (beta != 0.0) v = fma(beta, *cp, v);
    *cp = v;
  }
  __syncthreads();  // callers may reuse the scratch and read C right away
}

// Output shapes and K lengths that take the split-K path.
constexpr int kSkinnyK = 128;
static_assert(TTB_WARPS * 16 * 48 <= GSTAGES * GSTAGE_D, "split-K scratch must fit the ring");

// True when cta_gemm_pipe takes its tiled path for these operands (not the
// one-stage tile or the split-K product), the path whose output tiles may be
// shared out between the blocks of a cluster (tile0, tstride below).
static __device__ __forceinline__ bool gemm_pipe_tiled(CMat A, CMat B, int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0 || __isShared(A.p) || __isShared(B.p)) return false;
  if (K >= kSkinnyK && A.cs == 1 && B.rs == 1 && ((M <= 16 && N <= 48) || (M <= 48 && N <= 16)))
    return false;
  return true;
}

// The tiled path of cta_gemm_pipe for TM x TN output tiles (eight warps of
// 32 x 16, TN / 16 of them along N), K staged TK at a time through an
// NS-stage cp.async ring.  Each output element accumulates its K range in
// steps of four (one DMMA each) in increasing order whatever the tile
// shape, so every shape gives the same bits.
template <int TM, int TN, int TK, int NS>
static __device__ __forceinline__ void gemm_tiles(CMat A, CMat B, OMat C, int M, int N, int K,
                                                  double alpha, double beta, double* ring,
                                                  int tile0, int tstride) {
  static_assert(TTB_WARPS == 8 && TM * TN == 8 * 32 * 16, "eight warps of 32 x 16");
  static_assert(TK % 4 == 0, "K steps of four");
  constexpr int PA = TM + 4, PB = TN + 4;  // pitches: see GPITCH_A
  constexpr int SD = TK * (PA + PB);       // doubles of a stage
  static_assert(NS * SD <= GSTAGES * GSTAGE_D, "stages must fit the ring");
  constexpr int NA = (TM * TK) / TTB_THREADS;
  constexpr int NB = (TK * TN + TTB_THREADS - 1) / TTB_THREADS;
  static_assert(NA * TTB_THREADS == TM * TK, "A tile loads must divide evenly");
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int wm = (warp / (TN / 16)) * 32, wn = (warp % (TN / 16)) * 16;
  const int g = lane >> 2, t = lane & 3;
  const int tn = (N + TN - 1) / TN;
  const int nk = (K + TK - 1) / TK;
  const int tiles = ((M + TM - 1) / TM) * tn;
  const int nloc = tile0 < tiles ? (tiles - tile0 + tstride - 1) / tstride : 0;
  const int total = nloc * nk;
  const bool a_kfast = (A.cs == 1);
  const bool b_nfast = (B.cs == 1) || (B.rs != 1);
  auto issue = [&](int step) {
    if (step < total) {
      const int tile = tile0 + (step / nk) * tstride, kt = step % nk;
      const int m0 = (tile / tn) * TM, n0 = (tile % tn) * TN, k0 = kt * TK;
      double* sa = ring + (step % NS) * SD;
      double* sb = sa + TK * PA;
#pragma unroll
      for (int e = 0; e < NA; ++e) {
        const int idx = tid + e * TTB_THREADS;
        int mm, kk;
        if (a_kfast) { kk = idx % TK; mm = idx / TK; } else { mm = idx % TM; kk = idx / TM; }
        const int gm = m0 + mm, gk = k0 + kk;
        const bool oka = gm < M && gk < K;
        cp_async8(sa + kk * PA + mm, oka ? A.p + gm * A.rs + gk * A.cs : A.p, oka);
      }
#pragma unroll
      for (int e = 0; e < NB; ++e) {
        const int idx = tid + e * TTB_THREADS;
        if (idx >= TK * TN) break;
        int nn, kb;
        if (b_nfast) { nn = idx % TN; kb = idx / TN; } else { kb = idx % TK; nn = idx / TK; }
        const int gn = n0 + nn, gk2 = k0 + kb;
        const bool okb = gn < N && gk2 < K;
        cp_async8(sb + kb * PB + nn, okb ? B.p + gk2 * B.rs + gn * B.cs : B.p, okb);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int st = 0; st < NS - 1; ++st) issue(st);
  double acc[4][2][2];
  for (int step = 0; step < total; ++step) {
    const int kt = step % nk;
    if (kt == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
    __syncthreads();  // this step's operands landed; the previous step's reads are done
    issue(step + NS - 1);
    const double* sa = ring + (step % NS) * SD;
    const double* sb = sa + TK * PA;
    const int kvalid = K - kt * TK;  // the last slab's groups of four past K are zeros: skipped
#pragma unroll
    for (int kk = 0; kk < TK; kk += 4) {
      if (kk >= kvalid) break;
      double av[4], bv[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = sa[(kk + t) * PA + wm + 8 * i + g];
#pragma unroll
      for (int j = 0; j < 2; ++j) bv[j] = sb[(kk + t) * PB + wn + 8 * j + g];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
    }
    if (kt == nk - 1) {
      const int tile = tile0 + (step / nk) * tstride;
      const int m0 = (tile / tn) * TM, n0 = (tile % tn) * TN;
      i64 coff[2][2];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) coff[j][h] = C.col(n0 + wn + 8 * j + 2 * t + h);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int gm = m0 + wm + 8 * i + g;
        if (gm >= M) continue;
        double* crow = C.p + C.row(gm);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int gn = n0 + wn + 8 * j + 2 * t + h;
            if (gn >= N) continue;
            double v = alpha * acc[i][j][h];
            if (beta != 0.0) v = fma(beta, crow[coff[j][h]], v);
            crow[coff[j][h]] = v;
          }
      }
    }
  }
  cp_async_wait_all();
}


// ``tile0`` and ``tstride``: on the tiled path, compute only the output
// tiles tile0, tile0 + tstride, ... (row-major tile order), each exactly as
// the whole product computes it.
static __device__ __noinline__ void cta_gemm_pipe(CMat A, CMat B, OMat C, int M, int N, int K,
                                                  double alpha, double beta, double* ring,
                                                  int tile0 = 0, int tstride = 1) {
  if (M <= 0 || N <= 0) return;
  // cp.async copies from global memory only: operands in shared memory, and
  // K == 0 (C = beta * C), go through the one-stage tile
  if (K <= 0 || __isShared(A.p) || __isShared(B.p)) {
    cta_gemm(A, B, C, M, N, K, alpha, beta, *reinterpret_cast<GemmSmem*>(ring));
    return;
  }
  // (operands contiguous along K only: the split-K loads read 32-byte runs of K)
  if (K >= kSkinnyK && A.cs == 1 && B.rs == 1) {
    if (M <= 16 && N <= 48) {
      cta_gemm_skinny<2, 6>(A, B, C, M, N, K, alpha, beta, ring);
      return;
    }
    if (M <= 48 && N <= 16) {
      cta_gemm_skinny<6, 2>(A, B, C, M, N, K, alpha, beta, ring);
      return;
    }
  }
  // 128 x 32 tiles where they cover the output with at least a fifth less
  // padded area than 64 x 64 tiles (N <= 32 with M > 64, or N just above a
  // multiple of 64, as 65-96): their operand loads per MMA are a fifth
  // higher, so a smaller saving would not pay
  const i64 pad64 = (i64)((M + 63) / 64 * 64) * ((N + 63) / 64 * 64);
  const i64 pad128 = (i64)((M + 127) / 128 * 128) * ((N + 31) / 32 * 32);
  if (5 * pad128 <= 4 * pad64)
    gemm_tiles<128, 32, 12, 3>(A, B, C, M, N, K, alpha, beta, ring, tile0, tstride);
  else
    gemm_tiles<GBM, GBN, GBK, GSTAGES>(A, B, C, M, N, K, alpha, beta, ring, tile0, tstride);
  __syncthreads();  // callers may reuse the ring and read C right away
}

// The blocked factorisations take an optional GEMM ring: with one, their
// trailing-update products are pipelined (cta_gemm_pipe), else they use the
// one-stage tile in ``gsm``.
static __device__ __forceinline__ void gemm_sel(CMat A, CMat B, OMat C, int M, int N, int K,
                                                double alpha, double beta, GemmSmem& gsm,
                                                double* ring) {
  if (ring)
    cta_gemm_pipe(A, B, C, M, N, K, alpha, beta, ring);
  else
    cta_gemm(A, B, C, M, N, K, alpha, beta, gsm);
}

}  // namespace ttb
