// Factorisations executed by one thread block (ttb_factor.cu): Householder
// QR, thin SVD by one-sided Jacobi, and Gaussian elimination with partial
// pivoting.  Every thread of the block calls them together; matrices may be
// in shared or in global memory.
//
// TILED chooses the register-tiled Householder steps and the
// preconditioned, register-blocked Jacobi iteration; false takes the
// column-by-column steps and the plain iteration.  The whole-solve kernel
// takes false: the rank decisions of its sweeps react to the last digits of
// a factorisation, and its solves are held to recorded trajectories.
#pragma once

#include "ttb_device.cuh"

namespace ttb {

constexpr int LNB = 16;   // panel width of the blocked factorisations
constexpr int YCH = 512;  // columns per chunk of the blocked trailing updates
constexpr int LNB2 = 64;  // outer panel width of the two-level R-only QR

// W (column major, column step ldw) <- the m x k view A, reading along A's
// unit-stride direction.
static __device__ __forceinline__ void cta_load(CMat A, double* W, i64 ldw, int m, int k) {
  const int total = m * k;
  if (A.cs == 1) {
    for (int e = threadIdx.x; e < total; e += TTB_THREADS) {
      const int i = e / k, j = e - i * k;
      W[i + j * ldw] = A(i, j);
    }
  } else {
    for (int e = threadIdx.x; e < total; e += TTB_THREADS) {
      const int j = e / m, i = e - j * m;
      W[i + j * ldw] = A(i, j);
    }
  }
}

template <bool TILED>
__device__ void cta_qr(CMat A, int m, int k, double* W, i64 ldw, double* tau, Mat Q, Mat R,
                       double* red);
template <bool TILED>
__device__ void cta_qr_blocked(CMat A, int m, int k, double* W, double* tau, Mat Q, Mat R,
                               double* Y, double* G, double* Tm, double* red, GemmSmem& gsm,
                               double* ring = nullptr);
__device__ void cta_qr_r_blocked2(CMat A, int m, int k, double* W, double* tau, Mat R,
                                  double* pool, double* red, double* ring, int rank = 0,
                                  int size = 1);
template <bool TILED>
__device__ int cta_svd_tall(CMat A, int m, int k, double* W, i64 ldw, double* tau, double* Bsq,
                            double* V, double* sv, int* order, int* flag, double* tau2, Mat U,
                            double* S, Mat Vh, double* red);
template <bool TILED>
__device__ int cta_svd_tall_blocked(CMat A, int m, int k, double* W, double* tau, double* Bsq,
                                    double* V, double* sv, int* order, int* flag, double* tau2,
                                    Mat U, double* S, Mat Vh, double* Y, double* G, double* Tm,
                                    double* red, GemmSmem& gsm, double* ring = nullptr);

// cta_svd_tall_blocked in three kernels for large k (kClusterMin < k <=
// kClusterMax): before the Jacobi iteration, the iteration by a cluster of
// blocks (returns the sweeps, -1 at the cap), and after it; every matrix in
// global memory, flags three ints there.
constexpr int kClusterMin = 96, kClusterMax = 512;
__device__ void cta_svd_before(CMat A, int m, int k, double* W, double* tau, double* Bsq,
                               double* V, double* sv, int* order, int* flags, double* tau2, Mat U,
                               Mat Vh, double* Y, double* G, double* Tm, double* red,
                               GemmSmem& gsm);
__device__ int cluster_svd_iterate(bool left, bool right, int k, double* Bsq, double* V,
                                   int* flags);
__device__ void cta_svd_after(int m, int k, double* W, double* tau, double* Bsq, double* V,
                              double* sv, int* order, double* tau2, int* flag, Mat U, double* S,
                              Mat Vh, double* Y, double* G, double* Tm, double* red,
                              GemmSmem& gsm);
__device__ int cta_gepp_solve(double* W, i64 ld, double* b, int n, double* lbuf);
__device__ int cta_gepp_blocked(double* W, i64 ld, double* b, int n, double* panel, double* redv,
                                int* redi, int* ipiv, GemmSmem& gsm, double* ring = nullptr);

// Largest system cta_gepp_solve takes, and the doubles of its ``lbuf``.
constexpr int kLuWhole = 160;
__host__ __device__ constexpr int lu_buf_doubles(int n) { return 2 * ((n + 31) & ~31); }

// Doubles of the shared ``panel`` that cta_gepp_blocked needs for n unknowns
// (n <= kLuRows; beyond, LNB columns of n rows, in any memory): the panel at
// a pitch that spreads a fragment over the banks, and a strip of U12.
constexpr int kLuRows = 1024, kLuStrip = 128, kLuStripPitch = kLuStrip + 4;
__host__ __device__ constexpr int lu_pitch(int rows) { return ((rows + 15) & ~15) + 4; }
__host__ __device__ constexpr long long lu_panel_doubles(int n) {
  return n <= kLuRows ? LNB * (lu_pitch(n) + kLuStripPitch) : (long long)n * LNB;
}

// The steps of cta_gepp_blocked for n <= kLuRows (see there): for j0 = 0, LNB,
// ...: the panel, then its update (every block of a cluster, ``fetch`` where
// the panel was factored by another); at the end the back substitution.
__device__ int cta_gepp_panel(double* W, i64 ld, int n, int j0, double* pool, int* ipiv);
__device__ void cta_gepp_update(double* W, i64 ld, double* b, int n, int j0, double* pool,
                                const int* ipiv, bool fetch, int rank, int size);
__device__ void cta_back_substitute(const double* W, i64 ld, double* b, int n);

// Nodes of a tree of factorisations.  ``smem`` (may be NULL) holds node_smem
// doubles and is where the node's columns live meanwhile.
// cta_node_factor: Householder QR of the rows x k view A (rows <= 2048): the
// reflectors to W (column step ld, even) and tau, R (k x k, zero rows past
// ``rows``).  A may be W itself.
// cta_node_apply: columns c0 .. c0 + nc - 1 of X (rows x k) = the node's Q
// times [top; 0] (k x k, column step ktop), or times [I; 0] without top.
// cta_triangle_svd: SVD of the k x k upper-triangular R (column step k);
// ``work`` (triangle_svd_doubles) in any memory, Us a k x k scratch view for
// the case that both factors are wanted.  Vh may be NULL; ``top`` gets the
// left factor (column step k) unless it is NULL.
__host__ __device__ constexpr long long node_smem(int rows, int k) {
  return ((long long)((rows + 1) & ~1) + 2) * k;
}
__host__ __device__ constexpr long long triangle_svd_doubles(int k) {
  return 2LL * svd_step(k) * k + 3LL * k + 4;
}
__device__ void cta_node_factor(CMat A, int rows, int k, double* W, i64 ld, double* tau,
                                double* smem, Mat R);
__device__ void cta_node_apply(const double* W, i64 ld, int rows, int k, const double* tau,
                               double* smem, const double* top, i64 ktop, Mat X, int c0, int nc);
__device__ int cta_triangle_svd(const double* R, int k, double* work, Mat Us, double* S, Mat Vh,
                                double* top, double* red);

}  // namespace ttb
