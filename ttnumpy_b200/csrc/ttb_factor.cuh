// Factorisations executed by one thread block (ttb_factor.cu): Householder
// QR, thin SVD by one-sided Jacobi, and Gaussian elimination with partial
// pivoting.  Every thread of the block calls them together; matrices may be
// in shared or in global memory.
//
// ``tiled`` chooses the register-tiled Householder steps and the
// preconditioned, register-blocked Jacobi iteration; false takes the
// column-by-column steps and the plain iteration.  The whole-solve kernel
// passes false: the rank decisions of its sweeps react to the last digits of
// a factorisation, and its solves are held to recorded trajectories.
#pragma once

#include "ttb_device.cuh"

namespace ttb {

constexpr int LNB = 16;   // panel width of the blocked factorisations
constexpr int YCH = 512;  // columns per chunk of the blocked trailing updates
constexpr int LNB2 = 64;  // outer panel width of the two-level R-only QR

__device__ void cta_qr(CMat A, int m, int k, double* W, i64 ldw, double* tau, Mat Q, Mat R,
                       double* red, bool tiled = true);
__device__ void cta_qr_blocked(CMat A, int m, int k, double* W, double* tau, Mat Q, Mat R,
                               double* Y, double* G, double* Tm, double* red, GemmSmem& gsm,
                               double* ring = nullptr, bool tiled = true);
__device__ void cta_qr_r_blocked2(CMat A, int m, int k, double* W, double* tau, Mat R,
                                  double* pool, double* red, double* ring);
__device__ int cta_svd_tall(CMat A, int m, int k, double* W, i64 ldw, double* tau, double* Bsq,
                            double* V, double* sv, int* order, int* flag, double* tau2, Mat U,
                            double* S, Mat Vh, double* red, bool tiled = true);
__device__ int cta_svd_tall_blocked(CMat A, int m, int k, double* W, double* tau, double* Bsq,
                                    double* V, double* sv, int* order, int* flag, double* tau2,
                                    Mat U, double* S, Mat Vh, double* Y, double* G, double* Tm,
                                    double* red, GemmSmem& gsm, double* ring = nullptr,
                                    bool tiled = true);
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

}  // namespace ttb
