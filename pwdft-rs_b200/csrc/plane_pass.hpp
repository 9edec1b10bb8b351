// Launchers of the two-stage passes (hpsi_plane.cu), one set per radix pair.
// The pairs are spread over translation units (plane_len_*.cu): the driver
// loads a unit's kernels together when one of them is first named, 0.07 ms
// apiece (all 184 in one unit: 17.6 ms of the first handle of a process), and
// a handle runs those of one or two lengths.
#pragma once

#include "plane_fft.cuh"

namespace pwgpu {

// The two-stage lengths: radix pairs (R0, R1) with R0 the pruned radix.
#define PW_PAIRS_A(X) X(4, 3) X(5, 3) X(4, 4) X(6, 3) X(4, 5)
#define PW_PAIRS_B(X) X(8, 3) X(5, 5) X(9, 3) X(6, 5) X(8, 4)
#define PW_PAIRS_C(X) X(4, 9) X(8, 5) X(9, 5) X(8, 6) X(10, 5)
#define PW_PAIRS_D(X) X(6, 9) X(6, 10) X(8, 8) X(8, 9) X(8, 10)
#define PW_PAIRS_E(X) X(9, 9) X(10, 9) X(8, 12) X(10, 10) X(12, 9) X(12, 10)
#define PW_PAIRS(X) PW_PAIRS_A(X) PW_PAIRS_B(X) PW_PAIRS_C(X) PW_PAIRS_D(X) PW_PAIRS_E(X)

constexpr int pair_id(int r0, int r1) { return r0 * 16 + r1; }

constexpr size_t kPlaneSmemMax = 227 * 1024;
constexpr int kZCols = 32;  // columns per block of the z kernels

// One plane pass: nb bands in groups of bpc, d2 planes, `smem` bytes of shared memory.
template <typename R> struct PlaneRun {
  cplx<R>* A;
  const R* vz;
  int nb, bpc, d2;
  PlaneGeo geo;
  const cplx<R>*twx, *twy;
  size_t smem;
};
// The columns of a z pass.
struct ZColumns {
  const int *start, *lo;
  int ncol, m2;
};

template <typename R, int R0, int R1> struct PlaneLen {
  // shared-memory opt-ins of the z kernels and of the square-plane kernels, on the current device
  static cudaError_t opt_in_z();
  static cudaError_t opt_in_square();
  static void zi(const double2* psi, long ldpsi, cplx<R>* A, int nb, const ZColumns& c, const cplx<R>* tw, cudaStream_t s);
  static void zf(const cplx<R>* A, const double2* psi, long ldpsi, double2* hpsi, long ldh, const double* kin,
                 double scale, int nb, const ZColumns& c, const cplx<R>* tw, cudaStream_t s);
  static void plane(const PlaneRun<R>& p, cudaStream_t s);
  // rho partials of p.nb bands in p.bpc-band groups (p.vz unused); R = double
  static void rho(const PlaneRun<R>& p, const double* fw, double* part, cudaStream_t s);
};

// The plane pass with run-time radix pairs px, py (plane_rt.cu); rows: rows of the plane buffer.
template <typename R> cudaError_t plane_rt_opt_in();
template <typename R> void plane_rt(const PlaneRun<R>& p, int rows, int px, int py, cudaStream_t s);

// Shared memory ahead of the plane in plane_rt.
struct alignas(16) PlaneShared {
  PlaneGeo g;
  int rows;  // rows of the plane buffer
};

}  // namespace pwgpu
