// The kernels of the two-stage passes for compile-time radix pairs (order and
// bounds of the passes: hpsi_plane.cu), and their launchers.
#pragma once

#include "plane_pass.hpp"

namespace pwgpu {

namespace {

// Threads of the square-plane pass: the widest x stage of the plane (d1
// butterflies for each of max(X0, X1) groups) in the fewest equal rounds of at
// most 324, so that no round of a stage is mostly idle; at least 128.
constexpr int plane_threads(int x0, int x1) {
  const int wide = x0 * x1 * (x0 > x1 ? x0 : x1);
  const int rounds = (wide + 323) / 324;
  const int t = (wide + rounds - 1) / rounds;
  return t < 128 ? 128 : t;
}

// The pass for planes with equal x and y lengths (every cubic grid): strides
// and divisions are constants.  What bounds it: the shared-memory data path,
// 7,240 (FP64) and 3,920 (FP32) wavefronts a plane at 72 x 72, 67 and 65 % of
// its peak rate, and the block barriers, a quarter of the warps' stalls with 2
// and 3 blocks an SM; the FP64 and FP32 pipes are busy 43 and 42 %, HBM 6 %.  160 bands on 72^3: 0.484 ms FP64 and 0.265 ms FP32, against 0.915 and
// 0.461 ms for the form with two planes of shared memory, a V(r) plane and
// eight stages (one and two blocks an SM).  Threads per block at 72 x 72:
// 216 0.484 / 0.262, 324 0.484 / 0.269, 432 0.590 / 0.285, 648 0.564 / 0.354 ms.
template <typename R, int X0, int X1>
__global__ void __launch_bounds__(plane_threads(X0, X1), sizeof(R) == 4 ? 3 : (X0 > 9 || X1 > 9 ? 1 : 2))
    k_plane(cplx<R>* A, const R* __restrict__ vz, int nb, int bpc, int d2, PlaneGeo gin,
            const cplx<R>* __restrict__ twx, const cplx<R>* __restrict__ twy) {
  using C = cplx<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int d0 = X0 * X1, d1 = d0, ld = d1 | 1;
  PlaneGeo g = gin;
  g.d0 = d0; g.d1 = d1; g.ld = ld;
  C* P = reinterpret_cast<C*>(smem_raw);
  C* TX = P + (g.d0 + (g.Xp > g.avail ? g.Xp - g.avail : 0)) * ld;
  C* TY = TX + d0;
  const int z = blockIdx.x, tid = threadIdx.x, T = blockDim.x;
  const long ncol = (long)g.Xp * g.Yp;
  for (int i = tid; i < d0; i += T) TX[i] = twx[i];
  for (int i = tid; i < d1; i += T) TY[i] = twy[i];
  launch_wait();
  launch_release();
  __syncthreads();
  const R* vp = vz + (long)z * d0 * d1;
  const int b0 = blockIdx.y * bpc, b1 = min(nb, b0 + bpc);
  for (int b = b0; b < b1; ++b) {
    C* Ab = A + ((long)b * d2 + z) * ncol;
    plane_ya<X0, X1>(Ab, P, g, TY, tid, T);
    plane_yb<X0, X1>(P, g, tid, T);
    plane_xa<X0, X1>(P, g, TX, tid, T);
    plane_xvx<X0, X1>(P, g, vp, TX, tid, T);
    plane_xd<X0, X1>(P, g, tid, T);
    plane_yc<X0, X1>(P, g, TY, tid, T);
    plane_yd<X0, X1>(Ab, P, g, tid, T);
  }
}

// Density: rho partials of one z-plane for a group of bands, y-inverse and
// x-inverse as in k_plane, the last x stage adding fw |psi(r)|^2 into the
// thread's registers (its butterflies are the same for every band).  part:
// [group][z][x][y]; the groups of bands fill the GPU, which one block per line
// tile, all bands in turn, did not: 20 bands on 36^3 took 59 us in three
// kernels (z, y, x with the sum: 8 + 8 + 44), now 4 + 8 + 4 us.
template <int X0, int X1>
__global__ void __launch_bounds__(plane_threads(X0, X1), X0 > 9 || X1 > 9 ? 1 : 2)
    k_plane_rho(const double2* __restrict__ A, const double* __restrict__ fw, int nb, int bpc, int d2, PlaneGeo gin,
                const double2* __restrict__ twx, const double2* __restrict__ twy, double* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int d0 = X0 * X1, d1 = d0, ld = d1 | 1, T = plane_threads(X0, X1);
  constexpr int kRounds = (X0 * d1 + T - 1) / T;
  PlaneGeo g = gin;
  g.d0 = d0; g.d1 = d1; g.ld = ld;
  double2* P = reinterpret_cast<double2*>(smem_raw);
  double2* TX = P + (g.d0 + (g.Xp > g.avail ? g.Xp - g.avail : 0)) * ld;
  double2* TY = TX + d0;
  const int z = blockIdx.x, tid = threadIdx.x;
  const long ncol = (long)g.Xp * g.Yp;
  for (int i = tid; i < d0; i += T) TX[i] = twx[i];
  for (int i = tid; i < d1; i += T) TY[i] = twy[i];
  double acc[kRounds][X1];
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
#pragma unroll
    for (int k = 0; k < X1; ++k) acc[r][k] = 0.0;
  const int b0 = blockIdx.y * bpc, b1 = min(nb, b0 + bpc);
  for (int b = b0; b < b1; ++b) {
    __syncthreads();  // the tables, and the previous band's readers
    plane_ya<X0, X1>(A + ((long)b * d2 + z) * ncol, P, g, TY, tid, T);
    plane_yb<X0, X1>(P, g, tid, T);
    plane_xa<X0, X1>(P, g, TX, tid, T);
    const double f = fw[b];
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int t = tid + r * T;
      if (t >= X0 * d1) break;
      const int k1 = fast_div(t, d1, g.md1), y = t - k1 * d1;
      const double2* base = P + X1 * k1 * ld + y;
      double2 v[X1];
#pragma unroll
      for (int j = 0; j < X1; ++j) v[j] = base[j * ld];
      dft_n<X1, +1>(v);
#pragma unroll
      for (int k = 0; k < X1; ++k) acc[r][k] += f * (v[k].x * v[k].x + v[k].y * v[k].y);
    }
  }
  double* out = part + ((long)blockIdx.y * d2 + z) * d0 * d1;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int t = tid + r * T;
    if (t >= X0 * d1) break;
    const int k1 = fast_div(t, d1, g.md1), y = t - k1 * d1;
#pragma unroll
    for (int k = 0; k < X1; ++k) out[(k1 + X0 * k) * d1 + y] = acc[r][k];
  }
}

// The z kernels read psi and write H psi at the columns' own basis points (no
// scatter, no point lists) and hold one buffer of kZCols columns; both stages
// run in one round of threads.  Bound by L2 latency and traffic (psi or the
// planes in, the planes or H psi out).  160 bands on 72^3: 97 + 101 us FP64, 57
// + 60 us FP32, against 236 + 213 and 132 + 127 us with two buffers, a zero
// fill and a scatter pass.
// K1: z-inverse of kZCols sphere columns per block.  Column c holds the basis
// points col_start[c] .. col_start[c + 1] - 1 at consecutive n2 from col_lo[c].
template <typename R, int Z0, int Z1>
__global__ void __launch_bounds__(kZCols * (Z0 > Z1 ? Z0 : Z1))
    k_zi(const double2* psi, long ldpsi, cplx<R>* A, const int* __restrict__ col_start,
         const int* __restrict__ col_lo, int ncol, int m2, const cplx<R>* __restrict__ tw) {
  using C = cplx<R>;
  constexpr int d2 = Z0 * Z1, ld = d2 | 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int c0 = blockIdx.x * kZCols, tid = threadIdx.x;
  launch_wait();
  launch_release();
  const double2* ps = psi + (long)blockIdx.y * ldpsi;
  if (tid < kZCols * Z1) {
    const int c = tid / Z1, j = tid - c * Z1, col = c0 + c;
    C v[Z0];
#pragma unroll
    for (int r = 0; r < Z0; ++r) v[r] = cmake<C>(0.0, 0.0);
    if (col < ncol) {
      const int s = col_start[col], cnt = col_start[col + 1] - s, lo = col_lo[col];
#pragma unroll
      for (int r = 0; r < Z0; ++r)
        if (slot_live<Z0>(r)) {
          const int e = j + Z1 * r;
          const int k = (e <= m2 ? e : e - d2) - lo;  // n2 - lo; the gap between falls outside [0, cnt)
          if ((unsigned)k < (unsigned)cnt && (e <= m2 || e >= d2 - m2)) {
            const double2 x = ps[s + k];
            v[r] = cmake<C>(x.x, x.y);
          }
        }
    }
    bf_a<Z0>(v, j, tw);
    C* row = buf + c * ld + j;
#pragma unroll
    for (int k = 0; k < Z0; ++k) row[Z1 * k] = v[k];
  }
  __syncthreads();
  if (tid < kZCols * Z0) {
    const int c = tid % kZCols, k1 = tid / kZCols, col = c0 + c;
    const C* row = buf + c * ld + Z1 * k1;
    C v[Z1];
#pragma unroll
    for (int j = 0; j < Z1; ++j) v[j] = row[j];
    dft_n<Z1, +1>(v);
    if (col < ncol) {
      C* out = A + ((long)blockIdx.y * d2 + k1) * ncol + col;
#pragma unroll
      for (int k = 0; k < Z1; ++k) out[(long)Z0 * k * ncol] = v[k];
    }
  }
}

// K5: z-forward of kZCols columns, Hpsi = value / N + T psi at the sphere points.
template <typename R, int Z0, int Z1>
__global__ void __launch_bounds__(kZCols * (Z0 > Z1 ? Z0 : Z1))
    k_zf(const cplx<R>* A, const double2* __restrict__ psi, long ldpsi, double2* hpsi, long ldh,
         const double* __restrict__ kin, double scale, const int* __restrict__ col_start,
         const int* __restrict__ col_lo, int ncol, int m2, const cplx<R>* __restrict__ tw) {
  using C = cplx<R>;
  constexpr int d2 = Z0 * Z1, ld = d2 | 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int c0 = blockIdx.x * kZCols, tid = threadIdx.x;
  launch_wait();
  launch_release();
  if (tid < kZCols * Z0) {
    const int c = tid % kZCols, k1 = tid / kZCols, col = c0 + c;
    C v[Z1];
    const C* in = A + ((long)blockIdx.y * d2 + k1) * ncol + col;
#pragma unroll
    for (int k = 0; k < Z1; ++k) v[k] = col < ncol ? in[(long)Z0 * k * ncol] : cmake<C>(0.0, 0.0);
    bf_c<Z1>(v, k1, tw);
    C* row = buf + c * ld + Z1 * k1;
#pragma unroll
    for (int m = 0; m < Z1; ++m) row[m] = v[m];
  }
  __syncthreads();
  if (tid < kZCols * Z1) {
    const int c = tid / Z1, m = tid - c * Z1, col = c0 + c;
    if (col >= ncol) return;
    const C* row = buf + c * ld + m;
    const int s = col_start[col], cnt = col_start[col + 1] - s, lo = col_lo[col];
    C v[Z0];
#pragma unroll
    for (int k = 0; k < Z0; ++k) v[k] = row[Z1 * k];
    dft_n<Z0, -1>(v);
    const double2* ps = psi + (long)blockIdx.y * ldpsi + s;
    double2* hs = hpsi + (long)blockIdx.y * ldh + s;
#pragma unroll
    for (int q = 0; q < Z0; ++q)
      if (slot_live<Z0>(q)) {
        const int e = m + Z1 * q;
        const int k = (e <= m2 ? e : e - d2) - lo;
        if ((unsigned)k < (unsigned)cnt && (e <= m2 || e >= d2 - m2)) {
          const double2 p = ps[k];
          const double t = kin[s + k];
          hs[k] = make_double2((double)v[q].x * scale + t * p.x, (double)v[q].y * scale + t * p.y);
        }
      }
  }
}

}  // namespace

template <typename K> cudaError_t plane_opt_in(K* kern, size_t bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <typename R, int R0, int R1> cudaError_t PlaneLen<R, R0, R1>::opt_in_z() {
  const size_t bytes = (size_t)kZCols * ((R0 * R1) | 1) * sizeof(cplx<R>);
  const cudaError_t e = plane_opt_in(k_zi<R, R0, R1>, bytes);
  return e == cudaSuccess ? plane_opt_in(k_zf<R, R0, R1>, bytes) : e;
}

template <typename R, int R0, int R1> cudaError_t PlaneLen<R, R0, R1>::opt_in_square() {
  cudaError_t e = plane_opt_in(k_plane<R, R0, R1>, kPlaneSmemMax);
  if constexpr (sizeof(R) == sizeof(double))
    if (e == cudaSuccess) e = plane_opt_in(k_plane_rho<R0, R1>, kPlaneSmemMax);
  return e;
}

template <typename R, int R0, int R1>
void PlaneLen<R, R0, R1>::zi(const double2* psi, long ldpsi, cplx<R>* A, int nb, const ZColumns& c, const cplx<R>* tw,
                             cudaStream_t s) {
  launch_early(k_zi<R, R0, R1>, dim3((c.ncol + kZCols - 1) / kZCols, nb), kZCols * (R0 > R1 ? R0 : R1),
               (size_t)kZCols * ((R0 * R1) | 1) * sizeof(cplx<R>), s, psi, ldpsi, A, c.start, c.lo, c.ncol, c.m2, tw);
  count_launch();
}

template <typename R, int R0, int R1>
void PlaneLen<R, R0, R1>::zf(const cplx<R>* A, const double2* psi, long ldpsi, double2* hpsi, long ldh,
                             const double* kin, double scale, int nb, const ZColumns& c, const cplx<R>* tw,
                             cudaStream_t s) {
  launch_early(k_zf<R, R0, R1>, dim3((c.ncol + kZCols - 1) / kZCols, nb), kZCols * (R0 > R1 ? R0 : R1),
               (size_t)kZCols * ((R0 * R1) | 1) * sizeof(cplx<R>), s, A, psi, ldpsi, hpsi, ldh, kin, scale, c.start,
               c.lo, c.ncol, c.m2, tw);
  count_launch();
}

template <typename R, int R0, int R1> void PlaneLen<R, R0, R1>::plane(const PlaneRun<R>& p, cudaStream_t s) {
  launch_early(k_plane<R, R0, R1>, dim3(p.d2, (p.nb + p.bpc - 1) / p.bpc), plane_threads(R0, R1), p.smem, s, p.A, p.vz,
               p.nb, p.bpc, p.d2, p.geo, p.twx, p.twy);
  count_launch();
}

template <typename R, int R0, int R1>
void PlaneLen<R, R0, R1>::rho(const PlaneRun<R>& p, const double* fw, double* part, cudaStream_t s) {
  if constexpr (sizeof(R) == sizeof(double)) {
    k_plane_rho<R0, R1><<<dim3(p.d2, (p.nb + p.bpc - 1) / p.bpc), plane_threads(R0, R1), p.smem, s>>>(
        p.A, fw, p.nb, p.bpc, p.d2, p.geo, p.twx, p.twy, part);
    count_launch();
  }
}

#define PW_PLANE_LEN(r0, r1)                \
  template struct PlaneLen<double, r0, r1>; \
  template struct PlaneLen<float, r0, r1>;

}  // namespace pwgpu
