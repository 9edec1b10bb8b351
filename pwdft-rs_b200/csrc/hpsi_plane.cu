// Local part of H|psi> on grids whose axes are two-stage lengths: kinetic term
// plus V_eff through sphere-pruned FFTs in three kernels per chunk of bands
// (the matrix-free form of scf/potentials.rs:163-190, see hpsi.cu):
//   k_zi     psi(G) -> z-inverse of the sphere columns, z-major planes A
//   k_plane  per z-plane, in place in shared memory: y-inverse, x-inverse,
//            V(r), x-forward, y-forward, the sphere rows back to A
//   k_zf     z-forward, sphere points, 1/N, + T psi
// The stage order (plane_fft.cuh) joins the last x-inverse stage, the product
// and the first x-forward stage in registers and needs one plane of shared
// memory, not two.
#include <cstdint>

#include <algorithm>
#include <mutex>
#include <set>
#include <string>

#include "handle.hpp"
#include "plane_fft.cuh"

namespace pwgpu {

namespace {

// The two-stage lengths: radix pairs (R0, R1) with R0 the pruned radix.
#define PW_PAIRS(X)                                                                                              \
  X(4, 3) X(5, 3) X(4, 4) X(6, 3) X(4, 5) X(8, 3) X(5, 5) X(9, 3) X(6, 5) X(8, 4) X(4, 9) X(8, 5) X(9, 5) X(8, 6) \
  X(10, 5) X(6, 9) X(6, 10) X(8, 8) X(8, 9) X(8, 10) X(9, 9) X(10, 9) X(8, 12) X(10, 10) X(12, 9) X(12, 10)

constexpr size_t kPlaneSmemMax = 227 * 1024;
constexpr int kZCols = 32;  // columns per block of the z kernels

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
// and divisions are constants.  What bounds it: shared-memory wavefronts (41k
// complex accesses a plane at 72 x 72) and the FP64 or FP32 pipe, about
// equally, with the block barriers hidden by 2 (FP64) or 3 (FP32) blocks an
// SM.  160 bands on 72^3: 0.484 ms FP64 and 0.265 ms FP32, against 0.915 and
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

// The same pass with the radix pairs of x and y chosen at run time, each phase
// a function of its own (called once per phase and band), for planes whose x
// and y lengths differ; on a 72 x 72 plane it takes 1.05 (FP64) and 1.09
// (FP32) times k_plane.
struct alignas(16) PlaneShared {
  PlaneGeo g;
  int rows;  // rows of the plane buffer
};

template <typename R> __device__ __forceinline__ cplx<R>* plane_buf(PlaneGeo& g, cplx<R>*& TX, cplx<R>*& TY) {
  using C = cplx<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PlaneShared* sh = reinterpret_cast<const PlaneShared*>(smem_raw);
  g = sh->g;
  C* P = reinterpret_cast<C*>(smem_raw + sizeof(PlaneShared));
  TX = P + sh->rows * g.ld;
  TY = TX + g.d0;
  return P;
}
template <typename R, int R0, int R1> __device__ __noinline__ void rt_y_inv(const cplx<R>* Ab) {
  PlaneGeo g;
  cplx<R>*TX, *TY, *P = plane_buf<R>(g, TX, TY);
  plane_ya<R0, R1>(Ab, P, g, TY, threadIdx.x, blockDim.x);
  plane_yb<R0, R1>(P, g, threadIdx.x, blockDim.x);
}
template <typename R, int R0, int R1> __device__ __noinline__ void rt_x(const R* vp) {
  PlaneGeo g;
  cplx<R>*TX, *TY, *P = plane_buf<R>(g, TX, TY);
  plane_xa<R0, R1>(P, g, TX, threadIdx.x, blockDim.x);
  plane_xvx<R0, R1>(P, g, vp, TX, threadIdx.x, blockDim.x);
  plane_xd<R0, R1>(P, g, threadIdx.x, blockDim.x);
}
template <typename R, int R0, int R1> __device__ __noinline__ void rt_y_fwd(cplx<R>* Ab) {
  PlaneGeo g;
  cplx<R>*TX, *TY, *P = plane_buf<R>(g, TX, TY);
  plane_yc<R0, R1>(P, g, TY, threadIdx.x, blockDim.x);
  plane_yd<R0, R1>(Ab, P, g, threadIdx.x, blockDim.x);
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

// rho[x][y][z] += sum over the groups, in order, of part[g][z][x][y]; 32 x 32 tiles of (y, z) turned in shared memory.
__global__ void __launch_bounds__(256) k_rho_add(const double* __restrict__ part, int groups, int d0, int d1, int d2,
                                                 double* __restrict__ rho) {
  __shared__ double tile[32][33];
  const int x = blockIdx.x, y0 = blockIdx.y * 32, z0 = blockIdx.z * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long n = (long)d0 * d1 * d2;
  for (int r = ty; r < 32; r += 8) {
    const int y = y0 + tx, z = z0 + r;
    if (y >= d1 || z >= d2) continue;
    double s = 0.0;
    for (int g = 0; g < groups; ++g) s += part[g * n + ((long)z * d0 + x) * d1 + y];
    tile[r][tx] = s;
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int y = y0 + r, z = z0 + tx;
    if (y < d1 && z < d2) rho[((long)x * d1 + y) * d2 + z] += tile[tx][r];
  }
}

constexpr int pair_id(int r0, int r1) { return r0 * 16 + r1; }

template <typename R>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 3 : 2)
    k_plane_rt(cplx<R>* A, const R* __restrict__ vz, int nb, int bpc, int d2, PlaneGeo gin, int rows,
               int px, int py, const cplx<R>* __restrict__ twx, const cplx<R>* __restrict__ twy) {
  using C = cplx<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PlaneShared* sh = reinterpret_cast<PlaneShared*>(smem_raw);
  if (threadIdx.x == 0) {
    sh->g = gin;
    sh->rows = rows;
  }
  C* TX = reinterpret_cast<C*>(smem_raw + sizeof(PlaneShared)) + rows * gin.ld;
  C* TY = TX + gin.d0;
  const int z = blockIdx.x;
  for (int i = threadIdx.x; i < gin.d0; i += blockDim.x) TX[i] = twx[i];
  for (int i = threadIdx.x; i < gin.d1; i += blockDim.x) TY[i] = twy[i];
  launch_wait();
  launch_release();
  __syncthreads();
  const R* vp = vz + (long)z * gin.d0 * gin.d1;
  const long ncol = (long)gin.Xp * gin.Yp;
  const int b0 = blockIdx.y * bpc, b1 = min(nb, b0 + bpc);
  for (int b = b0; b < b1; ++b) {
    C* Ab = A + ((long)b * d2 + z) * ncol;
    switch (py) {
#define PW_CASE(r0, r1) case pair_id(r0, r1): rt_y_inv<R, r0, r1>(Ab); break;
      PW_PAIRS(PW_CASE)
#undef PW_CASE
    }
    switch (px) {
#define PW_CASE(r0, r1) case pair_id(r0, r1): rt_x<R, r0, r1>(vp); break;
      PW_PAIRS(PW_CASE)
#undef PW_CASE
    }
    switch (py) {
#define PW_CASE(r0, r1) case pair_id(r0, r1): rt_y_fwd<R, r0, r1>(Ab); break;
      PW_PAIRS(PW_CASE)
#undef PW_CASE
    }
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

int pair_of(int L) {
  switch (L) {
#define PW_CASE(r0, r1) case r0 * r1: return pair_id(r0, r1);
    PW_PAIRS(PW_CASE)
#undef PW_CASE
    default: return -1;
  }
}

int plane_rows(const GridMaps& g) { return std::max(g.d[0], 2 * g.Xp); }

template <typename R> size_t plane_smem(const GridMaps& g) {
  return sizeof(PlaneShared) +
         ((size_t)plane_rows(g) * (g.d[1] | 1) + g.d[0] + g.d[1]) * sizeof(cplx<R>);
}

PlaneGeo geometry(const GridMaps& g) {
  PlaneGeo p;
  p.d0 = g.d[0];
  p.d1 = g.d[1];
  p.ld = g.d[1] | 1;
  p.Xp = g.Xp;
  p.Yp = g.Yp;
  p.m0 = g.m[0];
  p.m1 = g.m[1];
  p.avail = g.d[0] - g.Xp;
  p.mXp = div_magic(g.Xp);
  p.md1 = div_magic(g.d[1]);
  return p;
}

// Opt every kernel of this file into the shared memory it may need (per device).
Status configure() {
  static std::mutex mu;
  static std::set<int> done;
  int dev = 0;
  PW_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (done.count(dev)) return kOk;
  cudaError_t e = cudaSuccess;
  auto set = [&](const void* f, size_t bytes) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  set((const void*)k_plane_rt<double>, kPlaneSmemMax);
  set((const void*)k_plane_rt<float>, kPlaneSmemMax);
#define PW_CASE(r0, r1)                                                                        \
  set((const void*)k_plane<double, r0, r1>, kPlaneSmemMax);                                    \
  set((const void*)k_plane<float, r0, r1>, kPlaneSmemMax);                                     \
  set((const void*)k_plane_rho<r0, r1>, kPlaneSmemMax);                                        \
  set((const void*)k_zi<double, r0, r1>, (size_t)kZCols * ((r0 * r1) | 1) * sizeof(double2));  \
  set((const void*)k_zi<float, r0, r1>, (size_t)kZCols * ((r0 * r1) | 1) * sizeof(float2));    \
  set((const void*)k_zf<double, r0, r1>, (size_t)kZCols * ((r0 * r1) | 1) * sizeof(double2));  \
  set((const void*)k_zf<float, r0, r1>, (size_t)kZCols * ((r0 * r1) | 1) * sizeof(float2));
  PW_PAIRS(PW_CASE)
#undef PW_CASE
  if (e != cudaSuccess) return fail(kCuda, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  done.insert(dev);
  return kOk;
}

template <typename R> struct Tables;
template <> struct Tables<double> {
  static const double2* tw(const GridMaps& g, int a) { return g.tw64[a]; }
  static const double* vz(const Handle& h, int spin) { return h.veff_rz[spin]; }
};
template <> struct Tables<float> {
  static const float2* tw(const GridMaps& g, int a) { return g.tw32[a]; }
  static const float* vz(const Handle& h, int spin) { return h.veff_rz32[spin]; }
};

}  // namespace

Status plane_setup(Handle& h) {
  GridMaps& g = h.g;
  g.plane_ok = false;
  for (int a = 0; a < 3; ++a) {
    g.pair[a] = pair_of(g.d[a]);
    if (g.pair[a] < 0 || 4 * g.m[a] >= g.d[a]) return kOk;
  }
  if (!g.contiguous || plane_smem<double>(g) > kPlaneSmemMax) return kOk;
  Status st = configure();
  if (st != kOk) return st;
  g.plane_ok = true;
  return kOk;
}

template <typename R>
static void launch_zi(const Handle& h, const double2* psi, long ldpsi, cplx<R>* A, int nb, cudaStream_t s) {
  const GridMaps& g = h.g;
  const dim3 grid((g.ncol + kZCols - 1) / kZCols, nb);
  const size_t sm = (size_t)kZCols * (g.d[2] | 1) * sizeof(cplx<R>);
  switch (g.pair[2]) {
#define PW_CASE(r0, r1)                                                                                              \
  case pair_id(r0, r1):                                                                                              \
    launch_early(k_zi<R, r0, r1>, grid, kZCols*(r0 > r1 ? r0 : r1), sm, s, psi, ldpsi, A, g.col_start, g.col_lo,     \
                 g.ncol, g.m[2], Tables<R>::tw(g, 2));                                                               \
    break;
    PW_PAIRS(PW_CASE)
#undef PW_CASE
  }
  count_launch();
}

// rho += sum_b fw[b] |psi_b(r)|^2; the partial sums take work_b.
Status density_plane(Handle& h, const double2* psi, long ldpsi, int nb, const double* fw_dev, double* rho,
                     cudaStream_t s) {
  const GridMaps& g = h.g;
  const int d0 = g.d[0], d1 = g.d[1], d2 = g.d[2];
  double2* A = static_cast<double2*>(h.work_a);
  double* part = static_cast<double*>(h.work_b);
  const int cap = std::max(1, (int)((double)h.chunk * 2.0 * g.Xp / d0));  // groups that fit work_b
  const PlaneGeo geo = geometry(g);
  for (int c0 = 0; c0 < nb; c0 += h.chunk_a) {
    const int cnt = std::min(h.chunk_a, nb - c0);
    launch_zi<double>(h, psi + (long)c0 * ldpsi, ldpsi, A, cnt, s);
    int groups = std::min(std::min(cap, cnt), std::max(1, (4 * 148 + d2 - 1) / d2));
    const int bpc = (cnt + groups - 1) / groups;
    groups = (cnt + bpc - 1) / bpc;
    switch (g.pair[0]) {
#define PW_CASE(r0, r1)                                                                                            \
  case pair_id(r0, r1):                                                                                            \
    k_plane_rho<r0, r1><<<dim3(d2, groups), plane_threads(r0, r1), plane_smem<double>(g), s>>>(                    \
        A, fw_dev + c0, cnt, bpc, d2, geo, g.tw64[0], g.tw64[1], part);                                            \
    break;
      PW_PAIRS(PW_CASE)
#undef PW_CASE
    }
    count_launch();
    k_rho_add<<<dim3(d0, (d1 + 31) / 32, (d2 + 31) / 32), 256, 0, s>>>(part, groups, d0, d1, d2, rho);
    count_launch();
  }
  PW_CUDA_TRY(cudaGetLastError());
  return kOk;
}

template <typename R>
Status local_plane(Handle& h, int spin, int ik, const double2* psi, long ldpsi, int nb, double2* hpsi, long ldh,
                   cudaStream_t s, void* scratch, StageTimer* tm) {
  using C = cplx<R>;
  const GridMaps& g = h.g;
  C* A = static_cast<C*>(scratch);
  const C *tw0 = Tables<R>::tw(g, 0), *tw1 = Tables<R>::tw(g, 1), *tw2 = Tables<R>::tw(g, 2);
  const R* vz = Tables<R>::vz(h, spin);
  const dim3 zgrid((g.ncol + kZCols - 1) / kZCols, nb);
  const size_t zsm = (size_t)kZCols * (g.d[2] | 1) * sizeof(C);
  launch_zi<R>(h, psi, ldpsi, A, nb, s);
  mark(tm, 0, s);
  const PlaneGeo geo = geometry(g);
  const int d2 = g.d[2];
  const int bpc = std::max(1, std::min(8, (int)((long)nb * d2 / (148 * 8))));
  const dim3 pgrid(d2, (nb + bpc - 1) / bpc);
  if (g.pair[0] == g.pair[1]) {
    switch (g.pair[0]) {
#define PW_CASE(r0, r1)                                                                                       \
  case pair_id(r0, r1):                                                                                       \
    launch_early(k_plane<R, r0, r1>, pgrid, plane_threads(r0, r1), plane_smem<R>(g), s, A, vz, nb, bpc, d2,   \
                 geo, tw0, tw1);                                                                              \
    break;
      PW_PAIRS(PW_CASE)
#undef PW_CASE
    }
  } else {
    launch_early(k_plane_rt<R>, pgrid, 256, plane_smem<R>(g), s, A, vz, nb, bpc, d2, geo, plane_rows(g), g.pair[0],
                 g.pair[1], tw0, tw1);
  }
  count_launch();
  mark(tm, 2, s);
  switch (g.pair[2]) {
#define PW_CASE(r0, r1)                                                                                      \
  case pair_id(r0, r1):                                                                                      \
    launch_early(k_zf<R, r0, r1>, zgrid, kZCols*(r0 > r1 ? r0 : r1), zsm, s, A, psi, ldpsi, hpsi, ldh,       \
                 h.kp[ik].kinetic, 1.0 / (double)g.N, g.col_start, g.col_lo, g.ncol, g.m[2], tw2);           \
    break;
    PW_PAIRS(PW_CASE)
#undef PW_CASE
  }
  count_launch();
  mark(tm, 4, s);
  PW_CUDA_TRY(cudaGetLastError());
  return kOk;
}

template Status local_plane<double>(Handle&, int, int, const double2*, long, int, double2*, long, cudaStream_t, void*,
                                    StageTimer*);
template Status local_plane<float>(Handle&, int, int, const double2*, long, int, double2*, long, cudaStream_t, void*,
                                   StageTimer*);

}  // namespace pwgpu
