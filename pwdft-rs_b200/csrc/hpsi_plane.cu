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
// The kernels stand in plane_kernels.cuh (radix pairs at compile time) and
// plane_rt.cu (unequal x and y lengths).
#include <algorithm>
#include <string>

#include "handle.hpp"
#include "plane_pass.hpp"

namespace pwgpu {

namespace {

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

// Opt the kernels that a grid of these radix pairs runs into the shared memory they may need.
Status configure(const int (&pair)[3]) {
  cudaError_t e = cudaSuccess;
  auto keep = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  switch (pair[2]) {
#define PW_CASE(r0, r1)                             \
  case pair_id(r0, r1):                             \
    keep(PlaneLen<double, r0, r1>::opt_in_z());     \
    keep(PlaneLen<float, r0, r1>::opt_in_z());      \
    break;
    PW_PAIRS(PW_CASE)
#undef PW_CASE
  }
  if (pair[0] != pair[1]) {
    keep(plane_rt_opt_in<double>());
    keep(plane_rt_opt_in<float>());
  } else {
    switch (pair[0]) {
#define PW_CASE(r0, r1)                              \
  case pair_id(r0, r1):                              \
    keep(PlaneLen<double, r0, r1>::opt_in_square()); \
    keep(PlaneLen<float, r0, r1>::opt_in_square());  \
    break;
      PW_PAIRS(PW_CASE)
#undef PW_CASE
    }
  }
  if (e != cudaSuccess) return fail(kCuda, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
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
  Status st = configure(g.pair);
  if (st != kOk) return st;
  g.plane_ok = true;
  return kOk;
}

template <typename R>
static void launch_zi(const Handle& h, const double2* psi, long ldpsi, cplx<R>* A, int nb, cudaStream_t s) {
  const GridMaps& g = h.g;
  const ZColumns c{g.col_start, g.col_lo, g.ncol, g.m[2]};
  switch (g.pair[2]) {
#define PW_CASE(r0, r1) \
  case pair_id(r0, r1): PlaneLen<R, r0, r1>::zi(psi, ldpsi, A, nb, c, Tables<R>::tw(g, 2), s); break;
    PW_PAIRS(PW_CASE)
#undef PW_CASE
  }
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
    const PlaneRun<double> p{A, nullptr, cnt, bpc, d2, geo, g.tw64[0], g.tw64[1], plane_smem<double>(g)};
    switch (g.pair[0]) {
#define PW_CASE(r0, r1) \
  case pair_id(r0, r1): PlaneLen<double, r0, r1>::rho(p, fw_dev + c0, part, s); break;
      PW_PAIRS(PW_CASE)
#undef PW_CASE
    }
    k_rho_add<<<dim3(d0, (d1 + 31) / 32, (d2 + 31) / 32), 256, 0, s>>>(part, groups, d0, d1, d2, rho);
    count_launch();
  }
  PW_CUDA_TRY(cudaGetLastError());
  return kOk;
}

template <typename R>
Status local_plane(Handle& h, int spin, int ik, const double2* psi, long ldpsi, int nb, double2* hpsi, long ldh,
                   cudaStream_t s, void* scratch, StageTimer* tm) {
  const GridMaps& g = h.g;
  cplx<R>* A = static_cast<cplx<R>*>(scratch);
  launch_zi<R>(h, psi, ldpsi, A, nb, s);
  mark(tm, 0, s);
  const int d2 = g.d[2];
  const int bpc = std::max(1, std::min(8, (int)((long)nb * d2 / (148 * 8))));
  const PlaneRun<R> p{A, Tables<R>::vz(h, spin), nb, bpc, d2, geometry(g), Tables<R>::tw(g, 0), Tables<R>::tw(g, 1),
                      plane_smem<R>(g)};
  if (g.pair[0] == g.pair[1]) {
    switch (g.pair[0]) {
#define PW_CASE(r0, r1) \
  case pair_id(r0, r1): PlaneLen<R, r0, r1>::plane(p, s); break;
      PW_PAIRS(PW_CASE)
#undef PW_CASE
    }
  } else {
    plane_rt<R>(p, plane_rows(g), g.pair[0], g.pair[1], s);
  }
  mark(tm, 2, s);
  const ZColumns c{g.col_start, g.col_lo, g.ncol, g.m[2]};
  switch (g.pair[2]) {
#define PW_CASE(r0, r1)                                                                                          \
  case pair_id(r0, r1):                                                                                          \
    PlaneLen<R, r0, r1>::zf(A, psi, ldpsi, hpsi, ldh, h.kp[ik].kinetic, 1.0 / (double)g.N, nb, c,                \
                            Tables<R>::tw(g, 2), s);                                                             \
    break;
    PW_PAIRS(PW_CASE)
#undef PW_CASE
  }
  mark(tm, 4, s);
  PW_CUDA_TRY(cudaGetLastError());
  return kOk;
}

template Status local_plane<double>(Handle&, int, int, const double2*, long, int, double2*, long, cudaStream_t, void*,
                                    StageTimer*);
template Status local_plane<float>(Handle&, int, int, const double2*, long, int, double2*, long, cudaStream_t, void*,
                                   StageTimer*);

}  // namespace pwgpu
