// The plane pass with radix pairs chosen at run time.
#include "plane_pass.hpp"

namespace pwgpu {

namespace {

// The same pass with the radix pairs of x and y chosen at run time, each phase
// a function of its own (called once per phase and band), for planes whose x
// and y lengths differ; on a 72 x 72 plane it takes 1.05 (FP64) and 1.09
// (FP32) times k_plane.
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

}  // namespace

template <typename R> cudaError_t plane_rt_opt_in() {
  return cudaFuncSetAttribute(k_plane_rt<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlaneSmemMax);
}

template <typename R> void plane_rt(const PlaneRun<R>& p, int rows, int px, int py, cudaStream_t s) {
  launch_early(k_plane_rt<R>, dim3(p.d2, (p.nb + p.bpc - 1) / p.bpc), 256, p.smem, s, p.A, p.vz, p.nb, p.bpc, p.d2,
               p.geo, rows, px, py, p.twx, p.twy);
  count_launch();
}

template cudaError_t plane_rt_opt_in<double>();
template cudaError_t plane_rt_opt_in<float>();
template void plane_rt<double>(const PlaneRun<double>&, int, int, int, cudaStream_t);
template void plane_rt<float>(const PlaneRun<float>&, int, int, int, cudaStream_t);

}  // namespace pwgpu
