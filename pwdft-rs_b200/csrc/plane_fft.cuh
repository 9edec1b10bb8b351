// Two-stage line FFTs for the fused local pipeline: a length L = R0 * R1 is
// transformed in the order inverse A, B, then forward C, D, chosen so that
// the last inverse stage and the first forward stage of a line touch the same
// elements:
//   A  for j < R1:   u[k1] = sum_r x[j + R1 r] w_R0^(r k1), times w_L^(j k1),
//                    kept at slot j + R1 k1 (the elements it read)
//   B  for k1 < R0:  y[k1 + R0 k2] = sum_j u[j, k1] w_R1^(j k2)
//   C  for k1 < R0:  t[m] = sum_k2 y[k1 + R0 k2] w'_R1^(k2 m), times
//                    w'_L^(k1 m), kept at slot m + R1 k1
//   D  for m < R1:   X[m + R1 q] = sum_k1 t[k1, m] w'_R0^(k1 q)
// (w = e^(+2 pi i / .), w' its conjugate.)  A pass that multiplies by V(r)
// between the two transforms runs B, the product and C on one thread's
// registers, and every stage is in place, so a line needs one buffer.
//
// Sphere pruning: the caller's lines hold data only at e <= m and e >= L - m
// with 4 m < L, so the elements j + R1 r with 4 r >= R0 and 4 (r + 1) <= 3 R0
// are zero on input (A) and not wanted on output (D); these r are known at
// compile time, and radix 8 and 4 drop their arithmetic too.
#pragma once

#include "fft_smem.cuh"

namespace pwgpu {

// 6 and 10 points as 2 x 3 and 2 x 5, 12 points as 3 x 4 (coprime factors, so
// the index maps n -> (n mod ., n mod .) leave no inner twiddles).
template <int S, typename C> __device__ __forceinline__ void dft6(C* v) {
  C s[3] = {v[0] + v[3], v[2] + v[5], v[4] + v[1]};
  C d[3] = {v[0] - v[3], v[2] - v[5], v[4] - v[1]};
  dft3<S>(s);
  dft3<S>(d);
  v[0] = s[0]; v[4] = s[1]; v[2] = s[2];
  v[3] = d[0]; v[1] = d[1]; v[5] = d[2];
}

template <int S, typename C> __device__ __forceinline__ void dft10(C* v) {
  C s[5] = {v[0] + v[5], v[2] + v[7], v[4] + v[9], v[6] + v[1], v[8] + v[3]};
  C d[5] = {v[0] - v[5], v[2] - v[7], v[4] - v[9], v[6] - v[1], v[8] - v[3]};
  dft5<S>(s);
  dft5<S>(d);
  v[0] = s[0]; v[6] = s[1]; v[2] = s[2]; v[8] = s[3]; v[4] = s[4];
  v[5] = d[0]; v[1] = d[1]; v[7] = d[2]; v[3] = d[3]; v[9] = d[4];
}

template <int S, typename C> __device__ __forceinline__ void dft12(C* v) {
  C t[4][3];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    C a[3] = {v[(3 * n2) % 12], v[(3 * n2 + 4) % 12], v[(3 * n2 + 8) % 12]};
    dft3<S>(a);
    t[n2][0] = a[0]; t[n2][1] = a[1]; t[n2][2] = a[2];
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    dft4<S>(t[0][a], t[1][a], t[2][a], t[3][a]);
    // X[k], k = a mod 3 and k = b mod 4: k = 4 a + 9 b mod 12
#pragma unroll
    for (int b = 0; b < 4; ++b) v[(4 * a + 9 * b) % 12] = t[b][a];
  }
}

template <int N, int S, typename C> __device__ __forceinline__ void dft_n(C* v) {
  if constexpr (N == 6) dft6<S>(v);
  else if constexpr (N == 10) dft10<S>(v);
  else if constexpr (N == 12) dft12<S>(v);
  else dft<N, S>(v);
}

// Whether slot r of the pruned radix R0 can hold a sphere element.
template <int R0> __device__ __host__ constexpr bool slot_live(int r) { return 4 * r < R0 || 4 * (r + 1) > 3 * R0; }

// First inverse stage: radix R0 with the dead slots zero on entry.
template <int R0, typename C> __device__ __forceinline__ void dft_pruned_in(C* v) {
  if constexpr (R0 == 8) {
    // v2 .. v5 are zero: the two 4-point transforms have their outer inputs only
    const C a0 = v[0] + v[6], a2 = v[0] - v[6], b0 = v[1] + v[7], b2 = v[1] - v[7];
    const C ia = mul_si<1>(v[6]), ib = mul_si<1>(v[7]);
    const C e1 = v[0] - ia, e3 = v[0] + ia, o1 = v[1] - ib, o3 = v[1] + ib;
    using R = decltype(v[0].x);
    C t1, t3;
    t1.x = (R)PW_SQRT1_2 * (o1.x - o1.y);
    t1.y = (R)PW_SQRT1_2 * (o1.y + o1.x);
    const C t2 = mul_si<1>(b2);
    t3.x = (R)PW_SQRT1_2 * (-o3.x - o3.y);
    t3.y = (R)PW_SQRT1_2 * (-o3.y + o3.x);
    v[0] = a0 + b0; v[4] = a0 - b0;
    v[1] = e1 + t1; v[5] = e1 - t1;
    v[2] = a2 + t2; v[6] = a2 - t2;
    v[3] = e3 + t3; v[7] = e3 - t3;
  } else if constexpr (R0 == 4) {
    // v1, v2 are zero
    const C a = v[0], b = v[3], ib = mul_si<1>(v[3]);
    v[0] = a + b; v[2] = a - b; v[1] = a - ib; v[3] = a + ib;
  } else {
    dft_n<R0, +1>(v);
  }
}

// A: pruned radix-R0 inverse butterfly j with its twiddles (tw[m] = e^(-2 pi i m / L)).
template <int R0, typename C> __device__ __forceinline__ void bf_a(C* v, int j, const C* __restrict__ tw) {
  dft_pruned_in<R0>(v);
#pragma unroll
  for (int k = 1; k < R0; ++k) v[k] = cmulc(v[k], tw[j * k]);
}
// C: radix-R1 forward butterfly k1 with its twiddles.
template <int R1, typename C> __device__ __forceinline__ void bf_c(C* v, int k1, const C* __restrict__ tw) {
  dft_n<R1, -1>(v);
#pragma unroll
  for (int m = 1; m < R1; ++m) v[m] = cmul(v[m], tw[k1 * m]);
}

// Geometry of one z-plane in shared memory: d0 x rows of ld complex entries
// (d1 used, ld odd so that a walk along x is free of bank conflicts), and the
// y-lines between the two y stages in the rows that carry no sphere plane
// (avail = d0 - Xp of them, then rows past d0).
struct PlaneGeo {
  int d0, d1, ld, Xp, Yp, m0, m1, avail;
  unsigned mXp, md1;
  __device__ __forceinline__ int xrow(int p) const { return p < m0 ? p - m0 + d0 : p - m0; }
  __device__ __forceinline__ int srow(int p) const { return p < avail ? m0 + 1 + p : d0 + p - avail; }
};

// ---- stages of the plane, each ending at a block barrier ----

// y-inverse, stage A: Xp compact lines of Ab ([p][q], q the sphere row) into the scratch rows
template <int Y0, int Y1, typename C>
__device__ __forceinline__ void plane_ya(const C* Ab, C* P, const PlaneGeo& g, const C* TY, int tid, int T) {
  for (int t = tid; t < g.Xp * Y1; t += T) {
    const int p = t / Y1, j = t - p * Y1;
    C v[Y0];
#pragma unroll
    for (int r = 0; r < Y0; ++r) {
      v[r] = cmake<C>(0.0, 0.0);
      if (slot_live<Y0>(r)) {
        const int e = j + Y1 * r;
        const bool low = e <= g.m1;
        if (low || e >= g.d1 - g.m1) v[r] = Ab[p * g.Yp + (low ? e + g.m1 : e - g.d1 + g.m1)];
      }
    }
    bf_a<Y0>(v, j, TY);
    C* row = P + g.srow(p) * g.ld + j;
#pragma unroll
    for (int k = 0; k < Y0; ++k) row[Y1 * k] = v[k];
  }
  __syncthreads();
}

// y-inverse, stage B: scratch rows -> the x rows of the sphere planes
template <int Y0, int Y1, typename C>
__device__ __forceinline__ void plane_yb(C* P, const PlaneGeo& g, int tid, int T) {
  for (int t = tid; t < g.Xp * Y0; t += T) {
    const int k1 = fast_div(t, g.Xp, g.mXp), p = t - k1 * g.Xp;
    const C* src = P + g.srow(p) * g.ld + Y1 * k1;
    C v[Y1];
#pragma unroll
    for (int j = 0; j < Y1; ++j) v[j] = src[j];
    dft_n<Y1, +1>(v);
    C* dst = P + g.xrow(p) * g.ld + k1;
#pragma unroll
    for (int k = 0; k < Y1; ++k) dst[Y0 * k] = v[k];
  }
  __syncthreads();
}

// x-inverse, stage A, in place (rows outside the sphere planes count as zero)
template <int X0, int X1, typename C>
__device__ __forceinline__ void plane_xa(C* P, const PlaneGeo& g, const C* TX, int tid, int T) {
  for (int t = tid; t < X1 * g.d1; t += T) {
    const int j = fast_div(t, g.d1, g.md1), y = t - j * g.d1;
    C* base = P + j * g.ld + y;
    C v[X0];
#pragma unroll
    for (int r = 0; r < X0; ++r) {
      v[r] = cmake<C>(0.0, 0.0);
      if (slot_live<X0>(r)) {
        const int e = j + X1 * r;
        if (e <= g.m0 || e >= g.d0 - g.m0) v[r] = base[X1 * r * g.ld];
      }
    }
    bf_a<X0>(v, j, TX);
#pragma unroll
    for (int k = 0; k < X0; ++k) base[X1 * k * g.ld] = v[k];
  }
  __syncthreads();
}

// x-inverse stage B, the product with V(r), x-forward stage C, in place
template <int X0, int X1, typename R, typename C>
__device__ __forceinline__ void plane_xvx(C* P, const PlaneGeo& g, const R* __restrict__ vp, const C* TX, int tid,
                                          int T) {
  for (int t = tid; t < X0 * g.d1; t += T) {
    const int k1 = fast_div(t, g.d1, g.md1), y = t - k1 * g.d1;
    C* base = P + X1 * k1 * g.ld + y;
    const R* vb = vp + k1 * g.d1 + y;
    R w[X1];
#pragma unroll
    for (int k = 0; k < X1; ++k) w[k] = vb[X0 * k * g.d1];
    C v[X1];
#pragma unroll
    for (int j = 0; j < X1; ++j) v[j] = base[j * g.ld];
    dft_n<X1, +1>(v);
#pragma unroll
    for (int k = 0; k < X1; ++k) v[k] = v[k] * w[k];
    bf_c<X1>(v, k1, TX);
#pragma unroll
    for (int m = 0; m < X1; ++m) base[m * g.ld] = v[m];
  }
  __syncthreads();
}

// x-forward, stage D, in place; only the slots that can hold sphere planes are kept
template <int X0, int X1, typename C>
__device__ __forceinline__ void plane_xd(C* P, const PlaneGeo& g, int tid, int T) {
  for (int t = tid; t < X1 * g.d1; t += T) {
    const int m = fast_div(t, g.d1, g.md1), y = t - m * g.d1;
    C* base = P + m * g.ld + y;
    C v[X0];
#pragma unroll
    for (int k = 0; k < X0; ++k) v[k] = base[X1 * k * g.ld];
    dft_n<X0, -1>(v);
#pragma unroll
    for (int q = 0; q < X0; ++q)
      if (slot_live<X0>(q)) base[X1 * q * g.ld] = v[q];
  }
  __syncthreads();
}

// y-forward, stage C: the x rows of the sphere planes -> scratch rows
template <int Y0, int Y1, typename C>
__device__ __forceinline__ void plane_yc(C* P, const PlaneGeo& g, const C* TY, int tid, int T) {
  for (int t = tid; t < g.Xp * Y0; t += T) {
    const int k1 = fast_div(t, g.Xp, g.mXp), p = t - k1 * g.Xp;
    const C* src = P + g.xrow(p) * g.ld + k1;
    C v[Y1];
#pragma unroll
    for (int k = 0; k < Y1; ++k) v[k] = src[Y0 * k];
    bf_c<Y1>(v, k1, TY);
    C* dst = P + g.srow(p) * g.ld + Y1 * k1;
#pragma unroll
    for (int m = 0; m < Y1; ++m) dst[m] = v[m];
  }
  __syncthreads();
}

// y-forward, stage D: scratch rows -> the sphere rows of Ab
template <int Y0, int Y1, typename C>
__device__ __forceinline__ void plane_yd(C* Ab, const C* P, const PlaneGeo& g, int tid, int T) {
  for (int t = tid; t < g.Xp * Y1; t += T) {
    const int p = t / Y1, m = t - p * Y1;
    const C* row = P + g.srow(p) * g.ld + m;
    C v[Y0];
#pragma unroll
    for (int k = 0; k < Y0; ++k) v[k] = row[Y1 * k];
    dft_n<Y0, -1>(v);
#pragma unroll
    for (int q = 0; q < Y0; ++q) {
      if (!slot_live<Y0>(q)) continue;
      const int e = m + Y1 * q;
      const bool low = e <= g.m1;
      if (low || e >= g.d1 - g.m1) Ab[p * g.Yp + (low ? e + g.m1 : e - g.d1 + g.m1)] = v[q];
    }
  }
  __syncthreads();
}

}  // namespace pwgpu
