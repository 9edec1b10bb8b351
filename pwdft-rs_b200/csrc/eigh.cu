// Dense Hermitian / real symmetric eigensolver of the Rayleigh-Ritz step, one
// thread-block cluster per problem.
//
// Replaces the dense self_adjoint_eigen of the reference's per-k solve
// (pwdft-core/src/eigensolver/dense.rs:50-98, faer 0.24) where the
// matrix-free eigensolver needs it: the lowest nev eigenpairs of the
// m x m subspace matrix of each LOBPCG step (m <= 544).  One kernel does
// the whole solve on C = 1..16 CTAs of one cluster:
//
//  1. Householder reduction to real symmetric tridiagonal form, unblocked
//     (the zhetd2 recurrence: v, tau from the column below the diagonal,
//     p = tau A v, w = p - tau/2 (p^H v) v, A -= v w^H + w v^H).  The matrix
//     stays in shared memory for the whole reduction: column j lives in CTA
//     (j mod C), so the product A v needs no cross-CTA reduction (each CTA
//     owns whole columns of a Hermitian matrix = whole rows of A v).  Every
//     CTA keeps v and w whole and forms each reflector itself, so a step
//     exchanges once: the entries of p, the partials of p^H v and the next
//     column go through L2 under one cluster barrier.  Small matrices are
//     reduced by one CTA, with two block barriers a step (tridiag_one).
//  2. Eigenvalues of the tridiagonal T by multisection: one warp per
//     eigenvalue index, 32 Sturm counts per round (the three-term
//     recurrence of det(T - x I) with power-of-two rescaling), until the
//     interval is a few ulps wide.
//  3. Eigenvectors of T by inverse iteration, one thread per eigenvalue:
//     Gaussian elimination of T - lambda I with partial pivoting (a zero
//     pivot is replaced by eps ||T||), then two solves from a seeded start
//     vector.  Vectors whose eigenvalues lie within 1e-5 ||T|| of each
//     other are orthonormalised group by group (modified Gram-Schmidt,
//     twice), one warp per group; elsewhere inverse iteration leaves them
//     orthogonal to eps ||T|| / gap.
//  4. Back-transform x = H(0) ... H(m-2) z, one warp per eigenvector, the
//     vector in registers and the reflectors streamed through shared memory.
//
// What bounds it: latency.  The steps of 1 are serial, and a step at m = 540
// is ~7,400 cycles: the pass over the owned columns ~3,000 (shared-memory
// wavefronts and load latency), the cluster barrier ~1,250, the reads from L2
// ~1,300, two warp-wide sums with a square root and a division ~1,800.  One
// solve, lowest third of the pairs (all at 180), B200, against the form with
// two cluster barriers a step and a back-transform in panels: m = 540 2.8 ms
// (3.8), 360 1.65 (2.06), 180 0.77 (0.96), 66 0.18 (0.25); complex m = 64
// 0.21, 30 0.10 ms.  The one-CTA Jacobi solver takes 1.8 ms at m = 64.
//
// Every loop is bounded and every thread reaches the same sequence of
// cluster barriers.  Status: 0 ok, 1 a non-finite eigenvalue or vector.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <set>
#include <string>

#include "handle.hpp"
#include "dense_ops.cuh"
#include "linalg.hpp"

namespace cg = cooperative_groups;

// Phase timestamps for development builds (-DPWGPU_EIGH_PHASES): thread 0 of
// CTA 0 records %globaltimer at each phase boundary into eigh_phase_ns[].
#ifdef PWGPU_EIGH_PHASES
__device__ unsigned long long eigh_phase_ns[8];
#define EIGH_MARK(n)                                                            \
  do {                                                                          \
    if (rank == 0 && tid == 0) {                                                \
      unsigned long long t_;                                                    \
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                    \
      eigh_phase_ns[n] = t_;                                                    \
    }                                                                           \
  } while (0)
#else
#define EIGH_MARK(n) \
  do {               \
  } while (0)
#endif

namespace pwgpu {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kRegRows = 17;               // rows per lane in the back-transform
constexpr int kMaxM = 32 * kRegRows;       // 544
constexpr int kRowGroups = (kRegRows + 3) / 4;  // groups of four row slots of the back-transform
constexpr int kRowsPerThread = (kMaxM + kThreads - 1) / kThreads;
constexpr int kMaxCluster = 16;
constexpr int kBisectRounds = 48;
constexpr double kEps = 1.1102230246251565e-16;  // 2^-53
constexpr size_t kSmemLimit = 227 * 1024;

using namespace dense;

// The two halves of a cluster barrier (release on arrival, acquire on the
// wait); every thread of every CTA arrives once, then waits, per phase.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }

// Shared-memory layout of one CTA (identical on host and device).
struct Layout {
  size_t a, v, p, c, d, e2, tau, eig, grp, red, total;
};
__host__ __device__ inline size_t align16(size_t x) { return (x + 15) / 16 * 16; }
__host__ __device__ inline Layout layout(int m, int Ct, int tsz) {
  Layout L;
  const int ncl = (m + Ct - 1) / Ct;
  size_t o = 0;
  const size_t stage = (size_t)4 * ((m + 127) & ~127);  // staged reflectors of the back-transform, two by two
  L.a = o;   o = align16(o + ((size_t)ncl * m > stage ? (size_t)ncl * m : stage) * tsz);  // owned columns
  L.v = o;   o = align16(o + 2 * (size_t)m * tsz);    // Householder vectors of this and the last step
  L.p = o;   o = align16(o + (size_t)m * tsz);        // p = tau A v (one CTA)
  L.c = o;   o = align16(o + (size_t)m * tsz);        // the column to be reflected next
  L.d = o;   o = align16(o + (size_t)m * sizeof(double));
  L.e2 = o;  o = align16(o + (size_t)m * sizeof(double));
  L.tau = o; o = align16(o + 2 * (size_t)m * tsz);  // tau of every step, then w of the last step
  L.eig = o; o = align16(o + (size_t)m * sizeof(double));
  L.grp = o; o = align16(o + (size_t)(m + 1) * sizeof(int));
  L.red = o; o = align16(o + kWarps * (size_t)tsz);
  L.total = o;
  return L;
}

// Number of eigenvalues of the tridiagonal (d, ne2 = -e^2 <= -1e-40, scaled to
// ||T|| <= 1) below x: sign changes of the three-term sequence of
// det(T - x I), read off the sign bits.  A zero term cannot repeat, since
// e2 > 0, and the term after it has the opposite sign of the one before it,
// so the pair counts one change whichever sign the zero carries.  With
// ||T|| <= 1 a term grows by at most 3x a step, so the power-of-two rescaling
// is checked once every eight steps.  The value chain is one fused
// multiply-add per step; the loop is bound by the FP64 pipe (subtract,
// multiply, FMA per step), so the sign logic stays on the integer pipe.
__device__ __forceinline__ int sturm_count(const double* __restrict__ d, const double* __restrict__ ne2, int m,
                                           double x) {
  double pp = 1.0, p = d[0] - x;
  int hp = __double2hiint(p);
  unsigned cnt = (unsigned)hp >> 31;
  int i = 1;
  for (; i + 8 <= m; i += 8) {
    double dd[8], ee[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      dd[u] = d[i + u] - x;
      ee[u] = ne2[i + u - 1];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const double pn = fma(dd[u], p, ee[u] * pp);
      const int hn = __double2hiint(pn);
      cnt += (unsigned)(hn ^ hp) >> 31;
      hp = hn;
      pp = p;
      p = pn;
    }
    const double ap = fmax(fabs(p), fabs(pp));
    if (ap > 0x1p+400) {
      p *= 0x1p-400;
      pp *= 0x1p-400;
    } else if (ap < 0x1p-400) {
      p *= 0x1p+400;
      pp *= 0x1p+400;
    }
  }
  for (; i < m; ++i) {
    const double pn = fma(d[i] - x, p, ne2[i - 1] * pp);
    const int hn = __double2hiint(pn);
    cnt += (unsigned)(hn ^ hp) >> 31;
    hp = hn;
    pp = p;
    p = pn;
  }
  return (int)cnt;
}

// Offset (in doubles) of the reflectors in the work buffer (m x m, complex size): after the 7 m nev doubles of
// phase 3, rounded up to 32 bytes so that complex entries are aligned.
__host__ __device__ inline size_t vglob_offset(int m, int nev) { return ((size_t)7 * m * nev + 3) / 4 * 4; }
// Offset of the exchange buffers of the tridiagonalisation (4 m + 2 x 16 CTAs x 16 warps entries), and of the
// eigenvectors' norms (m) after them.
__host__ __device__ inline size_t xchg_offset(int m, int nev) { return vglob_offset(m, nev) + (size_t)2 * m * m; }
__host__ __device__ inline size_t norm_offset(int m, int nev) {
  return xchg_offset(m, nev) + 2 * ((size_t)4 * m + 2 * kMaxCluster * kWarps);
}

// Seeded start vector entry in [-1, 1).
__device__ __forceinline__ double start_entry(int i, int j) {
  uint64_t x = 0x9E3779B97F4A7C15ull * (uint64_t)(i + 1) + 0xD1B54A32D192ED03ull * (uint64_t)(j + 7);
  x ^= x >> 31;
  x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27;
  x *= 0x94D049BB133111EBull;
  x ^= x >> 33;
  return (double)(x >> 11) * 0x1p-52 - 1.0;
}

template <typename T> __device__ __forceinline__ T shfl_xor(T v, int o);
template <> __device__ __forceinline__ double shfl_xor<double>(double v, int o) {
  return __shfl_xor_sync(0xffffffffu, v, o);
}
template <> __device__ __forceinline__ double2 shfl_xor<double2>(double2 v, int o) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

// x - a b, as fused multiply-adds
__device__ __forceinline__ double nmadd(double x, double a, double b) { return fma(-a, b, x); }
__device__ __forceinline__ double2 nmadd(double2 x, double2 a, double2 b) {
  return make_double2(fma(a.y, b.y, fma(-a.x, b.x, x.x)), fma(-a.y, b.x, fma(-a.x, b.y, x.y)));
}

// Sum over the warp in every lane, on the FP64 tensor core: the 8 x 8 x 4 product with a matrix of ones adds
// the four lanes of a column of B, the two entries a lane gets back are added, and a second product adds the four
// distinct values left (two products and one addition against five shuffle-and-add stages).
__device__ __forceinline__ double warp_all(double v) {
  double c[2] = {0.0, 0.0}, d[2] = {0.0, 0.0};
  dmma(c, 1.0, v);
  dmma(d, 1.0, c[0] + c[1]);
  return d[0];
}
__device__ __forceinline__ double2 warp_all(double2 v) { return make_double2(warp_all(v.x), warp_all(v.y)); }

__device__ __forceinline__ double pick(bool c, double a, double b) { return c ? a : b; }
__device__ __forceinline__ double2 pick(bool c, double2 a, double2 b) {
  return make_double2(c ? a.x : b.x, c ? a.y : b.y);
}

// v[0 .. 3] summed over the warp: lanes 8 q .. 8 q + 7 hold the sum of v[q].
template <typename T> __device__ __forceinline__ T warp_sum4(T (&v)[4], int lane) {
  const bool hi = lane & 16, h8 = lane & 8;
  const T v0 = v[0], v1 = v[1], v2 = v[2], v3 = v[3];
  const T a = add(pick(hi, v2, v0), shfl_xor(pick(hi, v0, v2), 16));
  const T b = add(pick(hi, v3, v1), shfl_xor(pick(hi, v1, v3), 16));
  T c = add(pick(h8, b, a), shfl_xor(pick(h8, a, b), 8));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) c = add(c, shfl_xor(c, o));
  return c;
}

// tau, 1 / (alpha - beta) and beta of the reflector of a column whose entry
// below the diagonal is alpha and whose further entries have the squared norm s2.
template <typename T> __device__ __forceinline__ void reflector(T alpha, double s2, T& tau, T& scale, double& beta) {
  const double ar = re(alpha), ai = im(alpha);
  double tr = 0.0, ti = 0.0, sr = 0.0, si = 0.0;
  beta = ar;
  if (s2 > 0.0 || ai != 0.0) {
    const double x = ar * ar + ai * ai + s2;
    double ib;
    if (x > 1e-290 && x < 1e290) {
      const double r = rsqrt(x);
      beta = ar >= 0.0 ? -x * r : x * r;
      ib = ar >= 0.0 ? -r : r;
    } else {
      beta = ar >= 0.0 ? -sqrt(x) : sqrt(x);
      ib = 1.0 / beta;
    }
    tr = (beta - ar) * ib;
    ti = -ai * ib;
    const double dr = ar - beta, iden = 1.0 / (dr * dr + ai * ai);
    sr = dr * iden;
    si = -ai * iden;
  }
  tau = mk<T>(tr, ti);
  scale = mk<T>(sr, si);
}

// Tridiagonalisation of the m x m matrix a (shared memory) by one CTA, m <= 32 RPL: every warp keeps the vectors
// of a step (rows lane + 32 u) in its registers and forms w, the next column and its norm for itself, so a step has
// two block barriers and three warp-wide sums on its path.  Columns are spread over the warps four at a time; vs
// (2 m) and ws (m) carry v and w for the broadcast of their entries at the column index, pb (m) the entries of p.
template <typename T, int RPL>
__device__ void tridiag_one(T* a, int m, T* vs, T* ws, T* pb, double* dv, double* ev_off, T* tauv, T* vglob) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T z0 = mk<T>(0.0, 0.0);
  T c[RPL], v[RPL], vp[RPL], w[RPL];
#pragma unroll
  for (int u = 0; u < RPL; ++u) {
    const int i = lane + 32 * u;
    c[u] = i < m ? a[i] : z0;
    vp[u] = w[u] = z0;
    if (warp == 0 && i < m) ws[i] = vs[m + i] = z0;
  }
  for (int k = 0; k < m - 1; ++k) {
    const int par = k & 1;
    // reflector of column k
    double s2 = 0.0;
    T ca = z0, cd = z0;
#pragma unroll
    for (int u = 0; u < RPL; ++u) {
      const int i = lane + 32 * u;
      if (i >= k + 2) s2 += abs2(c[u]);
      ca = pick(u == (k + 1) >> 5, c[u], ca);
      cd = pick(u == k >> 5, c[u], cd);
    }
    s2 = warp_all(s2);
    ca = shfl(ca, (k + 1) & 31);
    T tau, scale;
    double beta;
    reflector(ca, s2, tau, scale, beta);
#pragma unroll
    for (int u = 0; u < RPL; ++u) {
      const int i = lane + 32 * u;
      v[u] = i > k + 1 ? mul(c[u], scale) : mk<T>(i == k + 1 ? 1.0 : 0.0, 0.0);
      if (warp == 0 && i < m) vs[par * m + i] = v[u];
      if (warp == 1 && i < m) vglob[(size_t)k * m + i] = v[u];
    }
    if (warp == 0 && lane == (k & 31)) {
      dv[k] = re(cd);
      ev_off[k] = beta;
      tauv[k] = tau;
    }
    __syncthreads();
    // rank-2 update of the last step and p = tau A v on the updated columns
    const T* vq = vs + (par ^ 1) * m;
    const int u0 = (k + 1) >> 5;
    for (int j0 = k + 1 + warp * 4; j0 < m; j0 += kWarps * 4) {
      T acc[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        acc[q] = z0;
        const int j = j0 + q;
        if (j < m) {
          T* col = a + (size_t)j * m;
          const T cw = cj(ws[j]), cv = cj(vq[j]);
#pragma unroll
          for (int u = 0; u < RPL; ++u) {
            const int i = lane + 32 * u;
            if (u < u0 || i >= m) continue;
            const T x = sub(col[i], add(mul(vp[u], cw), mul(w[u], cv)));
            col[i] = x;
            acc[q] = add(acc[q], mul(cj(x), v[u]));
          }
        }
      }
      const T s = warp_sum4(acc, lane);
      const int j = j0 + (lane >> 3);
      if ((lane & 7) == 0 && j < m) pb[j] = mul(tau, s);
    }
    __syncthreads();
    // w = p + alpha v and column k + 1
    T p[RPL];
    T ssum = z0;
#pragma unroll
    for (int u = 0; u < RPL; ++u) {
      const int i = lane + 32 * u;
      const bool in = i > k && i < m;
      p[u] = in ? pb[i] : z0;
      c[u] = in ? a[(size_t)(k + 1) * m + i] : z0;
      ssum = add(ssum, mul(cj(p[u]), v[u]));
    }
    const T al = mul(mul(tau, warp_all(ssum)), -0.5);
    const T cwk = cj(add(pb[k + 1], al));
#pragma unroll
    for (int u = 0; u < RPL; ++u) {
      const int i = lane + 32 * u;
      w[u] = add(p[u], mul(al, v[u]));
      c[u] = sub(c[u], add(mul(v[u], cwk), w[u]));
      vp[u] = v[u];
      if (warp == 0 && i < m) ws[i] = w[u];
    }
  }
  if (warp == 0) {
#pragma unroll
    for (int u = 0; u < RPL; ++u)
      if (lane + 32 * u == m - 1) dv[m - 1] = re(c[u]);
  }
}
constexpr int kOneMaxReal = 128, kOneMaxCplx = 64;  // sizes of tridiag_one

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
    k_eigh_cluster(const T* A, long lda, int m, int nev, int Ct, double gtol, double* w_out, T* Z, long ldz, double* work,
                   int* status) {
  extern __shared__ __align__(16) unsigned char smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Layout L = layout(m, Ct, (int)sizeof(T));
  T* a_loc = reinterpret_cast<T*>(smem + L.a);
  T* vbuf = reinterpret_cast<T*>(smem + L.v);
  T* pbuf = reinterpret_cast<T*>(smem + L.p);
  T* cbuf = reinterpret_cast<T*>(smem + L.c);
  double* dv = reinterpret_cast<double*>(smem + L.d);
  double* e2v = reinterpret_cast<double*>(smem + L.e2);
  T* tauv = reinterpret_cast<T*>(smem + L.tau);
  double* eig = reinterpret_cast<double*>(smem + L.eig);
  int* grp = reinterpret_cast<int*>(smem + L.grp);
  T* red = reinterpret_cast<T*>(smem + L.red);
  __shared__ double ev_off[kMaxM];  // off-diagonal e_k (the signed beta of each step)
  __shared__ double s2_part[kWarps];  // per-warp partial sums of the squared norm of the next column
  __shared__ double tnorm_s;
  __shared__ int bad;
  __shared__ int ngrp;
  const int nown = rank < Ct ? (m - rank + Ct - 1) / Ct : 0;  // columns rank, rank + Ct, ... below m
  const int lgCt = __ffs(Ct) - 1;                             // Ct is a power of two

  EIGH_MARK(0);
  if (tid == 0) bad = 0;
  launch_wait();
  if (rank == 0 && tid == 0) *status = 0;  // cluster barriers lie between this and a CTA that sets it
  for (int e = tid; e < nown * m; e += kThreads) {
    const int sl = e / m, i = e - sl * m;
    a_loc[e] = A[(long)(rank + sl * Ct) * lda + i];
  }
  __syncthreads();
  if (Ct > 1) cluster.sync();  // every CTA has started
  EIGH_MARK(1);

  // ---- 1. Householder tridiagonalisation on the first Ct CTAs ----
  // One cluster barrier per column.  Every CTA keeps the whole of v and w and
  // forms each reflector itself (the same operations in the same order, so the
  // copies agree bit for bit).  Step k:
  //   b  reflector v_k of column k (cbuf, updated through step k - 1)
  //   c  one pass over the owned columns j > k: the rank-2 update of step
  //      k - 1 and, on the updated entries, p_j = tau (A v)_j; a warp takes
  //      kColBlk columns at once, so v, v_prev and w are read once for them
  //   -  exchange through L2: entries of p, partials of p^H v, column k + 1
  //   a  w = p + alpha v, column k + 1 updated by this step, its norm
  // The exchange buffers alternate with the parity of k: a CTA writes a
  // parity again only after a barrier that every reader of it has passed.
  {
    T* xp = reinterpret_cast<T*>(work + xchg_offset(m, nev));  // [parity][m] entries of p
    T* xc = xp + 2 * m;                                        // [parity][m] column k + 1
    T* xs = xc + 2 * m;                                        // [parity][CTA][warp] partials of p^H v
    T* vglob_w = reinterpret_cast<T*>(work + vglob_offset(m, nev));
    T* wbuf = tauv + m;
    constexpr int kColBlk = sizeof(T) == sizeof(double) ? 3 : 2;
    const bool one = Ct == 1 && m <= (sizeof(T) == sizeof(double) ? kOneMaxReal : kOneMaxCplx);
    if (one && rank == 0) {
      if (m <= 32) tridiag_one<T, 1>(a_loc, m, vbuf, wbuf, pbuf, dv, ev_off, tauv, vglob_w);
      else if (m <= 64) tridiag_one<T, 2>(a_loc, m, vbuf, wbuf, pbuf, dv, ev_off, tauv, vglob_w);
      else if (sizeof(T) == sizeof(double)) tridiag_one<T, 4>(a_loc, m, vbuf, wbuf, pbuf, dv, ev_off, tauv, vglob_w);
    }
    if (!one && rank < Ct) {
      double s2 = 0.0;
      for (int i = tid; i < m; i += kThreads) {
        const T x = A[i];
        cbuf[i] = x;
        wbuf[i] = mk<T>(0.0, 0.0);
        vbuf[m + i] = mk<T>(0.0, 0.0);
        if (i >= 2) s2 += abs2(x);
      }
      s2 = warp_sum(s2);
      if (lane == 0) s2_part[warp] = s2;
      __syncthreads();
    }
    const int kend = !one && rank < Ct ? m - 1 : 0;
    for (int k = 0; k < kend; ++k) {
      const int par = k & 1;
      {
        // b: beta, tau and the scale 1 / (alpha - beta), by every thread
        T* v = vbuf + par * m;
        const T* vp = vbuf + (par ^ 1) * m;
        T tau, scale;
        {
          const double s2 = warp_all(lane < kWarps ? s2_part[lane] : 0.0);
          const T alpha = cbuf[k + 1];
          double beta;
          reflector(alpha, s2, tau, scale, beta);
          if (tid == 0) {
            dv[k] = re(cbuf[k]);
            ev_off[k] = beta;
            tauv[k] = tau;
          }
        }
        const bool store = rank == (k & (Ct - 1));
        for (int i = tid; i < m; i += kThreads) {
          T x = mk<T>(0.0, 0.0);
          if (i == k + 1) x = mk<T>(1.0, 0.0);
          if (i > k + 1) x = mul(cbuf[i], scale);
          if (i > k) v[i] = x;
          if (store) vglob_w[(size_t)k * m + i] = x;  // zero above the support, for the back-transform
        }
        __syncthreads();
        // c
        const int s0 = k + 1 > rank ? (k + 1 - rank + Ct - 1) >> lgCt : 0;  // first owned slot with column > k
        const int na = nown - s0;
        T part = mk<T>(0.0, 0.0);
        T* pout = Ct > 1 ? xp + par * m : pbuf;
        const int i0 = ((k + 1) & ~31) + lane;
        // columns a warp: as many as spread the owned ones over all warps, kColBlk at most
        const int cb = na <= kWarps ? 1 : (na <= 2 * kWarps ? 2 : kColBlk);
        for (int g = warp * cb; g < na; g += kWarps * cb) {
          T* col[kColBlk];
          T cw[kColBlk], cv[kColBlk], acc[kColBlk];
          const int nc = min(cb, na - g);
#pragma unroll
          for (int q = 0; q < kColBlk; ++q) {
            const int sl = s0 + g + (q < nc ? q : 0), j = rank + sl * Ct;
            col[q] = a_loc + (size_t)sl * m;
            cw[q] = cj(wbuf[j]);
            cv[q] = cj(vp[j]);
            acc[q] = mk<T>(0.0, 0.0);
          }
          T* xo = g == 0 && rank + s0 * Ct == k + 1 && Ct > 1 ? xc + par * m : nullptr;  // column k + 1 goes to the others
          // rows kUn chunks of 32 at a time, their loads ahead of the arithmetic
          constexpr int kUn = sizeof(T) == sizeof(double) ? 4 : 2;
          int i = i0;
          for (; i + 32 * (kUn - 1) < m; i += 32 * kUn) {
            T vi[kUn], pi[kUn], wi[kUn], x[kUn];
#pragma unroll
            for (int u = 0; u < kUn; ++u) {
              const bool in = i + 32 * u > k;  // rows above the step's range stay as they are
              vi[u] = in ? v[i + 32 * u] : mk<T>(0.0, 0.0);
              pi[u] = in ? vp[i + 32 * u] : mk<T>(0.0, 0.0);
              wi[u] = in ? wbuf[i + 32 * u] : mk<T>(0.0, 0.0);
            }
#pragma unroll
            for (int q = 0; q < kColBlk; ++q) {
              if (q >= nc) break;
#pragma unroll
              for (int u = 0; u < kUn; ++u) x[u] = col[q][i + 32 * u];
#pragma unroll
              for (int u = 0; u < kUn; ++u) {
                x[u] = sub(x[u], add(mul(pi[u], cw[q]), mul(wi[u], cv[q])));
                col[q][i + 32 * u] = x[u];
                acc[q] = add(acc[q], mul(cj(x[u]), vi[u]));
                if (q == 0 && xo) xo[i + 32 * u] = x[u];
              }
            }
          }
          for (; i < m; i += 32) {
            if (i <= k) continue;
            const T vi = v[i], pi = vp[i], wi = wbuf[i];
#pragma unroll
            for (int q = 0; q < kColBlk; ++q) {
              if (q >= nc) break;
              const T x = sub(col[q][i], add(mul(pi, cw[q]), mul(wi, cv[q])));
              col[q][i] = x;
              acc[q] = add(acc[q], mul(cj(x), vi));
              if (q == 0 && xo) xo[i] = x;
            }
          }
#pragma unroll
          for (int q = 0; q < kColBlk; ++q) {
            if (q >= nc) break;
            const int j = rank + (s0 + g + q) * Ct;
            const T pj = mul(tau, warp_all(acc[q]));
            if (lane == 0) pout[j] = pj;
            part = add(part, mul(cj(pj), v[j]));
          }
        }
        if (lane == 0) {
          if (Ct > 1) xs[(par * kMaxCluster + rank) * kWarps + warp] = part;
          else red[warp] = part;
        }
        if (Ct > 1) {
          cluster_arrive();
          cluster_wait();
        } else {
          __syncthreads();
        }
        // a
        T ssum = mk<T>(0.0, 0.0);
        const T* pin = Ct > 1 ? xp + par * m : pbuf;
        T pk1;
        if (Ct > 1) {
          const T* sx = xs + par * kMaxCluster * kWarps;
          T pt[kMaxCluster * kWarps / 32];
#pragma unroll
          for (int u = 0; u < kMaxCluster * kWarps / 32; ++u)
            pt[u] = lane + 32 * u < Ct * kWarps ? ldcg(sx + lane + 32 * u) : mk<T>(0.0, 0.0);
          pk1 = ldcg(pin + k + 1);
#pragma unroll
          for (int u = 0; u < kMaxCluster * kWarps / 32; ++u) ssum = add(ssum, pt[u]);
        } else {
          if (lane < kWarps) ssum = red[lane];
          pk1 = pin[k + 1];
        }
        T ci[kRowsPerThread], pi[kRowsPerThread];
#pragma unroll
        for (int u = 0; u < kRowsPerThread; ++u) {
          const int i = k + 1 + tid + u * kThreads;
          ci[u] = pi[u] = mk<T>(0.0, 0.0);
          if (i < m) {
            ci[u] = Ct > 1 ? ldcg(xc + par * m + i) : a_loc[(size_t)(k + 1) * m + i];
            pi[u] = Ct > 1 ? ldcg(pin + i) : pin[i];
          }
        }
        const T al = mul(mul(tau, warp_all(ssum)), -0.5);
        const T cwk = cj(add(pk1, al));  // conj(w_{k+1}); v_{k+1} = 1
        double s2 = 0.0;
#pragma unroll
        for (int u = 0; u < kRowsPerThread; ++u) {
          const int i = k + 1 + tid + u * kThreads;
          if (i >= m) break;
          const T vi = v[i], wi = add(pi[u], mul(al, vi));
          const T x = sub(ci[u], add(mul(vi, cwk), wi));
          wbuf[i] = wi;
          cbuf[i] = x;
          if (i >= k + 3) s2 += abs2(x);
        }
        s2 = warp_all(s2);
        if (lane == 0) s2_part[warp] = s2;
        __syncthreads();
      }
    }
    if (tid == 0) ev_off[m - 1] = 0.0;
    if (tid == 0 && !one && rank < Ct) dv[m - 1] = re(cbuf[m - 1]);
    if (Ct < C) {
      // the CTAs that took no part read T and tau through L2
      double* xt = reinterpret_cast<double*>(xp);  // free now: d, e, then tau
      T* xtau = xp + m;
      __syncthreads();
      if (rank == 0)
        for (int i = tid; i < m; i += kThreads) {
          xt[i] = dv[i];
          if (sizeof(T) == sizeof(double)) xc[i] = mk<T>(ev_off[i], 0.0);
          else xt[m + i] = ev_off[i];
          xtau[i] = i < m - 1 ? tauv[i] : mk<T>(0.0, 0.0);
        }
      cluster.sync();
      if (rank >= Ct)
        for (int i = tid; i < m; i += kThreads) {
          dv[i] = __ldcg(xt + i);
          ev_off[i] = sizeof(T) == sizeof(double) ? __ldcg(reinterpret_cast<double*>(xc) + i) : __ldcg(xt + m + i);
          tauv[i] = ldcg(xtau + i);
        }
      __syncthreads();
    } else {
      cluster.sync();
    }
  }
  EIGH_MARK(2);

  // ---- 2. eigenvalues by multisection on T / ||T|| ----
  if (warp == 0) {
    double gl = INFINITY, gu = -INFINITY;
    for (int i = lane; i < m; i += 32) {
      const double rr = (i > 0 ? fabs(ev_off[i - 1]) : 0.0) + fabs(ev_off[i]);
      gl = fmin(gl, dv[i] - rr);
      gu = fmax(gu, dv[i] + rr);
    }
    for (int o = 16; o > 0; o >>= 1) {
      gl = fmin(gl, __shfl_xor_sync(0xffffffffu, gl, o));
      gu = fmax(gu, __shfl_xor_sync(0xffffffffu, gu, o));
    }
    if (lane == 0) {
      const double tn = fmax(fabs(gl), fabs(gu));
      tnorm_s = tn > 0.0 && isfinite(tn) ? tn : 1.0;
      if (!isfinite(tn)) bad = 1;
    }
  }
  __syncthreads();
  const double tnorm = tnorm_s, itn = 1.0 / tnorm;
  for (int i = tid; i < m; i += kThreads) {
    dv[i] *= itn;
    ev_off[i] *= itn;
    // an off-diagonal below 1e-20 ||T|| counts as 1e-20 in the Sturm sequence, so a zero term never
    // propagates (a perturbation far below rounding)
    e2v[i] = -fmax(ev_off[i] * ev_off[i], 1e-40);
  }
  __syncthreads();
  {
    const double glo = -1.0 - 4.0 * kEps * m, ghi = 1.0 + 4.0 * kEps * m;  // the scaled Gershgorin interval
    const int tt = C * kThreads;
    int P = 32;  // points per eigenvalue and round
    while (P > 1 && (long)nev * P > tt) P >>= 1;
    const int pr = lane & (P - 1), seg = lane & ~(P - 1);
    const int ng = tt / P;
    for (int jb = (rank * kThreads + warp * 32) / P; jb < nev; jb += ng) {
      const int j = jb + lane / P;
      const bool act = j < nev;
      double lo = glo, hi = ghi;
      for (int round = 0; round < kBisectRounds; ++round) {
        const bool done = !act || hi - lo <= 2.0 * kEps * fmax(fabs(lo), fabs(hi)) + kEps;
        if (__all_sync(0xffffffffu, done)) break;
        const double x = lo + (hi - lo) * (double)(pr + 1) / (double)(P + 1);
        const int cnt = sturm_count(dv, e2v, m, x);
        const unsigned bits = (__ballot_sync(0xffffffffu, act && cnt > j) >> seg) & (P == 32 ? 0xffffffffu : ((1u << P) - 1u));
        const int l = bits ? __ffs(bits) - 1 : P;
        const double xhi = __shfl_sync(0xffffffffu, x, seg + (l < P ? l : P - 1));
        const double xlo = __shfl_sync(0xffffffffu, x, seg + (l > 0 ? l - 1 : 0));
        if (!done) {
          const double nlo = l > 0 ? xlo : lo;
          const double nhi = l < P ? xhi : hi;
          if (!(nhi < hi) && !(nlo > lo)) {
            hi = lo = 0.5 * (lo + hi);  // no representable progress
          } else {
            lo = nlo;
            hi = nhi;
          }
        }
      }
      if (act && pr == 0) {
        const double lam = 0.5 * (lo + hi);
        for (int q = 0; q < C; ++q) cluster.map_shared_rank(eig, q)[j] = lam;
        w_out[j] = lam * tnorm;
        if (!isfinite(lam)) bad = 1;
      }
    }
  }
  cluster.sync();
  EIGH_MARK(3);

  // ---- 3. inverse iteration on T / ||T||, one thread per eigenvalue ----
  // work: per row i and eigenvalue j (index i * nev + j) the U row {1/u0, u1, u2, rhs} as double4 and the
  // row operation {l, swapped} as double2; then the vectors, column j at zt + j * m
  {
    double4* U4 = reinterpret_cast<double4*>(work);
    double2* F2 = reinterpret_cast<double2*>(work + (size_t)4 * m * nev);
    double* zt = work + (size_t)6 * m * nev;
    const double piv_min = kEps;
    double* znorm = work + norm_offset(m, nev);
    const int nj = (nev + C - 1) / C;
    for (int jj = tid; jj < nj; jj += kThreads) {
      const int j = rank * nj + jj;
      if (j >= nev) break;
      const double lam = eig[j];
      // factorisation, the start vector carried as right-hand side
      double a = dv[0] - lam, b = m > 1 ? ev_off[0] : 0.0, cur = start_entry(0, j);
      for (int i = 0; i < m - 1; ++i) {
        const size_t o = (size_t)i * nev + j;
        const double c = ev_off[i];
        const double dn = dv[i + 1] - lam, en = i + 1 < m - 1 ? ev_off[i + 1] : 0.0;
        const double nxt = start_entry(i + 1, j);
        if (fabs(a) >= fabs(c)) {
          if (fabs(a) < piv_min) a = a < 0.0 ? -piv_min : piv_min;
          const double ia = 1.0 / a, l = c * ia;
          U4[o] = make_double4(ia, b, 0.0, cur);
          F2[o] = make_double2(l, 0.0);
          const double ncur = nxt - l * cur;
          a = dn - l * b;
          b = en;
          cur = ncur;
        } else {
          const double ic = 1.0 / c, l = a * ic;
          U4[o] = make_double4(ic, dn, en, nxt);
          F2[o] = make_double2(l, 1.0);
          const double ncur = cur - l * nxt;
          a = b - l * dn;
          b = -l * en;
          cur = ncur;
        }
      }
      if (fabs(a) < piv_min) a = a < 0.0 ? -piv_min : piv_min;
      U4[(size_t)(m - 1) * nev + j] = make_double4(1.0 / a, 0.0, 0.0, cur);
      double scale = 1.0;
      for (int it = 0; it < 2; ++it) {
        if (it > 0) {
          // the stored row operations on the normalised vector
          double c0 = U4[j].w * scale;
          int i = 0;
          for (; i + 8 <= m - 1; i += 8) {
            double2 f[8];
            double nx[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              f[q] = F2[(size_t)(i + q) * nev + j];
              nx[q] = U4[(size_t)(i + q + 1) * nev + j].w * scale;
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              double out;
              if (f[q].y == 0.0) {
                out = c0;
                c0 = nx[q] - f[q].x * c0;
              } else {
                out = nx[q];
                c0 = c0 - f[q].x * nx[q];
              }
              reinterpret_cast<double*>(&U4[(size_t)(i + q) * nev + j])[3] = out;
            }
          }
          for (; i < m - 1; ++i) {
            const double2 f = F2[(size_t)i * nev + j];
            const double nx = U4[(size_t)(i + 1) * nev + j].w * scale;
            double out;
            if (f.y == 0.0) {
              out = c0;
              c0 = nx - f.x * c0;
            } else {
              out = nx;
              c0 = c0 - f.x * nx;
            }
            reinterpret_cast<double*>(&U4[(size_t)i * nev + j])[3] = out;
          }
          reinterpret_cast<double*>(&U4[(size_t)(m - 1) * nev + j])[3] = c0;
        }
        // back-substitution, eight rows per batch of loads; the last one writes the vector itself
        double* zj = zt + (size_t)j * m;
        double y1 = 0.0, y2 = 0.0, nrm2 = 0.0;
        int i = m - 1;
        for (; i >= 7; i -= 8) {
          double4 u[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) u[q] = U4[(size_t)(i - q) * nev + j];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const double yi = (u[q].w - u[q].y * y1 - u[q].z * y2) * u[q].x;
            if (it == 0) reinterpret_cast<double*>(&U4[(size_t)(i - q) * nev + j])[3] = yi;
            else zj[i - q] = yi;
            nrm2 += yi * yi;
            y2 = y1;
            y1 = yi;
          }
        }
        for (; i >= 0; --i) {
          const double4 u = U4[(size_t)i * nev + j];
          const double yi = (u.w - u.y * y1 - u.z * y2) * u.x;
          if (it == 0) reinterpret_cast<double*>(&U4[(size_t)i * nev + j])[3] = yi;
          else zj[i] = yi;
          nrm2 += yi * yi;
          y2 = y1;
          y1 = yi;
        }
        const bool okn = nrm2 > 0.0 && isfinite(nrm2);
        scale = okn ? 1.0 / sqrt(nrm2) : 0.0;
        if (!okn) bad = 1;
      }
      znorm[j] = scale;  // applied where the vector is read
    }
  }
  __threadfence();
  cluster.sync();
  EIGH_MARK(4);

  const int gw = rank * kWarps + warp, nw = C * kWarps;
  // ---- 3b. groups of close eigenvalues: modified Gram-Schmidt, twice ----
  {
    double* zt = work + (size_t)6 * m * nev;
    if (tid == 0) {
      int n = 0;
      int start = 0;
      for (int j = 1; j <= nev; ++j) {
        if (j == nev || eig[j] - eig[j - 1] > gtol) {
          if (j - start > 1) {
            grp[2 * n] = start;
            grp[2 * n + 1] = j;
            ++n;
          }
          start = j;
        }
      }
      ngrp = n;
    }
    __syncthreads();
    for (int g = gw; g < ngrp; g += nw) {
      const int g0 = grp[2 * g], g1 = grp[2 * g + 1];
      for (int j = g0; j < g1; ++j) {
        double* zj = zt + (size_t)j * m;
        for (int pass = 0; pass < 2; ++pass) {
          for (int i = g0; i < j; ++i) {
            const double* zi = zt + (size_t)i * m;
            double dot = 0.0;
            for (int rr = lane; rr < m; rr += 32) dot += zi[rr] * zj[rr];
            dot = warp_sum(dot);
            for (int rr = lane; rr < m; rr += 32) zj[rr] -= dot * zi[rr];
            __syncwarp();
          }
        }
        double n2 = 0.0;
        for (int rr = lane; rr < m; rr += 32) n2 += zj[rr] * zj[rr];
        n2 = warp_sum(n2);
        const double scn = n2 > 0.0 ? 1.0 / sqrt(n2) : 0.0;
        if (!(n2 > 0.0) && lane == 0) bad = 1;
        for (int rr = lane; rr < m; rr += 32) zj[rr] *= scn;
        if (lane == 0) work[norm_offset(m, nev) + j] = 1.0;
        __syncwarp();
      }
    }
  }
  __threadfence();
  cluster.sync();
  EIGH_MARK(5);

  // ---- 4. back-transform x = H(0) ... H(m-2) z, one warp per vector, the vector in registers ----
  // The reflectors pass through shared memory in chunks, the next chunk copied while one is applied, so a CTA waits
  // twice a chunk and a warp's path through a reflector is one dot product over the warp and one update.  Rows of
  // a reflector above its support are zero in the store and the staged rows past m are zeroed once, so the loops
  // carry no predicates; groups of four row slots wholly above the support or past m are skipped (a test per slot
  // costs more than the slot's arithmetic).
  {
    const double* zt = work + (size_t)6 * m * nev;
    const double* znorm = work + norm_offset(m, nev);
    const T* vglob = reinterpret_cast<const T*>(work + vglob_offset(m, nev));
    const int mp = (m + 127) & ~127;
    const int ng = mp >> 7;
    const size_t cap = max((size_t)((m + Ct - 1) / Ct) * m, (size_t)4 * mp);  // entries of the column buffer
    const int R = (int)min((size_t)16, cap / (2 * (size_t)mp));             // reflectors per chunk
    T* sv = a_loc;
    const int waves = (nev + nw - 1) / nw;
    const int nchunk = (m - 1 + R - 1) / R;
    launch_release();
    auto stage = [&](int c) {
      const int k0 = m - 2 - R * c;  // reflectors k0, k0 - 1, ..., k0 - R + 1
      const int lo = max(0, k0 - R + 2) & ~127;
      T* dst = sv + (size_t)(c & 1) * R * mp;
      const int rows = m - lo;
      for (int e = tid; e < R * rows; e += kThreads) {
        const int q = e / rows, i = lo + e - q * rows, kq = k0 - q;
        if (kq >= 0) cp_async_zfill<sizeof(T)>(dst + q * mp + i, vglob + (size_t)kq * m + i, true);
      }
      cp_async_commit();
    };
    __syncthreads();
    for (int e = tid; e < 2 * R * mp; e += kThreads)
      if (e % mp >= m) sv[e] = mk<T>(0.0, 0.0);
    for (int wv = 0; wv < waves; ++wv) {
      const int j = gw + wv * nw;
      const bool live = j < nev;  // a warp without a vector still helps to stage
      const double zs = live ? __ldcg(znorm + j) : 0.0;
      T z[4 * kRowGroups];
#pragma unroll
      for (int t = 0; t < 4 * kRowGroups; ++t) {
        const int i = lane + 32 * t;
        z[t] = mk<T>(live && i < m ? __ldcg(zt + (size_t)j * m + i) * zs : 0.0, 0.0);
      }
      if (nchunk > 0) stage(0);
      for (int c = 0; c < nchunk; ++c) {
        if (c + 1 < nchunk) {
          stage(c + 1);
          cp_async_wait<1>();
        } else {
          cp_async_wait<0>();
        }
        __syncthreads();
        if (live) {
          const T* vc = sv + (size_t)(c & 1) * R * mp + lane;
          const int k0 = m - 2 - R * c, qn = min(R, k0 + 1);
          for (int q = 0; q < qn; ++q) {
            const T tau = tauv[k0 - q];
            const int g0 = (k0 - q + 1) >> 7;
            const T* vq = vc + q * mp;
            T s0 = mk<T>(0.0, 0.0), s1 = s0;
#pragma unroll
            for (int g = 0; g < kRowGroups; ++g) {
              if (g < g0 || g >= ng) continue;
#pragma unroll
              for (int t = 4 * g; t < 4 * g + 4; t += 2) {
                s0 = nmadd(s0, cj(vq[32 * t]), z[t]);
                s1 = nmadd(s1, cj(vq[32 * t + 32]), z[t + 1]);
              }
            }
            const T f = mul(tau, mul(warp_all(add(s0, s1)), -1.0));
#pragma unroll
            for (int g = 0; g < kRowGroups; ++g) {
              if (g < g0 || g >= ng) continue;
#pragma unroll
              for (int t = 4 * g; t < 4 * g + 4; ++t) z[t] = nmadd(z[t], vq[32 * t], f);
            }
          }
        }
        __syncthreads();  // the buffer may be filled again
      }
      if (live) {
        bool ok = true;
#pragma unroll
        for (int t = 0; t < 4 * kRowGroups; ++t) {
          const int i = lane + 32 * t;
          if (i < m) {
            Z[(size_t)j * ldz + i] = z[t];
            ok = ok && finite(z[t]);
          }
        }
        if (!ok) bad = 1;
      }
    }
  }
  __syncthreads();
  EIGH_MARK(6);
  if (tid == 0 && bad) atomicExch(status, 1);
  cluster.sync();  // no CTA leaves while another may still read its shared memory
}

bool layout_fits(int m, int Ct, int tsz) {
  return layout(m, Ct, tsz).total + 2 * kMaxM * sizeof(double) <= kSmemLimit;
}

// The smallest cluster whose CTAs hold the matrix in shared memory (0: none).
int min_cluster(int m, int tsz) {
  for (int C = 1; C <= kMaxCluster; C *= 2)
    if (layout_fits(m, C, tsz)) return C;
  return 0;
}

// CTAs that hold the matrix during the tridiagonalisation of a cluster of C:
// one as long as tridiag_one takes the size (real m = 128: 221 us against 335
// on eight CTAs; complex m = 64 108 against 204 at m = 65), else all.
int tridiag_ctas(int m, int C, int tsz) {
  return m <= (tsz == (int)sizeof(double) ? kOneMaxReal : kOneMaxCplx) && layout_fits(m, 1, tsz) ? 1 : C;
}

// The cluster size to use, never more CTAs than columns: sixteen from m = 161
// (real) or 181 (complex) on, where the phases after the reduction gain more
// from the wider cluster than its barrier costs (real m = 150, lowest third:
// 669 us on eight against 754 on sixteen; m = 180, all pairs: 985 and 773).
int pick_cluster(int m, int tsz) {
  const int c0 = min_cluster(m, tsz);
  if (c0 == 0) return 0;
  int want = m > (tsz == (int)sizeof(double) ? 160 : 180) ? 16 : 8;
  while (want > m) want /= 2;
  return std::max(c0, want);
}

// The shared-memory and cluster-size opt-ins are per-device attributes: set
// once per device, under a lock (solves on several host threads reach here).
template <typename T> Status set_attributes() {
  static std::mutex mu;
  static std::set<int> done;
  int dev = 0;
  PW_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (done.count(dev)) return kOk;
  auto kern = k_eigh_cluster<T>;
  cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kSmemLimit - 2 * kMaxM * sizeof(double)));
  if (err == cudaSuccess) err = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (err != cudaSuccess) return fail(kCuda, std::string("eigh_cluster attributes: ") + cudaGetErrorString(err));
  done.insert(dev);
  return kOk;
}

template <typename T>
cudaLaunchConfig_t launch_config(int m, int C, int Ct, cudaLaunchAttribute* attr, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = layout(m, Ct, (int)sizeof(T)).total;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Whether a cluster of C CTAs with this kernel's shared memory can be
// resident on the current device (checked once per cluster size).
template <typename T> bool cluster_fits(int m, int C) {
  static std::mutex mu;
  static int cache[2][kMaxCluster + 1] = {};  // [real, complex][C]: 0 unknown, 1 fits, 2 does not
  const int slot = sizeof(T) == sizeof(double) ? 0 : 1;
  std::lock_guard<std::mutex> lock(mu);
  // the largest m that uses a cluster size has the most shared memory: probe at that size
  int& c = cache[slot][C];
  if (c == 0) {
    if (set_attributes<T>() != kOk) return false;
    int mm = 1;  // the largest m a cluster of C CTAs can hold: the most shared memory
    for (int t = 1; t <= kMaxM; ++t)
      if (layout_fits(t, C, (int)sizeof(T))) mm = t;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = launch_config<T>(mm, C, C, attr, nullptr);
    int n = 0;
    cudaError_t e = cudaOccupancyMaxActiveClusters(&n, k_eigh_cluster<T>, &cfg);
    c = (e == cudaSuccess && n > 0) ? 1 : 2;
    if (e != cudaSuccess) cudaGetLastError();
  }
  return c == 1;
}

// The preferred cluster size, halved while such a cluster cannot be
// resident on this device (0 when none can).
template <typename T> int choose_cluster(int m) {
  if (m < 1 || m > kMaxM) return 0;
  const int c0 = min_cluster(m, (int)sizeof(T));
  if (c0 == 0) return 0;
  int C = pick_cluster(m, (int)sizeof(T));
  while (C > c0 && !cluster_fits<T>(m, C)) C /= 2;
  return cluster_fits<T>(m, C) ? C : 0;
}

template <typename T>
Status launch_eigh(const T* A, long lda, int m, int nev, double* w, T* Z, long ldz, double* work, int* status,
                   cudaStream_t s) {
  const int C = choose_cluster<T>(m);
  if (C == 0) return fail(kInvalid, "eigh_cluster: matrix too large for the cluster eigensolver");
  Status r = set_attributes<T>();
  if (r != kOk) return r;
  auto kern = k_eigh_cluster<T>;
  cudaLaunchAttribute attr[2];
  const int Ct = tridiag_ctas(m, C, (int)sizeof(T));
  cudaLaunchConfig_t cfg = launch_config<T>(m, C, Ct, attr, s);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  // Eigenvalues closer than gtol ||T|| are orthonormalised as one group: inverse iteration leaves the others
  // orthogonal to eps / gtol.  Up to m = 64 the groups are few and short, and the wide tolerance keeps the vectors
  // within 1e-12 of orthonormal (3.4e-14 over spread, repeated and graded spectra); above it the serial Gram-Schmidt of a wide group would dominate.
  const double gtol = m <= 64 ? 1e-3 : 1e-5;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, A, lda, m, nev, Ct, gtol, w, Z, ldz, work, status);
  count_launch();
  if (e != cudaSuccess) return fail(kCuda, std::string("eigh_cluster launch: ") + cudaGetErrorString(e));
  return kOk;
}


}  // namespace

size_t eigh_cluster_work_doubles(int m, int nev) {
  // U rows, row operations and vectors (7 m nev), the reflectors, the exchange buffers, the vectors' norms
  return norm_offset(m, std::max(nev, 1)) + m;
}

bool eigh_cluster_supported(int m, bool complex_matrix) {
  return eigh_cluster_size(m, complex_matrix) > 0;
}

int eigh_cluster_size(int m, bool complex_matrix) {
  return complex_matrix ? choose_cluster<double2>(m) : choose_cluster<double>(m);
}

Status eigh_cluster(const double* A, long lda, int m, int nev, double* w, double* Z, long ldz, double* work,
                    int* status, cudaStream_t s) {
  return launch_eigh<double>(A, lda, m, nev, w, Z, ldz, work, status, s);
}

Status eigh_cluster(const double2* A, long lda, int m, int nev, double* w, double2* Z, long ldz, double* work,
                    int* status, cudaStream_t s) {
  return launch_eigh<double2>(A, lda, m, nev, w, Z, ldz, work, status, s);
}

}  // namespace pwgpu
