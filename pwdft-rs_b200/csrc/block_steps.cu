// The block steps of the eigensolver for narrow blocks (at most kMaxBlock
// bands): orthonormalising the search directions W and P, the subspace matrix
// and the update, one launch each.
//
// What bounds these steps at 2 to 16 atoms is neither arithmetic nor memory
// but the number of dependent launches: a step of 27 bands over 1,045 plane
// waves is ~50 library GEMMs, split-K sums, norms, gathers and copies of a few
// microseconds each, plus host round trips for the Cholesky status.  Here
// the rows of the block are spread over one thread-block cluster (up to 16
// CTAs) and stay in shared memory from the first projection to the last
// Cholesky-QR pass; every small matrix (A^H Y over all rows) is summed
// from the CTAs' partials in rank order through L2, with one cluster barrier,
// and factored by every CTA alike.  Products run on the FP64 tensor cores
// (mma.sync m8n8k4), operands straight from L2 or shared memory.
//
// Against the library-call steps, with the same subspace eigensolver (B200):
// restart iteration of 8 Si atoms at Gamma (real, 22 columns, 2,945 rows)
// 27.7 -> 13.5 ms, of 2 atoms over 6 k-points (complex, 10 columns, 411 rows)
// 21.0 -> 7.9 ms, whole LSDA run of 8 C atoms (27 columns, 1,045 rows, 40
// blocks on 8 lanes) 405 -> 231 ms.  One Cholesky barrier a column instead of
// three, and one sum less for each of W and P, are 5 % of those; launches that
// begin beside the end of the one before them, and one copy of the column lists
// a step, another 3 to 7 %.  A cluster lets its successor begin only near its
// own end, so that a waiting cluster does not keep SMs from other lanes.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>
#include <set>
#include <string>

#include "dense_ops.cuh"
#include "handle.hpp"
#include "linalg.hpp"
#include "lobpcg.hpp"

namespace pwgpu {

namespace {

namespace cg = cooperative_groups;
using namespace dense;

constexpr int kT = 512;
constexpr int kW = kT / 32;
constexpr int kMaxC = 16;
constexpr size_t kSmemMax = 227 * 1024 - 4096;

template <typename T> __device__ __forceinline__ T zero() { return mk<T>(0.0, 0.0); }

template <typename T> struct Tile;
template <> struct Tile<double> {
  double c[2];
  __device__ __forceinline__ void clear() { c[0] = c[1] = 0.0; }
  __device__ __forceinline__ void mma(double a, double b) { dmma(c, a, b); }
  __device__ __forceinline__ double get(int h) const { return c[h]; }
};
template <> struct Tile<double2> {
  double re[2], im[2];
  __device__ __forceinline__ void clear() { re[0] = re[1] = im[0] = im[1] = 0.0; }
  __device__ __forceinline__ void mma(double2 a, double2 b) {
    dmma(re, a.x, b.x);
    dmma(im, a.x, b.y);
    dmma(re, -a.y, b.y);
    dmma(im, a.y, b.x);
  }
  __device__ __forceinline__ double2 get(int h) const { return make_double2(re[h], im[h]); }
};

// Row stride of a shared-memory block of `rows` rows: 4 mod 16, so that the
// operand reads of a tile (4 rows x 8 columns) touch every bank equally.
__host__ __device__ constexpr int pad_ld(int rows) { return (rows + 15) / 16 * 16 + 4; }

// Z (p x q, ld ldz in shared memory) = sum over the local rows of conj(A(i, a)) B(i, b).  Warps share the row
// tiles of Z (8 x up to 32 entries each) and, when those are fewer than the warps, slices of the rows, added in
// slice order.  la / lb return an entry, zero outside.  accumulate: added to Z.
template <typename T, typename LA, typename LB>
__device__ void local_gram(int rows, int p, int q, LA la, LB lb, T* Z, int ldz, bool accumulate = false) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kr = lane & 3, kc = lane >> 2;
  const int tp = (p + 7) >> 3, tg = (q + 31) >> 5;
  const int items = tp * tg;
  const int S = items >= kW ? 1 : kW / items;  // row slices
  const int per = ((rows + S - 1) / S + 3) & ~3;
  for (int base = 0; base < items * S; base += kW) {
    const int it = base + warp;
    const bool live = it < items * S;
    const int sl = live ? it / items : 0, tile = live ? it % items : 0;
    const int p0 = (tile % tp) * 8, q0 = (tile / tp) * 32;
    Tile<T> acc[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) acc[t].clear();
    if (live) {
      const int i1 = min(rows, (sl + 1) * per);
#pragma unroll 4
      for (int i = sl * per; i < i1; i += 4) {
        const bool in = i + kr < i1;
        const T a = in ? cj(la(i + kr, p0 + kc)) : zero<T>();
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (q0 + 8 * t >= q) break;
          acc[t].mma(a, in ? lb(i + kr, q0 + 8 * t + kc) : zero<T>());
        }
      }
    }
    for (int s = 0; s < S; ++s) {
      if (live && sl == s) {
        const int r = p0 + kc;
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int c = q0 + 8 * t + 2 * kr + h;
            if (r < p && c < q)
              Z[r + c * ldz] = s == 0 && !accumulate ? acc[t].get(h) : add(Z[r + c * ldz], acc[t].get(h));
          }
      }
      __syncthreads();
    }
  }
}

// Columns c < ncols of `rows` rows, src(c) -> first row of the column, copied to S (row stride lds) with asynchronous
// copies: whole rows of a column at a time, where the products' own operand reads would touch eight 32-byte sectors
// an instruction, again for every tile.
template <typename T, typename F> __device__ __forceinline__ void stage_cols(T* S, int lds, int rows, int ncols, F src) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = warp; c < ncols; c += kW) {
    const T* g = src(c);
    for (int i = lane; i < rows; i += 32) cp_async_zfill<sizeof(T)>(S + i + c * lds, g + i, true);
  }
  cp_async_commit();
}
__device__ __forceinline__ void stage_wait() {
  cp_async_wait<0>();
  __syncthreads();
}

// local_gram of the columns ca(a), a < p, and cb(b), b < q, staged through buf (cap entries, at least min_stage, or 0:
// read in place) in chunks of rows.  Returns the row stride when one chunk held all rows (the columns are then still
// in buf, A's first), else 0.
template <typename T, typename FA, typename FB>
__device__ int staged_gram(int rows, int p, int q, FA ca, FB cb, T* Z, int ldz, T* buf, int cap) {
  if (cap == 0) {
    local_gram<T>(
        rows, p, q, [&](int i, int c) { return c < p ? ca(c)[i] : zero<T>(); },
        [&](int i, int c) { return c < q ? cb(c)[i] : zero<T>(); }, Z, ldz);
    return 0;
  }
  int chunk = max(rows, 4), lds = pad_ld(chunk);
  while (chunk > 4 && (long)lds * (p + q) > cap) {
    chunk = max(4, ((chunk + 1) / 2 + 3) & ~3);
    lds = pad_ld(chunk);
  }
  const bool whole = chunk >= rows;
  int r = 0;
  do {
    const int nr = min(chunk, rows - r);
    stage_cols<T>(buf, lds, nr, p, [&](int c) { return ca(c) + r; });
    stage_cols<T>(buf + (size_t)lds * p, lds, nr, q, [&](int c) { return cb(c) + r; });
    stage_wait();
    const T *A = buf, *B = buf + (size_t)lds * p;
    local_gram<T>(
        nr, p, q, [&](int i, int c) { return c < p ? A[i + c * lds] : zero<T>(); },
        [&](int i, int c) { return c < q ? B[i + c * lds] : zero<T>(); }, Z, ldz, r > 0);
    r += chunk;
  } while (r < rows);
  return whole ? lds : 0;
}

// Entry e of the sum over the CTAs' partials (C x n in xch), in rank order.
template <typename T> __device__ __forceinline__ T rank_sum(const T* xch, int C, size_t n, size_t e) {
  T v[kMaxC];
#pragma unroll
  for (int r = 0; r < kMaxC; ++r) v[r] = r < C ? ldcg(xch + r * n + e) : zero<T>();
  T s = v[0];
#pragma unroll
  for (int r = 1; r < kMaxC; ++r) s = add(s, v[r]);
  return s;
}

// Sum of the CTAs' Z (p x q) into every CTA's Z, in rank order.  xch: this
// call's buffer in global memory ((C + 1) p q entries); consecutive calls
// alternate between two.  Every CTA adds up all entries (one barrier), or,
// from kTwoPhase entries on, its share of them, and reads the others' sums
// after a second barrier (C times fewer reads).
constexpr int kTwoPhase = 1024;
template <typename T>
__device__ void cluster_sum(cg::cluster_group& cl, T* Z, int ldz, int p, int q, T* xch) {
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  if (C == 1) return;
  const int n = p * q;
  for (int e = threadIdx.x; e < n; e += kT) xch[(size_t)rank * n + e] = Z[e % p + (e / p) * ldz];
  cl.sync();
  if (n < kTwoPhase) {
    for (int e = threadIdx.x; e < n; e += kT) Z[e % p + (e / p) * ldz] = rank_sum<T>(xch, C, n, e);
  } else {
    T* tot = xch + (size_t)C * n;
    for (int e = rank * kT + threadIdx.x; e < n; e += C * kT) tot[e] = rank_sum<T>(xch, C, n, e);
    cl.sync();
    for (int e = threadIdx.x; e < n; e += kT) Z[e % p + (e / p) * ldz] = ldcg(tot + e);
  }
  __syncthreads();
}

// out(i, c) = sum_k A(i, k) Z(k, c), or base(i, c) minus / plus it (OP -1 / +1), c < q, over 8-row strips of the
// local rows (NQ tiles of 8 columns in registers).  A strip is read whole before it is written, so out may alias A.
template <int NQ, int OP, typename T, typename LA, typename LC, typename ST>
__device__ void local_update(int rows, int kdim, int q, LA la, const T* Z, int ldz, LC lc, ST st) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kr = lane & 3, kc = lane >> 2;
  for (int i0 = warp * 8; i0 < rows; i0 += kW * 8) {
    Tile<T> acc[NQ];
#pragma unroll
    for (int t = 0; t < NQ; ++t) acc[t].clear();
    const bool rin = i0 + kc < rows;
#pragma unroll 4
    for (int k = 0; k < kdim; k += 4) {
      const bool kin = k + kr < kdim;
      const T a = rin && kin ? la(i0 + kc, k + kr) : zero<T>();
#pragma unroll
      for (int t = 0; t < NQ; ++t) {
        if (8 * t >= q) break;
        const int c = 8 * t + kc;
        acc[t].mma(a, kin && c < q ? Z[(k + kr) + c * ldz] : zero<T>());
      }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < NQ; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = 8 * t + 2 * kr + h;
        if (rin && c < q) {
          const T v = acc[t].get(h);
          st(i0 + kc, c, OP < 0 ? sub(lc(i0 + kc, c), v) : OP > 0 ? add(lc(i0 + kc, c), v) : v);
        }
      }
    __syncwarp();
  }
}

// Upper Cholesky factor of the q x q Hermitian G (upper triangle used) in place; false when a pivot is not
// positive.  *rmin: smallest diagonal entry; rinv[c] (shared) = 1 / R_cc.  Rows stay unscaled until the end (the update
// divides by the pivot), so a column costs one barrier.  All threads; ends at a block barrier.
template <typename T> __device__ bool block_cholesky(T* G, int ldg, int q, double* rmin, double* rinv) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  double dmin = 1e300;
  for (int c = 0; c < q; ++c) {
    const double d = re(G[c + c * ldg]);
    if (!(d > 0.0)) {  // the same value in every thread
      __syncthreads();
      return false;
    }
    dmin = fmin(dmin, d);
    const double id = 1.0 / d;
    for (int j = c + 1 + warp; j < q; j += kW) {
      const T g = mul(G[c + j * ldg], id);
      for (int i = c + 1 + lane; i <= j; i += 32) G[i + j * ldg] = sub(G[i + j * ldg], mul(cj(G[c + i * ldg]), g));
    }
    __syncthreads();
  }
  for (int c = warp; c < q; c += kW) {
    const double d = re(G[c + c * ldg]), r = sqrt(d), ir = 1.0 / r;
    __syncwarp();
    for (int j = c + lane; j < q; j += 32) G[c + j * ldg] = j == c ? mk<T>(r, 0.0) : mul(G[c + j * ldg], ir);
    if (lane == 0) rinv[c] = ir;
  }
  *rmin = sqrt(dmin);
  __syncthreads();
  return true;
}

// Ri = R^-1 (q x q, zero below the diagonal), one warp per column: lane l keeps entries l and l + 32.
template <typename T> __device__ void block_inverse(const T* R, int ldr, int q, const double* rinv, T* Ri, int ldi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = warp; c < q; c += kW) {
    T z0 = mk<T>(lane == c ? 1.0 : 0.0, 0.0), z1 = mk<T>(lane + 32 == c ? 1.0 : 0.0, 0.0);
    for (int i = c; i >= 0; --i) {
      const T zi = mul(i < 32 ? shfl(z0, i) : shfl(z1, i - 32), rinv[i]);
      if (lane < i) z0 = sub(z0, mul(R[lane + i * ldr], zi));
      if (lane + 32 < i) z1 = sub(z1, mul(R[lane + 32 + i * ldr], zi));
      if (lane == i) z0 = zi;
      if (lane + 32 == i) z1 = zi;
    }
    if (lane < q) Ri[lane + c * ldi] = lane <= c ? z0 : zero<T>();
    if (lane + 32 < q) Ri[lane + 32 + c * ldi] = lane + 32 <= c ? z1 : zero<T>();
  }
  __syncthreads();
}

// max |G - I| of the q x q Gram matrix (the same value in every thread)
template <typename T> __device__ double block_defect(const T* G, int ldg, int q, double* red) {
  double v = 0.0;
  for (int e = threadIdx.x; e < q * q; e += kT) {
    const int r = e % q, c = e / q;
    const T g = G[r + c * ldg];
    v = fmax(v, hypot(r == c ? re(g) - 1.0 : re(g), im(g)));
  }
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int w = 1; w < kW; ++w) v = fmax(v, red[w]);
  __syncthreads();
  return v;
}

constexpr double kSkipTol = 1e-12;  // a Cholesky-QR pass is skipped when its block is orthonormal to this

// W = orthonormal basis of the part of Tb(:, idx) outside span(X): two projections, columns scaled, two
// Cholesky-QR passes (a pass that finds the block orthonormal stops; a first pass that breaks down is repeated
// with a diagonal shift).  idx NULL: the columns in order.  status[0] = 1 when the block is rank deficient.
template <typename T, int NQ>
__global__ void __launch_bounds__(kT, 1)
    k_block_w(const T* __restrict__ X, int nd, const T* Tb, const int* __restrict__ idx, int na, T* W, long n,
              int rpc, int ldy, int ldz, int ldi, int staged, T* __restrict__ xch, long xch_len, int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[kW];
  __shared__ double scol[kMaxBlock], rinv[kMaxBlock];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  T* Y = reinterpret_cast<T*>(smem);       // rpc x na
  T* Z = Y + (size_t)ldy * na;             // max(nd, na) x na
  T* Ri = Z + (size_t)ldz * na;            // na x na
  T* S = Ri + (size_t)ldi * na;            // rpc x nd: X, when staged
  const long r0 = (long)rank * rpc;
  const int rows = (int)max(0L, min((long)rpc, n - r0));
  stage_cols<T>(Y, ldy, rows, na, [&](int c) { return Tb + r0 + (long)(idx ? idx[c] : c) * n; });
  if (staged) stage_cols<T>(S, ldy, rows, nd, [&](int c) { return X + r0 + (long)c * n; });
  stage_wait();
  int par = 0;
  auto ly = [&](int i, int c) { return c < na ? Y[i + c * ldy] : zero<T>(); };
  auto lx = [&](int i, int c) {
    return c >= nd ? zero<T>() : staged ? S[i + c * ldy] : X[r0 + i + (long)c * n];
  };
  auto sy = [&](int i, int c, T v) { Y[i + c * ldy] = v; };
  if (nd > 0) {
    local_gram<T>(rows, nd, na, lx, ly, Z, ldz);
    cluster_sum<T>(cl, Z, ldz, nd, na, xch + par * xch_len);
    par ^= 1;
    local_update<NQ, -1, T>(rows, nd, na, lx, Z, ldz, ly, sy);
    __syncthreads();
    // [X | Y]^H Y: the second projection and the Gram matrix in one sum.  Y - X Z has the Gram matrix G - Z^H Z,
    // with Z at rounding level after the first projection, so nothing cancels.
    local_gram<T>(
        rows, nd + na, na, [&](int i, int c) { return c < nd ? lx(i, c) : ly(i, c - nd); }, ly, Z, ldz);
    cluster_sum<T>(cl, Z, ldz, nd + na, na, xch + par * xch_len);
    par ^= 1;
    local_update<NQ, -1, T>(rows, nd, na, lx, Z, ldz, ly, sy);
    for (int e = threadIdx.x; e < na * na; e += kT) {
      const int r = e % na, c = e / na;
      T g = Z[nd + r + c * ldz];
      for (int k = 0; k < nd; ++k) g = sub(g, mul(cj(Z[k + r * ldz]), Z[k + c * ldz]));
      Ri[r + c * ldi] = g;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < na * na; e += kT) Z[e % na + (e / na) * ldz] = Ri[e % na + (e / na) * ldi];
    __syncthreads();
  }
  bool ok = true;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass > 0 || nd == 0) {
      local_gram<T>(rows, na, na, ly, ly, Z, ldz);
      cluster_sum<T>(cl, Z, ldz, na, na, xch + par * xch_len);
      par ^= 1;
    }
    if (pass == 0) {
      // the Gram matrix of the unit columns
      if (threadIdx.x < na) {
        const double d = re(Z[threadIdx.x + threadIdx.x * ldz]);
        scol[threadIdx.x] = d > 0.0 ? 1.0 / sqrt(d) : 0.0;
      }
      __syncthreads();
      for (int e = threadIdx.x; e < na * na; e += kT) {
        const int r = e % na, c = e / na;
        Z[r + c * ldz] = mul(Z[r + c * ldz], scol[r] * scol[c]);
      }
    } else if (threadIdx.x < na) {
      scol[threadIdx.x] = 1.0;
    }
    __syncthreads();
    if (block_defect<T>(Z, ldz, na, red) <= kSkipTol) {
      if (pass == 0) {
        for (int e = threadIdx.x; e < rows * na; e += kT) {
          const int i = e % rows, c = e / rows;
          Y[i + c * ldy] = mul(Y[i + c * ldy], scol[c]);
        }
        __syncthreads();
      }
      break;
    }
    double rmin;
    // keep a copy in Ri's place for the shifted retry
    for (int e = threadIdx.x; e < na * na; e += kT) Ri[e % na + (e / na) * ldi] = Z[e % na + (e / na) * ldz];
    __syncthreads();
    ok = block_cholesky<T>(Z, ldz, na, &rmin, rinv);
    if (!ok && pass == 0) {
      for (int e = threadIdx.x; e < na * na; e += kT) {
        const int r = e % na, c = e / na;
        T g = Ri[r + c * ldi];
        if (r == c) g = add(g, mk<T>(1e-10 * na, 0.0));
        Z[r + c * ldz] = g;
      }
      __syncthreads();
      ok = block_cholesky<T>(Z, ldz, na, &rmin, rinv);
    }
    if (!ok) break;
    block_inverse<T>(Z, ldz, na, rinv, Ri, ldi);
    for (int e = threadIdx.x; e < na * na; e += kT) {
      const int r = e % na, c = e / na;
      Ri[r + c * ldi] = mul(Ri[r + c * ldi], scol[r]);
    }
    __syncthreads();
    local_update<NQ, 0, T>(rows, na, na, ly, Ri, ldi, ly, sy);
    __syncthreads();
  }
  launch_release();
  for (int c = threadIdx.x >> 5; c < na; c += kW)
    for (int i = threadIdx.x & 31; i < rows; i += 32) W[r0 + i + (long)c * n] = Y[i + c * ldy];
  if (rank == 0 && threadIdx.x == 0) status[0] = ok ? 0 : 1;
}

// P, HP = the previous directions Pn(:, idx), HPn(:, idx) outside span(X, W), orthonormal: projection against the
// orthonormal columns [X | W], nx of them side by side in X and their H images in HX, columns that keep less than
// p_drop of their norm dropped, two Cholesky-QR passes.  status[1] = columns of P (0 when the block is nearly
// dependent).
template <typename T, int NQ>
__global__ void __launch_bounds__(kT, 1)
    k_block_p(const T* X, const T* HX, int nx, const T* __restrict__ Pn,
              const T* __restrict__ HPn, const int* idx, int np, T* P, T* HP, long n, int rpc, int ldy,
              int ldz, int ldi, int staged, double p_drop, T* xch, long xch_len, int* status) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[kW];
  __shared__ double scol[kMaxBlock], nu0[kMaxBlock], rinv[kMaxBlock];
  __shared__ int keep[kMaxBlock];
  __shared__ int nkeep_s;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  T* Y = reinterpret_cast<T*>(smem);
  T* Z = Y + (size_t)ldy * np;
  T* Ri = Z + (size_t)ldz * np;
  T* S = Ri + (size_t)ldi * np;     // rpc x nx, staged >= 1: [X | W], then [HX | HW]
  T* HY = S + (size_t)ldy * nx;     // rpc x np, staged == 2: HP
  launch_wait();
  const long r0 = (long)rank * rpc;
  const int rows = (int)max(0L, min((long)rpc, n - r0));
  stage_cols<T>(Y, ldy, rows, np, [&](int c) { return Pn + r0 + (long)idx[c] * n; });
  if (staged > 1) stage_cols<T>(HY, ldy, rows, np, [&](int c) { return HPn + r0 + (long)idx[c] * n; });
  auto stage = [&](const T* M) {
    if (!staged) return;
    __syncthreads();  // the readers of the last operand
    stage_cols<T>(S, ldy, rows, nx, [&](int c) { return M + r0 + (long)c * n; });
    stage_wait();
  };
  auto operand = [&](const T* M, int i, int c) { return staged ? S[i + c * ldy] : M[r0 + i + (long)c * n]; };
  stage(X);
  if (!staged) stage_wait();
  // squared column norms of this CTA's rows, summed with the projection (row nx of Z)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = warp; c < np; c += kW) {
    double s = 0.0;
    for (int i = lane; i < rows; i += 32) s += abs2(Y[i + c * ldy]);
    s = warp_sum(s);
    if (lane == 0) nu0[c] = s;
  }
  __syncthreads();
  int par = 0;
  auto ly = [&](int i, int c) { return c < np ? Y[i + c * ldy] : zero<T>(); };
  auto sy = [&](int i, int c, T v) { Y[i + c * ldy] = v; };
  auto lhp = [&](int i, int c) { return staged > 1 ? HY[i + c * ldy] : HP[r0 + i + (long)c * n]; };
  auto shp = [&](int i, int c, T v) {
    if (staged > 1) HY[i + c * ldy] = v;
    else HP[r0 + i + (long)c * n] = v;
  };
  // one projection against the orthonormal [X | W]
  local_gram<T>(rows, nx, np, [&](int i, int c) { return c < nx ? operand(X, i, c) : zero<T>(); }, ly, Z, ldz);
  if (threadIdx.x < np) Z[nx + threadIdx.x * ldz] = mk<T>(nu0[threadIdx.x], 0.0);
  __syncthreads();
  cluster_sum<T>(cl, Z, ldz, nx + 1, np, xch + par * xch_len);
  par ^= 1;
  if (threadIdx.x < np) nu0[threadIdx.x] = re(Z[nx + threadIdx.x * ldz]);
  local_update<NQ, -1, T>(rows, nx, np, [&](int i, int c) { return operand(X, i, c); }, Z, ldz, ly, sy);
  stage(HX);
  local_update<NQ, -1, T>(
      rows, nx, np, [&](int i, int c) { return operand(HX, i, c); }, Z, ldz,
      [&](int i, int c) { return staged > 1 ? HY[i + c * ldy] : HPn[r0 + i + (long)idx[c] * n]; }, shp);
  __syncthreads();
  int nk = np;
  bool ok = true;
  for (int pass = 0; pass < 2; ++pass) {
    auto lyk = [&](int i, int c) { return c < nk ? Y[i + c * ldy] : zero<T>(); };
    local_gram<T>(rows, nk, nk, lyk, lyk, Z, ldz);
    cluster_sum<T>(cl, Z, ldz, nk, nk, xch + par * xch_len);
    par ^= 1;
    if (pass == 0) {
      if (threadIdx.x == 0) {
        int k = 0;
        for (int c = 0; c < np; ++c) {
          const double d = re(Z[c + c * ldz]);
          if (d > p_drop * p_drop * nu0[c] && d > 0.0) {
            keep[k] = c;
            scol[k++] = 1.0 / sqrt(d);
          }
        }
        nkeep_s = k;
      }
      __syncthreads();
      nk = nkeep_s;
      if (nk == 0) break;
      // the scaled Gram matrix of the kept columns, through Ri
      for (int e = threadIdx.x; e < nk * nk; e += kT) {
        const int r = e % nk, c = e / nk;
        Ri[r + c * ldi] = mul(Z[keep[r] + keep[c] * ldz], scol[r] * scol[c]);
      }
      __syncthreads();
      for (int e = threadIdx.x; e < nk * nk; e += kT) Z[e % nk + (e / nk) * ldz] = Ri[e % nk + (e / nk) * ldi];
      __syncthreads();
    } else {
      if (threadIdx.x < nk) {
        keep[threadIdx.x] = threadIdx.x;
        scol[threadIdx.x] = 1.0;
      }
      __syncthreads();
      if (block_defect<T>(Z, ldz, nk, red) <= kSkipTol) break;
    }
    double rmin = 0.0;
    ok = block_cholesky<T>(Z, ldz, nk, &rmin, rinv);
    if (!ok || (pass == 0 && rmin < p_drop)) {
      nk = 0;
      break;
    }
    block_inverse<T>(Z, ldz, nk, rinv, Ri, ldi);
    for (int e = threadIdx.x; e < nk * nk; e += kT) {
      const int r = e % nk, c = e / nk;
      Ri[r + c * ldi] = mul(Ri[r + c * ldi], scol[r]);
    }
    __syncthreads();
    local_update<NQ, 0, T>(
        rows, nk, nk, [&](int i, int c) { return Y[i + keep[c] * ldy]; }, Ri, ldi, ly, sy);
    local_update<NQ, 0, T>(
        rows, nk, nk, [&](int i, int c) { return lhp(i, keep[c]); }, Ri, ldi, lhp, shp);
    __syncthreads();
  }
  for (int c = warp; c < nk; c += kW)
    for (int i = lane; i < rows; i += 32) {
      P[r0 + i + (long)c * n] = Y[i + c * ldy];
      if (staged > 1) HP[r0 + i + (long)c * n] = HY[i + c * ldy];
    }
  if (rank == 0 && threadIdx.x == 0) status[1] = nk;
}

// Subspace matrix Hs (m x m, m = nx + q) over [X(:, cols) | B]: diag(lam) (or (XX + XX^H) / 2 when XX is given), Z = B^H
// HX(:, cols), (G + G^H) / 2 with G = B^H HB.  cols NULL: the columns in order.
template <typename T>
__global__ void __launch_bounds__(kT, 1)
    k_block_rr(const T* B, const T* HB, int q, const T* HX,
               const int* __restrict__ cols, int nx, const double* __restrict__ lam, const T* __restrict__ XX, long n,
               int rpc, int ldz, int cap, T* __restrict__ xch, T* __restrict__ Hs) {
  extern __shared__ __align__(16) unsigned char smem[];
  T* Z = reinterpret_cast<T*>(smem);  // q x (nx + q), then the staging buffer
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const long r0 = (long)rank * rpc;
  const int rows = (int)max(0L, min((long)rpc, n - r0));
  const int m = nx + q, nz = q * m;
  staged_gram<T>(
      rows, q, m, [&](int c) { return B + r0 + (long)c * n; },
      [&](int c) { return c < nx ? HX + r0 + (long)(cols ? cols[c] : c) * n : HB + r0 + (long)(c - nx) * n; }, Z, ldz,
      Z + (size_t)ldz * m, cap);
  for (int e = threadIdx.x; e < nz; e += kT) xch[(size_t)rank * nz + e] = Z[e % q + (e / q) * ldz];
  cl.sync();
  launch_release();
  // entry (r, c) of B^H [HX | HB], summed over the CTAs
  auto entry = [&](int r, int c) { return rank_sum<T>(xch, C, nz, r + (size_t)c * q); };
  for (int e = rank * kT + threadIdx.x; e < m * m; e += C * kT) {
    const int r = e % m, c = e / m;
    T v;
    if (r < nx && c < nx) {
      if (XX) {
        const T a = XX[r + (long)c * nx], b = cj(XX[c + (long)r * nx]);
        v = mul(add(a, b), mk<T>(0.5, 0.0));
      } else {
        v = mk<T>(r == c ? lam[r] : 0.0, 0.0);
      }
    } else if (c < nx) {
      v = entry(r - nx, c);
    } else if (r < nx) {
      v = cj(entry(c - nx, r));
    } else {
      v = mul(add(entry(r - nx, c), cj(entry(c - nx, r))), mk<T>(0.5, 0.0));
    }
    Hs[e] = v;
  }
}

// Update of V = X (blockIdx.y 0) and of HV (1) over 8-row strips, one warp each: T = B C_b (C's rows nx .. nx + q - 1),
// Pn(:, t) = T(:, pcols[t]), X(:, cols) <- X(:, cols) C_x + T in place (a strip is read whole before it is written).
// Nothing is written when the eigensolve or W of this step failed (status[0], status[1]): the host reads the status a step
// late, and a failed step leaves the bands as they were.
constexpr int kUpdThreads = 128;
template <typename T, int NQ>
__global__ void __launch_bounds__(kUpdThreads)
    k_block_update(T* X, const T* __restrict__ B, T* Pn, T* HX, const T* __restrict__ HB, T* HPn, const T* Cm, int m, int nx, int q,
                   const int* __restrict__ cols, const int* __restrict__ pcols, int np, long n, const int* status) {
  T* x = blockIdx.y ? HX : X;
  const T* b = blockIdx.y ? HB : B;
  T* pn = blockIdx.y ? HPn : Pn;
  __shared__ int pos[kMaxBlock];  // column of Pn that takes column j of T, or -1
  __shared__ int xc[kMaxBlock];   // column of X behind subspace column j
  for (int j = threadIdx.x; j < nx; j += kUpdThreads) {
    pos[j] = -1;
    xc[j] = cols ? cols[j] : j;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < np; t += kUpdThreads) pos[pcols ? pcols[t] : t] = t;
  __syncthreads();
  launch_wait();
  launch_release();
  if (status[0] != 0 || status[1] != 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kr = lane & 3, kc = lane >> 2;
  const long i = ((long)blockIdx.x * (kUpdThreads / 32) + warp) * 8 + kc;
  const bool in = i < n;
  Tile<T> acc[NQ];
#pragma unroll
  for (int t = 0; t < NQ; ++t) acc[t].clear();
  auto run = [&](int k0, int kdim, auto la) {
#pragma unroll 4
    for (int k = 0; k < kdim; k += 4) {
      const bool kin = k + kr < kdim;
      const T a = in && kin ? la(k + kr) : zero<T>();
#pragma unroll
      for (int t = 0; t < NQ; ++t) {
        if (8 * t >= nx) break;
        const int c = 8 * t + kc;
        acc[t].mma(a, kin && c < nx ? Cm[k0 + k + kr + (long)c * m] : zero<T>());
      }
    }
  };
  run(nx, q, [&](int k) { return b[i + (long)k * n]; });
#pragma unroll
  for (int t = 0; t < NQ; ++t)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = 8 * t + 2 * kr + h;
      if (in && c < nx && pos[c] >= 0) pn[i + (long)pos[c] * n] = acc[t].get(h);
    }
  run(0, nx, [&](int k) { return x[i + (long)xc[k] * n]; });
  __syncwarp();
#pragma unroll
  for (int t = 0; t < NQ; ++t)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = 8 * t + 2 * kr + h;
      if (in && c < nx) x[i + (long)xc[c] * n] = acc[t].get(h);
    }
}

// hpsi += B D B^H psi: P = B^H psi summed over the cluster, Q = D P (D block-diagonal over atoms, blocks row-major) and
// the update of the rows, in one launch; one cluster for every bw bands.  Only the update reads what the launch before it
// (the last pass of the local part) wrote, so the sums run beside that pass.
template <typename T, int NQ>
__global__ void __launch_bounds__(kT, 1)
    k_block_nl(const T* __restrict__ B, int n_ch, const T* __restrict__ psi, long ldpsi, int nb_all, int bw,
               T* hpsi, long ldh, long n, int rpc, int ldz, int cap, T* xch, const int* __restrict__ ch_atom,
               const int* __restrict__ atom_ch_start, const int* __restrict__ d_off,
               const double* __restrict__ d_vals) {
  extern __shared__ __align__(16) unsigned char smem[];
  cg::cluster_group cl = cg::this_cluster();
  const int group = blockIdx.x / (int)cl.num_blocks(), first = group * bw, nb = min(bw, nb_all - first);
  psi += first * ldpsi;
  hpsi += first * ldh;
  xch += (size_t)group * (kMaxC + 1) * n_ch * bw;
  T* Z = reinterpret_cast<T*>(smem);    // n_ch x bw
  T* Q = Z + (size_t)ldz * bw;          // n_ch x bw
  const long r0 = (long)cl.block_rank() * rpc;
  const int rows = (int)max(0L, min((long)rpc, n - r0));
  T* buf = Q + (size_t)ldz * bw;
  const int lds = staged_gram<T>(
      rows, n_ch, nb, [&](int c) { return B + r0 + (long)c * n; },
      [&](int c) { return psi + r0 + (long)c * ldpsi; }, Z, ldz, buf, cap);
  auto lb = [&](int i, int c) { return lds ? buf[i + c * lds] : B[r0 + i + (long)c * n]; };
  cluster_sum<T>(cl, Z, ldz, n_ch, nb, xch);
  for (int e = threadIdx.x; e < n_ch * nb; e += kT) {
    const int c = e % n_ch, b = e / n_ch, a = ch_atom[c], s = atom_ch_start[a], nc = atom_ch_start[a + 1] - s;
    const double* drow = d_vals + d_off[a] + (long)(c - s) * nc;
    T acc = zero<T>();
    for (int j = 0; j < nc; ++j) acc = add(acc, mul(Z[s + j + b * ldz], drow[j]));
    Q[c + b * ldz] = acc;
  }
  __syncthreads();
  launch_wait();
  launch_release();
  for (int b0 = 0; b0 < nb; b0 += 8 * NQ)
    local_update<NQ, 1, T>(
        rows, n_ch, min(8 * NQ, nb - b0), lb, Q + (size_t)b0 * ldz, ldz,
        [&](int i, int c) { return hpsi[r0 + i + (long)(b0 + c) * ldh]; },
        [&](int i, int c, T v) { hpsi[r0 + i + (long)(b0 + c) * ldh] = v; });
}

// Rows per CTA and cluster size for n rows: at least 32 rows a CTA, rows in multiples of 8.
void split_rows(long n, int& C, int& rpc) {
  C = kMaxC;
  while (C > 1 && n < 32L * C) C /= 2;
  rpc = (int)(((n + C - 1) / C + 7) / 8 * 8);
}

template <typename T> size_t step_smem(int rpc, int cols, int zrows) {
  return ((size_t)pad_ld(rpc) + pad_ld(zrows) + pad_ld(cols)) * cols * sizeof(T);
}

// Bytes of a staging buffer for `cols` columns of up to rpc rows: all rows, or what is left, or 0 where that is less
// than the four rows a chunk needs.
template <typename T> size_t stage_bytes(int rpc, int cols, size_t left) {
  const size_t all = (size_t)pad_ld(std::max(rpc, 4)) * cols * sizeof(T);
  const size_t least = (size_t)pad_ld(4) * cols * sizeof(T);
  return all <= left ? all : left >= least ? left / sizeof(T) * sizeof(T) : 0;
}

template <typename K> Status opt_in(K kern, bool cluster) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  if (e == cudaSuccess && cluster) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return fail(kCuda, std::string("block step attributes: ") + cudaGetErrorString(e));
  return kOk;
}

// Per-device attributes, and whether 16-CTA clusters of these kernels can be resident.
template <typename T> Status configure(bool* fits) {
  static std::mutex mu;
  static std::set<int> good, bad;
  int dev = 0;
  PW_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (!good.count(dev) && !bad.count(dev)) {
    Status r;
    if ((r = opt_in(k_block_w<T, 4>, true)) != kOk || (r = opt_in(k_block_w<T, 8>, true)) != kOk ||
        (r = opt_in(k_block_p<T, 4>, true)) != kOk || (r = opt_in(k_block_p<T, 8>, true)) != kOk ||
        (r = opt_in(k_block_rr<T>, true)) != kOk || (r = opt_in(k_block_nl<T, 4>, true)) != kOk)
      return r;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(kMaxC, 1, 1);
    cfg.blockDim = dim3(kT, 1, 1);
    cfg.dynamicSmemBytes = kSmemMax;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kMaxC;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    const bool ok = cudaOccupancyMaxActiveClusters(&n, k_block_p<T, 8>, &cfg) == cudaSuccess && n > 0;
    if (!ok) cudaGetLastError();
    (ok ? good : bad).insert(dev);
  }
  *fits = good.count(dev) > 0;
  return kOk;
}

template <typename... P, typename... A>
Status launch_clusters(void (*kern)(P...), int C, int clusters, bool early, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(C * clusters, 1, 1);
  cfg.blockDim = dim3(kT, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  count_launch();
  if (e != cudaSuccess) return fail(kCuda, std::string("block step launch: ") + cudaGetErrorString(e));
  return kOk;
}
template <typename... P, typename... A>
Status launch(void (*kern)(P...), int C, bool early, size_t smem, cudaStream_t s, A... args) {
  return launch_clusters(kern, C, 1, early, smem, s, args...);
}

// Bands per cluster of the projector term: groups of eight or more, eight clusters at most.
int nl_group(int nb) {
  const int groups = std::min(8, (nb + 7) / 8);
  return ((nb + groups - 1) / groups + 7) / 8 * 8;
}

}  // namespace

template <typename T> bool block_steps_fit(long n, int nd) {
  if (nd < 1 || nd > kMaxBlock) return false;
  int C, rpc;
  split_rows(n, C, rpc);
  // P's block: nd columns, small matrices of 2 nd + 1 rows; the subspace matrix: 2 nd rows, 3 nd columns
  if (step_smem<T>(rpc, nd, 2 * nd + 1) > kSmemMax) return false;
  if ((size_t)pad_ld(2 * nd) * 3 * nd * sizeof(T) > kSmemMax) return false;
  bool fits = false;
  return configure<T>(&fits) == kOk && fits;
}

// One cluster of 16 SMs against library products on the whole GPU: the
// products of a step are ~n m^2 (m the columns of [X | W | P]), its serial
// part (Cholesky, inverse) ~m^2, the library's cost mostly its launches.  One
// step with every band active (m = 3 nd), library / fused in us, B200: real
// 1,045 rows nd 48 1220 / 980, 60 1390 / 1400; 2,517 rows nd 45 1200 / 1120,
// 56 1400 / 1530; 3,431 rows nd 40 940 / 830, 56 1450 / 1670; 6,187 rows nd 32
// 825 / 700, 40 980 / 1060; 22,119 rows nd 16 727 / 623; complex 1,045 rows
// nd 40 1210 / 1020; 2,517 rows nd 32 1040 / 910, 40 1180 / 1280; 6,187 rows nd
// 24 1030 / 860, 28 1090 / 1110.  Narrow blocks keep their gain in large boxes:
// 61,037 rows real nd 4 722 / 520, complex nd 3 960 / 642.
template <typename T> bool block_step_gains(long n, int m) {
  const double most = sizeof(T) == sizeof(double) ? 35e3 : 20e3;
  return (double)m * m * (1.0 + n / 3000.0) <= most;
}

size_t block_steps_xch(int nd) {
  // two buffers of (2 nd + 1) x nd, or one of 2 nd x 3 nd, per CTA and for the total
  return (size_t)(kMaxC + 1) * std::max<size_t>(2 * (size_t)(2 * nd + 1) * nd, (size_t)6 * nd * nd);
}

template <typename T>
Status block_w(const T* X, int nd, const T* Tb, const int* idx, int na, T* W, long n, T* xch, int* status,
               cudaStream_t s) {
  int C, rpc;
  split_rows(n, C, rpc);
  const int zr = nd + na, ldy = pad_ld(rpc), ldz = pad_ld(zr);
  size_t sm = step_smem<T>(rpc, na, zr);
  const size_t more = (size_t)ldy * nd * sizeof(T);
  const int staged = nd > 0 && sm + more <= kSmemMax;
  if (staged) sm += more;
  const long xl = (long)(kMaxC + 1) * (nd + na) * na;
  if (na <= 32)
    return launch(k_block_w<T, 4>, C, false, sm, s, X, nd, Tb, idx, na, W, n, rpc, ldy, ldz, pad_ld(na), staged, xch, xl, status);
  return launch(k_block_w<T, 8>, C, false, sm, s, X, nd, Tb, idx, na, W, n, rpc, ldy, ldz, pad_ld(na), staged, xch, xl, status);
}

template <typename T>
Status block_p(const T* X, const T* HX, int nx, const T* Pn, const T* HPn, const int* idx, int np, T* P, T* HP,
               long n, double p_drop, T* xch, int* status, cudaStream_t s) {
  int C, rpc;
  split_rows(n, C, rpc);
  const int ldy = pad_ld(rpc), ldz = pad_ld(nx + 1);
  size_t sm = step_smem<T>(rpc, np, nx + 1);
  const size_t op = (size_t)ldy * nx * sizeof(T), hp = (size_t)ldy * np * sizeof(T);
  const int staged = sm + op + hp <= kSmemMax ? 2 : sm + op <= kSmemMax ? 1 : 0;
  sm += staged == 2 ? op + hp : staged == 1 ? op : 0;
  const long xl = (long)(kMaxC + 1) * (nx + 1) * np;
  if (np <= 32)
    return launch(k_block_p<T, 4>, C, true, sm, s, X, HX, nx, Pn, HPn, idx, np, P, HP, n, rpc, ldy, ldz, pad_ld(np), staged,
                  p_drop, xch, xl, status);
  return launch(k_block_p<T, 8>, C, true, sm, s, X, HX, nx, Pn, HPn, idx, np, P, HP, n, rpc, ldy, ldz, pad_ld(np), staged,
                p_drop, xch, xl, status);
}

template <typename T>
Status block_rr(const T* B, const T* HB, int q, const T* HX, const int* cols, int nx, const double* lam, const T* XX,
                long n, T* xch, T* Hs, cudaStream_t s) {
  int C, rpc;
  split_rows(n, C, rpc);
  const int ldz = pad_ld(q);
  const size_t zb = (size_t)ldz * (nx + q) * sizeof(T);
  const size_t buf = stage_bytes<T>(rpc, nx + 2 * q, kSmemMax - zb);
  return launch(k_block_rr<T>, C, false, zb + buf, s, B, HB, q, HX, cols, nx, lam, XX, n, rpc, ldz, (int)(buf / sizeof(T)),
                xch, Hs);
}

template <typename T>
Status block_update(T* X, const T* B, T* Pn, T* HX, const T* HB, T* HPn, const T* Cm, int m, int nx, int q,
                    const int* cols, const int* pcols, int np, long n, const int* status, cudaStream_t s) {
  const dim3 grid((unsigned)((n + 8 * (kUpdThreads / 32) - 1) / (8 * (kUpdThreads / 32))), 2);
  if (nx <= 32)
    PW_CUDA_TRY(launch_early(k_block_update<T, 4>, grid, kUpdThreads, 0, s, X, B, Pn, HX, HB, HPn, Cm, m, nx, q, cols,
                             pcols, np, n, status));
  else
    PW_CUDA_TRY(launch_early(k_block_update<T, 8>, grid, kUpdThreads, 0, s, X, B, Pn, HX, HB, HPn, Cm, m, nx, q, cols,
                             pcols, np, n, status));
  count_launch();
  PW_CUDA_TRY(cudaGetLastError());
  return kOk;
}

// One launch is the faster form while the products are small: the clusters'
// tile products reach a fraction of the library products' rate, and each
// cluster reads all of B (n_ch columns) and its share of psi and H psi with 16
// SMs.  H|psi> in library / fused form, us, B200, by n_pw x channels x bands
// (complex): 1045 x 40 x 28 39 / 22, 1743 x 80 x 8 1.44 times as fast, 6187 x
// 24 x 16 1.16, 10059 x 8 x 16 62 / 53, 10059 x 16 x 28 88 / 84, 15419 x 4 x
// 16 1.13; but 2517 x 80 x 16 42 / 45, 6187 x 80 x 1 43 / 66, 12533 x 16 x 1
// 0.89, 10059 x 40 x 4 49 / 59, 22119 x 8 x 4 56 / 59, 76957 x 4 x 1 44 / 91.
// Packed real (a real entry is half the bytes, a multiply-add a quarter):
// 10059 x 40 x 16 72 / 60, 6187 x 80 x 16 71 / 65, 15419 x 16 x 28 74 / 72;
// but 15419 x 40 x 1 66 / 71, 22119 x 16 x 16 73 / 82, 10059 x 4 x 57 91 / 97,
// 6187 x 40 x 57 74 / 79.
template <typename T> bool nl_fused_ok(const Handle& h, int nb) {
  const double n = (double)h.n_pw, nc = (double)h.n_ch;
  if (h.n_ch < 1) return false;
  if (sizeof(T) == sizeof(double)) {
    if (n * nc * nb > 1.2e7 || n * (nc + 16) > 6e5 || n * nb > 4.4e5) return false;
  } else {
    if (n * nc * nb > 5e6 || n * (nc + 16) > 3.3e5 || n * nc > 1.95e5) return false;
  }
  if ((size_t)2 * pad_ld(h.n_ch) * nl_group(nb) * sizeof(T) > kSmemMax) return false;
  bool fits = false;
  return configure<T>(&fits) == kOk && fits;
}

// Room in the exchange buffer for nb bands (more bands never need less).
template <typename T> static Status ensure_nl_xch(Handle& h, int nb) {
  const int bw = nl_group(nb), clusters = (nb + bw - 1) / bw;
  const size_t need = (size_t)clusters * (kMaxC + 1) * h.n_ch * bw * sizeof(T);
  if (need <= h.nl_xch_bytes) return kOk;
  if (h.nl_xch) cudaFree(h.nl_xch);
  h.nl_xch = nullptr;
  h.nl_xch_bytes = 0;
  cudaError_t e = cudaMalloc(&h.nl_xch, need);
  if (e != cudaSuccess) return fail(kOom, std::string("cudaMalloc (projector exchange): ") + cudaGetErrorString(e));
  h.nl_xch_bytes = need;
  return kOk;
}

template <typename T> Status nl_fused_reserve(Handle& h, int nb) {
  if (!nl_fused_ok<T>(h, 1)) return kOk;
  while (!nl_fused_ok<T>(h, nb)) --nb;
  return ensure_nl_xch<T>(h, nb);
}

template <typename T>
Status nl_fused(Handle& h, const T* B, const T* psi, long ldpsi, int nb, T* hpsi, long ldh, cudaStream_t s) {
  const int bw = nl_group(nb), clusters = (nb + bw - 1) / bw;
  const Status st = ensure_nl_xch<T>(h, nb);
  if (st != kOk) return st;
  int C, rpc;
  split_rows(h.n_pw, C, rpc);
  const int ldz = pad_ld(h.n_ch);
  const size_t zb = (size_t)2 * ldz * bw * sizeof(T);
  const size_t buf = stage_bytes<T>(rpc, h.n_ch + bw, kSmemMax - zb);
  return launch_clusters(k_block_nl<T, 4>, C, clusters, true, zb + buf, s, B, h.n_ch, psi, ldpsi, nb, bw, hpsi, ldh,
                         (long)h.n_pw, rpc, ldz, (int)(buf / sizeof(T)), static_cast<T*>(h.nl_xch),
                         (const int*)h.ch_atom, (const int*)h.atom_ch_start, (const int*)h.d_off,
                         (const double*)h.d_vals);
}

#define PW_BLOCK(T)                                                                                                  \
  template bool nl_fused_ok<T>(const Handle&, int);                                                                 \
  template Status nl_fused_reserve<T>(Handle&, int);                                                                \
  template Status nl_fused<T>(Handle&, const T*, const T*, long, int, T*, long, cudaStream_t);                       \
  template bool block_steps_fit<T>(long, int);                                                                      \
  template bool block_step_gains<T>(long, int);                                                                     \
  template Status block_w<T>(const T*, int, const T*, const int*, int, T*, long, T*, int*, cudaStream_t);            \
  template Status block_p<T>(const T*, const T*, int, const T*, const T*, const int*, int, T*, T*, long, double, T*, \
                             int*, cudaStream_t);                                                                   \
  template Status block_rr<T>(const T*, const T*, int, const T*, const int*, int, const double*, const T*, long,     \
                              T*, T*, cudaStream_t);                                                                 \
  template Status block_update<T>(T*, const T*, T*, T*, const T*, T*, const T*, int, int, int, const int*,           \
                                  const int*, int, long, const int*, cudaStream_t);
PW_BLOCK(double)
PW_BLOCK(double2)
#undef PW_BLOCK

}  // namespace pwgpu
