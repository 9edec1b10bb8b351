// Block eigensolver of one (spin, k) Hamiltonian on the device (lobpcg.cu).
#pragma once

#include <vector>

#include "handle.hpp"

namespace pwgpu {

// Ritz block of one (spin, k): persists across SCF iterations.  V and HV hold
// n_pw x 3 nd columns, the current block X (nd), the preconditioned
// residual directions W and the previous-step directions P of the active
// bands.  X is orthonormal on return from the solver.
struct EigVecs {
  double2* V = nullptr;
  double2* HV = nullptr;
  std::vector<double> evals;  // nd Ritz values, ascending
  bool init = false;
};

// Scratch shared by all (spin, k) blocks of one handle.
struct EigWork {
  int nd = 0;
  long n = 0;
  double2* T = nullptr;    // n x nd: preconditioned residuals, then the new X
  double2* HXn = nullptr;  // n x nd: new HX
  double2* Pn = nullptr;   // n x nd: P of the last step (active bands)
  double2* HPn = nullptr;  // n x nd
  double2* Hs = nullptr;   // m x m (m <= 3 nd): subspace matrix, then eigenvectors (cuSOLVER)
  double2* Cs = nullptr;   // m x m: eigenvectors of the subspace matrix
  double2* G = nullptr;    // m x m: Gram / coupling blocks
  double2* Z = nullptr;    // m x m: coupling block, projection coefficients
  double2* Id = nullptr;   // m x m: identity of a shifted Cholesky, then the inverse of the factor
  double* lam = nullptr;   // m: Ritz values of the last subspace solve
  double* lam0 = nullptr;  // nd: Ritz values the residuals refer to
  double* colsq = nullptr; // 3 nd
  double* partials = nullptr;
  int* idx = nullptr;      // 3 nd
  int* status = nullptr;   // [0] subspace eigensolve, [1] W rank deficient, [2] columns of P (block steps)
  double2* xch = nullptr;  // exchange buffer of the block steps (nd <= kMaxBlock)
  double2* solver_work = nullptr;
  size_t solver_lwork = 0;
  int* info = nullptr;
  double* eigh_work = nullptr;  // scratch of the cluster eigensolver (eigh.cu)
  double2* XX = nullptr;        // nd x nd: X^H HX at the start of a solve
  double* defect = nullptr;     // max |Y^H Y - I| of a Cholesky-QR pass
  size_t eigh_work_len = 0;
};

struct EigStats {
  long happ = 0;     // H|psi> columns applied
  int iters = 0;     // block iterations
  double max_res = 0.0;  // largest residual norm over the first nconv bands, eV
};

Status eig_work_alloc(EigWork& w, long n, int nd);
void eig_work_release(EigWork& w);
Status eig_vecs_alloc(EigVecs& v, long n, int nd);
void eig_vecs_release(EigVecs& v);

// Lowest nd eigenpairs of H(spin, k) until the first nconv residual norms
// |H x - lambda x| fall below tol (eV) or max_iter block steps have run.
// HX is recomputed in FP64 on entry; the search directions W use
// `precision` (0 FP64, 1 mixed).  v0: mean V_eff(r), the preconditioner's
// diagonal shift.
Status lobpcg(Handle& h, EigWork& w, EigVecs& k, int spin, int ik, double v0, double tol, int max_iter, int nconv,
              int precision, EigStats& out);

// Fused block steps for narrow blocks (block_steps.cu), T = double or double2.
// block_steps_fit: whether a block of nd columns of n rows takes them.
constexpr int kMaxBlock = 64;
template <typename T> bool block_steps_fit(long n, int nd);
// block_step_gains: whether a step over a subspace of m columns is the faster one in these launches.
template <typename T> bool block_step_gains(long n, int m);
size_t block_steps_xch(int nd);  // entries of T in the exchange buffer
// W (n x na) = orthonormal basis of Tb(:, idx) outside span(X) (idx NULL: columns in order; nd 0: no projection, W
// may be Tb); status[0] = 1 when rank deficient.
template <typename T>
Status block_w(const T* X, int nd, const T* Tb, const int* idx, int na, T* W, long n, T* xch, int* status,
               cudaStream_t s);
// P, HP from Pn(:, idx), HPn(:, idx): projected out of the orthonormal columns [X | W] (nx of them side by side in X,
// their H images in HX), near-dependent columns dropped, orthonormal; status[1] = columns kept.
template <typename T>
Status block_p(const T* X, const T* HX, int nx, const T* Pn, const T* HPn, const int* idx, int np, T* P, T* HP,
               long n, double p_drop, T* xch, int* status, cudaStream_t s);
// Subspace matrix over [X(:, cols) | B], B = [W | P] with q columns (cols NULL: all in order).
template <typename T>
Status block_rr(const T* B, const T* HB, int q, const T* HX, const int* cols, int nx, const double* lam, const T* XX,
                long n, T* xch, T* Hs, cudaStream_t s);
// X(:, cols) and Pn from the subspace eigenvectors Cm (m x nx), and the same for HX, HPn; nothing when status[0] or
// status[1] (EigWork::status) tells that the step failed.
template <typename T>
Status block_update(T* X, const T* B, T* Pn, T* HX, const T* HB, T* HPn, const T* Cm, int m, int nx, int q,
                    const int* cols, const int* pcols, int np, long n, const int* status, cudaStream_t s);

}  // namespace pwgpu
