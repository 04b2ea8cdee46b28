// pb_gmres.cuh -- device-resident GMRES for the Jacobi-Davidson correction
// equations (instantiated in pb_gmres_D.cu and pb_gmres_S.cu).
//
// PHIST's subspacejada solves, per outer iteration, k correction equations
//     (I - Q Q')(A - sigma_j I) t_j = r_j
// with its blocked GMRES (src/jada/phist_jadaCorrectionSolver_def.hpp:372-
// 583; src/krylov/phist_blockedgmres_def.hpp).  There every Arnoldi step
// orthogonalises by iterated modified Gram-Schmidt, one mvec_dot_mvec per
// previous basis block, each a host round trip, and the Hessenberg matrix
// and Givens rotations live on the host.  Here the k systems run as k
// columns of one block: every basis block V_i is a contiguous n x k array,
// the Hessenberg matrices, rotations and residual estimates stay on the
// device, and the Gram-Schmidt step is classical with selective
// reorthogonalisation.  A step is the SpMMV and three passes over the basis
// (MINRES: two), each with the projection and the small dense work of the
// step inside (pb_krylov.cuh), without host synchronisation; after each step
// the host looks (without waiting) at a step counter and converged count the
// device writes into mapped host memory, and stops launching once every
// system has converged.
//
// The arithmetic of the GMRES iterate is PHIST's: x_0 = 0, Krylov space of
// the projected operator, Givens-rotated least squares; convergence when
// |g_{j+1}| < 1000 eps (absolute) or |g_{j+1}| / ||r_j|| < tol_j
// (phist_blockedgmres_def.hpp:604-606); restart after maxBas steps with the
// current iterate; at most maxIter steps in all; the solutions returned with
// unit norm (phist_jadaCorrectionSolver_def.hpp:576-578).  The small dense
// part (Hessenberg, rotations, triangular solve) is FP64 in both precisions.
//
// MINRES (phist_b200_{D,S}jadaCorrection_minres) is the same solver with
// PHIST's blocked MINRES step (src/krylov/phist_blockedminres_def.hpp:
// 185-277) in place of the Gram-Schmidt step: the Lanczos three-term
// recurrence alpha = V_j'W, W -= alpha V_j + beta V_{j-1} with beta the
// previous step's norm, beta' = ||W||, so H is tridiagonal and a step costs
// two passes over W whatever its index; the basis is kept (PHIST's ring
// buffer) for the update of the iterate, the rotations, least squares and
// restarts are GMRES's, and the absolute threshold is 100 eps
// (blockedminres_def.hpp:157).  For symmetric A and real shifts only, as in
// PHIST.
#pragma once
#include <algorithm>
#include <atomic>
#include <cmath>
#include <limits>
#include <vector>

#include "pb_api.cuh"
#include "pb_krylov.cuh"
#include "pb_spmmv_lz.cuh"

namespace pb {
namespace {

template <class T>
struct DBuf {
  T* p = nullptr;
  explicit DBuf(size_t count) { p = (T*)rt().dmalloc(sizeof(T) * (count ? count : 1)); }
  ~DBuf() { rt().dfree(p); }
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
};

template <class T>
void raw_view(Mvec<T>& m, T* d, int64_t n, int w, int64_t ld)
{
  m.map = nullptr;
  m.nrows = (int32_t)n;
  m.nvec = w;
  m.lda = ld;
  m.root = &m;
  m.col_off = 0;
  m.d_base = d;
  m.h_base = nullptr;
}

// dst(i, s) = src(i, s) * f[s]
template <class T>
__global__ void k_gm_scale_cols(const T* __restrict__ src, int64_t lds, T* dst, int64_t ldd, int64_t n, int k,
                                const T* __restrict__ f)
{
  PB_FOR_ELEMS(n, k, i, s) dst[i * ldd + s] = src[i * lds + s] * f[s];
}

// y_s = H(0:J_s, 0:J_s, s)^{-1} g(0:J_s, s), J_s = jcount[s], stored negated
// and with the basis factors as update coefficients: Y[i*k + s] = -F_i y_s(i)
// for i < J_s, 0 up to Jmax (x -= sum_i V_i Y_i is then x += V y).  One warp
// per system, 8 systems a block (the registers of 32 warps would not fit one
// SM): lane l holds the rows l and l + 32 and the columns go from the right,
// 4 columns of H loaded ahead of the chain of subtractions.
constexpr int GM_SOLVE_NW = 8;
template <class T>
__global__ void __launch_bounds__(32 * GM_SOLVE_NW)
k_gm_solve(const double* __restrict__ H, const double* __restrict__ g, const int* __restrict__ jcount, int k, int m,
           int Jmax, const T* __restrict__ F, T* Y)
{
  const int s = blockIdx.x * GM_SOLVE_NW + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (s >= k) return;
  const int J = jcount[s];
  double v0 = lane < J ? g[lane * k + s] : 0.0;
  double v1 = lane + 32 < J ? g[(lane + 32) * k + s] : 0.0;
  double y0 = 0.0, y1 = 0.0;
  for (int l0 = J - 1; l0 >= 0; l0 -= 4) {
    double h0[4], h1[4], d[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int l = l0 - u;
      h0[u] = (l >= 0 && lane < l) ? H[((int64_t)lane * m + l) * k + s] : 0.0;
      h1[u] = (l >= 0 && lane + 32 < l) ? H[((int64_t)(lane + 32) * m + l) * k + s] : 0.0;
      d[u] = l >= 0 ? H[((int64_t)l * m + l) * k + s] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int l = l0 - u;
      if (l < 0) break;
      const double v = __shfl_sync(0xffffffffu, l < 32 ? v0 : v1, l & 31);
      const double y = d[u] != 0.0 ? v / d[u] : 0.0;
      if (l == lane) y0 = y;
      if (l == lane + 32) y1 = y;
      v0 -= h0[u] * y;
      v1 -= h1[u] * y;
    }
  }
  if (lane < Jmax) Y[lane * k + s] = lane < J ? (T)(-(double)F[lane * k + s] * y0) : T(0);
  if (lane + 32 < Jmax) Y[(lane + 32) * k + s] = lane + 32 < J ? (T)(-(double)F[(lane + 32) * k + s] * y1) : T(0);
}

// The grid of a pass: want blocks for all groups of systems, the groups side by
// side, at most one wave of perSM blocks; partials and counters for it (the
// first level of the sum as in pb_frag.cu, the lane's 64 counters shared out)
template <class T>
dim3 kry_grid(KryArgs<T>& a, int64_t want, int perSM)
{
  const int ngrp = (int)ceil_div(a.k, KRY_MAXC);
  const int grid = (int)std::min<int64_t>(want, std::max(1, perSM * rt().num_sms() / ngrp));
  a.cnt_step = 64 / ngrp;
  a.gsz = std::max((int)std::ceil(std::sqrt((double)grid)), (int)ceil_div(grid, a.cnt_step - 2));
  a.part_step = (grid + ceil_div(grid, a.gsz)) * KRY_MAXOUT;
  a.part = (double*)rt().scratch(sizeof(double) * (size_t)a.part_step * ngrp);
  a.counters = rt().counters();
  return dim3((unsigned)grid, (unsigned)ngrp);
}

template <class T, int MQ, int MJ, bool UPD, bool DOTS>
void kry_launch(KryArgs<T>& a)
{
  // two blocks per SM: the launch bound
  launch_pdl(k_kry<T, MQ, MJ, UPD, DOTS>, kry_grid(a, ceil_div(a.n, 32 * FRAG_NW), 2), FRAG_BS, 0, a);
  PB_LAUNCH_CHECK();
}

// the instantiation with the fewest register-held blocks that cover a.nb
template <class T, int MQ, bool UPD>
void kry_dots_mj(KryArgs<T>& a)
{
  if (a.nb <= 2) kry_launch<T, MQ, 2, UPD, true>(a);
  else if (a.nb <= 8) kry_launch<T, MQ, 8, UPD, true>(a);
  else if (a.nb <= 16) kry_launch<T, MQ, 16, UPD, true>(a);
  else kry_launch<T, MQ, KRY_MAXJ, UPD, true>(a);
}

// sums of Q'W, V'W (and an update before them): a.nq columns of Q
template <class T, bool UPD>
void kry_dots(KryArgs<T>& a)
{
  if (a.nq == 0) kry_dots_mj<T, 0, UPD>(a);
  else if (a.nq <= 16) kry_dots_mj<T, 2, UPD>(a);
  else kry_dots_mj<T, 4, UPD>(a);
}

// the update alone; blocks beyond two go without Q
template <class T>
void kry_update(KryArgs<T>& a)
{
  if (a.nb <= 2) {
    if (a.nq == 0) kry_launch<T, 0, 2, true, false>(a);
    else if (a.nq <= 16) kry_launch<T, 2, 2, true, false>(a);
    else kry_launch<T, 4, 2, true, false>(a);
  } else if (a.nb <= 8) kry_launch<T, 0, 8, true, false>(a);
  else if (a.nb <= 16) kry_launch<T, 0, 16, true, false>(a);
  else kry_launch<T, 0, KRY_MAXJ, true, false>(a);
}

// W = (A - sigma I) V_j F_j with Q'W and V_j'W (pb_spmmv_lz.cuh): 4 or 8
// systems whose rows are one 16- or 32-byte vector a thread, rows of at most 8
// entries, at most 16 projection columns.  False otherwise.
template <class T, int NV>
bool spmv_lanczos_nv(const SparseMat<T>* A, const T* negsig, const Mvec<T>* X, Mvec<T>* W, const T* cscale,
                     KryArgs<T>& a)
{
  constexpr int TPR = 2, VB = NV / TPR * (int)sizeof(T);
  if (((uintptr_t)X->d() | (uintptr_t)W->d()) % VB != 0) return false;
  SpmvArgs<T> p;
  memset(&p, 0, sizeof(p));
  p.alpha = T(1);
  p.x = X->d();
  p.ldx = X->lda;
  p.y = W->d();
  p.ldy = W->lda;
  p.nvec = NV;
  p.cscale = cscale;
  p.has_shift = 1;
  for (int s = 0; s < NV; s++) p.sh[s] = negsig[s];
  auto kern = k_sell_spmmv_lz<T, NV, TPR, VB>;
  static std::atomic<int> occ{0};
  int o = occ.load();
  if (o == 0) {
    PB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, LZ_NT, 0));
    o = std::max(1, o);
    occ.store(o);
  }
  launch_pdl(kern, kry_grid(a, ceil_div(A->nchunks, LZ_NT / TPR / 32), o), LZ_NT, 0, sell_dev(A), p, a);
  PB_LAUNCH_CHECK();
  return true;
}

template <class T>
bool spmv_lanczos(const SparseMat<T>* A, const T* negsig, const Mvec<T>* X, Mvec<T>* W, const T* cscale,
                  KryArgs<T>& a)
{
  if (!rt().spmv_pf || !rt().spmv_v256 || A->C != 32 || A->max_row_len > 8 || A->nnz == 0) return false;
  if (a.nq < 1 || a.nq > LZ_MAXQ) return false;
  if (a.k == 8) return spmv_lanczos_nv<T, 8>(A, negsig, X, W, cscale, a);
  if (a.k == 4) return spmv_lanczos_nv<T, 4>(A, negsig, X, W, cscale, a);
  return false;
}

}  // namespace

// W = alpha V C + beta W on device operands (C col-major m x k, ld ldc)
template <class T>
static void gm_mvsd(int64_t n, int m, int k, T alpha, const T* V, int64_t ldv, const T* C, int64_t ldc, T beta, T* W,
                    int64_t ldw)
{
  RowGemmArgs<T> a = rowgemm_args<T>();
  a.n = n;
  a.m = m;
  a.k = k;
  a.mv = 0;
  a.V = V;
  a.ldv = ldv;
  a.W = W;
  a.ldw = ldw;
  a.C = C;
  a.ldc = ldc;
  a.alpha = alpha;
  a.beta = beta;
  a.mode = RM_MVSD;
  a.gram = GM_NONE;
  launch_rowgemm<T>(a);
}

// lanczos: MINRES (three-term recurrence), else GMRES
template <class T>
int jada_krylov(const SparseMat<T>* A, const Mvec<T>* Q, const Mvec<T>* R, const int* resIndex, int k,
                const double* sigma, const double* tol, int maxIter, int maxBas, Mvec<T>* t, bool lanczos)
{
  PB_REQUIRE(A && R && t && sigma && tol, PB_INVALID_INPUT, "NULL argument");
  PB_REQUIRE(k >= 1 && k <= 32, PB_INVALID_INPUT, "1..32 systems per call (got %d)", k);
  PB_REQUIRE(t->nvec == k, PB_INVALID_INPUT, "t has %d columns, expected %d", t->nvec, k);
  PB_REQUIRE(maxIter >= 1, PB_INVALID_INPUT, "maxIter must be >= 1");
  const int64_t n = A->nrows;
  PB_REQUIRE(A->ncols == n && R->nrows == n && t->nrows == n && (!Q || Q->nrows == n), PB_INVALID_INPUT,
             "operand rows do not match the matrix");
  for (int s = 0; s < k; s++) {
    const int idx = resIndex ? resIndex[s] : s;
    PB_REQUIRE(idx >= 0 && idx < R->nvec, PB_INVALID_INPUT, "resIndex[%d] = %d out of range", s, idx);
  }
  if (n == 0) return 0;  // every residual is zero: converged with no step
  const int nq = Q ? Q->nvec : 0;
  // a projection block of at most KRY_MAXQ columns goes with the passes over
  // the basis, a wider one in products of its own
  const bool fuse = nq > 0 && nq <= KRY_MAXQ;
  const int m = std::max(1, std::min(std::min(maxBas > 0 ? maxBas : maxIter, maxIter), 63));
  const int64_t nk = n * (int64_t)k;  // one basis block
  const double eps_abs = (lanczos ? 100.0 : 1000.0) * std::numeric_limits<T>::epsilon();

  DBuf<T> V((size_t)nk * (m + 1)), X((size_t)nk);
  DBuf<T> Y((size_t)(m + 1) * k), Cq((size_t)std::max(nq, 2) * k), F((size_t)(m + 1) * k), f(k);
  DBuf<T> hv((size_t)(m + 1) * k), hv2((size_t)(m + 1) * k);
  DBuf<double> H((size_t)(m + 1) * m * k), cs((size_t)m * k), sn((size_t)m * k), g((size_t)(m + 1) * k), bnorm(k);
  DBuf<double> h1((size_t)(m + 1) * k), h2((size_t)(m + 1) * k), nrm0(k), nf(k);
  const int ngrp = (int)ceil_div(k, KRY_MAXC);
  DBuf<int> conv(k), jcount(k), reorth(ngrp), gflag(ngrp);
  std::vector<T> negsig(k);
  for (int s = 0; s < k; s++) negsig[s] = (T)(-sigma[s]);
  volatile unsigned long long* hflags = (volatile unsigned long long*)rt().mailbox_host();
  const int gw = grid_for(n * (int64_t)k);
  DBuf<double> gq((size_t)(fuse ? nq + m + 2 : 0) * k);  // g0, gam, dq

  Mvec<T> mX, mW, mVj;
  raw_view(mX, X.p, n, k, k);

  KryArgs<T> base;
  memset(&base, 0, sizeof(base));
  base.n = n;
  base.k = k;
  base.per = (int)ceil_div(k, ngrp);  // even groups: they share the SMs evenly
  base.Q = fuse ? Q->d() : nullptr;
  base.ldq = fuse ? Q->lda : 0;
  base.vstep = nk;
  base.R = R->d();
  base.ldr = R->lda;
  {
    KryEpi<T>& e = base.e;
    e.k = k;
    e.m = m;
    e.lanczos = lanczos ? 1 : 0;
    e.H = H.p; e.cs = cs.p; e.sn = sn.p; e.g = g.p; e.bnorm = bnorm.p;
    e.h1 = h1.p; e.h2 = h2.p; e.nrm0 = nrm0.p; e.nf = nf.p;
    e.F = F.p; e.cq = Cq.p; e.hv = hv.p; e.hv2 = hv2.p; e.finv = f.p;
    e.conv = conv.p; e.jcount = jcount.p;
    e.eps_abs = eps_abs;
    // 100 eps of the new direction: dots of a pass that left nothing but
    // rounding stay below it
    const double lim = 100.0 * std::numeric_limits<T>::epsilon();
    e.h2_lim = lim * lim;
    e.g0 = gq.p; e.gam = gq.p + (size_t)nq * k; e.dq = e.gam + (size_t)(m + 1) * k;
    e.flags = (unsigned long long*)rt().mailbox_dev();
    e.reorth = reorth.p;
    e.gflag = fuse ? gflag.p : nullptr;
    for (int s = 0; s < k; s++) {
      base.idx.v[s] = resIndex ? resIndex[s] : s;
      e.tol.v[s] = tol[s];
    }
  }
  // W = P W with P = I - Q Q' (outside the fused passes)
  auto project = [&](T* W) {
    if (nq == 0) return;
    launch_mvTmv<T>(n, nq, k, T(1), Q->d(), Q->lda, W, k, T(0), Cq.p, nq);
    gm_mvsd<T>(n, nq, k, T(-1), Q->d(), Q->lda, Cq.p, nq, T(1), W, k);
  };

  auto converged = [&] {
    int c = 0;
    for (int q = 0; q < ngrp; q++) c += (int)(hflags[q] >> 32);
    return c;
  };
  int total = 0, nconv = 0;
  for (int cycle = 0; total < maxIter && nconv < k; cycle++) {
    if (cycle > 0) {
      // restart from the current iterate: V_0 = R - P (A - sigma I) X, converged systems zero
      raw_view(mW, V.p, n, k, k);
      spmv_general<T>(T(1), A, negsig.data(), &mX, T(0), &mW, nullptr, nullptr, T(0), T(0), nullptr);
      project(V.p);
    }
    {
      KryArgs<T> a = base;
      a.W = V.p;
      a.restart = cycle > 0 ? 1 : 0;
      a.e.first = cycle == 0 ? 1 : 0;
      a.e.kind = fuse ? KE_NONE : KE_START;
      launch_pdl(k_kry_start<T>, kry_grid(a, ceil_div(n * std::min(k, KRY_MAXC), 4 * FRAG_BS), 4), FRAG_BS, 0, a);
      PB_LAUNCH_CHECK();
      if (fuse) {
        // the norms together with Q'V_0
        a.nq = nq;
        a.V = a.W;
        a.Win = a.W;
        a.e.kind = KE_START;
        kry_dots<T, false>(a);
      }
    }
    for (int q = 0; q < ngrp; q++) hflags[q] = 0;
    int j = 0, steps = 0;
    const int jmax = std::min(m, maxIter - total);
    bool stop = false;
    for (j = 0; j < jmax && !stop; j++) {
      // W = (A - sigma I) v_j, in the place of V_{j+1}
      T* Wj = V.p + (int64_t)(j + 1) * nk;
      raw_view(mVj, V.p + (int64_t)j * nk, n, k, k);
      raw_view(mW, Wj, n, k, k);
      bool dotted = false;  // Q'W and V_j'W came with the SpMMV
      if (lanczos && fuse && ngrp == 1) {
        KryArgs<T> a = base;
        a.nq = nq;
        a.e.j = j;
        a.e.kind = KE_LZ;
        dotted = spmv_lanczos<T>(A, negsig.data(), &mVj, &mW, F.p + (int64_t)j * k, a);
      }
      if (!dotted)
        spmv_general<T>(T(1), A, negsig.data(), &mVj, T(0), &mW, nullptr, nullptr, T(0), T(0), nullptr,
                        F.p + (int64_t)j * k);
      if (!fuse) project(Wj);
      const int J = j + 1;
      // one pass: blocks [i0, i0 + nb), with Q when it is the first
      auto pass = [&](bool upd, bool dots, int i0, int nb, bool withq, const T* hc, int kind, bool last,
                      const int* skip) {
        KryArgs<T> a = base;
        a.W = Wj;
        a.Win = Wj;
        a.nq = (fuse && withq) ? nq : 0;
        a.V = V.p + (int64_t)i0 * nk;
        a.nb = nb;
        a.cq = Cq.p;
        a.hv = hc;
        a.skip = skip;
        a.e.j = j;
        a.e.i0 = i0;
        a.e.kind = kind;
        a.e.last = last;
        if (upd && lanczos) a.vstep = -nk;  // V_j, then V_{j-1}
        if (upd && dots) kry_dots<T, true>(a);
        else if (dots) kry_dots<T, false>(a);
        else kry_update<T>(a);
      };
      if (lanczos) {
        // [Q V_j]'W; W -= Q (Q'W) + v_j alpha + v_{j-1} beta and its norm
        // (alpha = v_j'(P W) from both dots; PHIST's order: projection,
        // then the Lanczos terms)
        if (!dotted) pass(false, true, j, 1, true, nullptr, KE_LZ, true, nullptr);
        pass(true, false, j, j > 0 ? 2 : 1, true, hv.p, KE_STEP, true, nullptr);
      } else {
        // Gram-Schmidt against Q and V_0..V_j: h1 = V'(P W) from V'W and Q'W
        // (kry_epilogue); W -= Q (Q'W) + V h1 and h2 = V'W of the result; a
        // second subtraction only where that is needed (a device flag); the
        // rest of the step follows in whichever launch finishes W
        if (J <= KRY_MAXJ) {
          pass(false, true, 0, J, true, nullptr, KE_GS, true, nullptr);
          pass(true, true, 0, J, true, hv.p, KE_GS2, true, nullptr);
        } else {
          for (int i0 = 0; i0 < J; i0 += KRY_MAXJ)
            pass(false, true, i0, std::min(KRY_MAXJ, J - i0), i0 == 0, nullptr, KE_GS, true, nullptr);
          if (fuse) pass(true, false, 0, 0, true, hv.p, KE_NONE, true, nullptr);
          for (int i0 = 0; i0 < J; i0 += KRY_MAXJ)
            pass(true, false, i0, std::min(KRY_MAXJ, J - i0), false, hv.p + (int64_t)i0 * k, KE_NONE, true, nullptr);
          for (int i0 = 0; i0 < J; i0 += KRY_MAXJ)
            pass(false, true, i0, std::min(KRY_MAXJ, J - i0), false, nullptr, KE_GS2, i0 + KRY_MAXJ >= J, nullptr);
        }
        for (int i0 = 0; i0 < J; i0 += KRY_MAXJ) {
          const bool end = i0 + KRY_MAXJ >= J;
          pass(true, false, i0, std::min(KRY_MAXJ, J - i0), false, hv2.p + (int64_t)i0 * k, end ? KE_STEP : KE_NONE,
               true, reorth.p);
        }
      }
      steps = j + 1;
      // stop launching once the device reports every system converged (a
      // look at the flags, no wait: the host never blocks inside a cycle,
      // so concurrent solves on other threads keep their cores)
      if (converged() >= k) stop = true;
    }
    total += steps;
    // x += [V_0..V_{J-1}] y with J the largest step count of a system
    rt().sync();
    nconv = converged();
    const int J = steps;
    k_gm_solve<T><<<(int)ceil_div(k, GM_SOLVE_NW), 32 * GM_SOLVE_NW, 0, stream()>>>(H.p, g.p, jcount.p, k, m, J, F.p, Y.p);
    PB_LAUNCH_CHECK();
    for (int i0 = 0; i0 < J; i0 += KRY_MAXJ) {
      KryArgs<T> a = base;
      a.W = X.p;
      a.Win = (cycle == 0 && i0 == 0) ? nullptr : a.W;
      a.V = V.p + (int64_t)i0 * nk;
      a.nb = std::min(KRY_MAXJ, J - i0);
      a.hv = Y.p + (int64_t)i0 * k;
      a.e.kind = KE_NORM;
      kry_update<T>(a);
    }
  }
  // t = x / ||x||, column by column
  k_gm_scale_cols<T><<<gw, 256, 0, stream()>>>(X.p, k, t->d(), t->lda, n, k, f.p);
  PB_LAUNCH_CHECK();
  std::vector<int> hc(k);
  PB_CUDA(cudaMemcpyAsync(hc.data(), conv.p, sizeof(int) * k, cudaMemcpyDeviceToHost, stream()));
  rt().sync();
  int unconverged = 0;
  for (int s = 0; s < k; s++) unconverged += hc[s] ? 0 : 1;
  return unconverged;
}

template <class T>
int jada_gmres(const SparseMat<T>* A, const Mvec<T>* Q, const Mvec<T>* R, const int* resIndex, int k,
               const double* sigma, const double* tol, int maxIter, int maxBas, Mvec<T>* t)
{
  return jada_krylov<T>(A, Q, R, resIndex, k, sigma, tol, maxIter, maxBas, t, false);
}
template <class T>
int jada_minres(const SparseMat<T>* A, const Mvec<T>* Q, const Mvec<T>* R, const int* resIndex, int k,
                const double* sigma, const double* tol, int maxIter, int maxBas, Mvec<T>* t)
{
  return jada_krylov<T>(A, Q, R, resIndex, k, sigma, tol, maxIter, maxBas, t, true);
}

}  // namespace pb
