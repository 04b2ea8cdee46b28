// pb_prec.cuh -- compensated block products for PHIST_ROBUST_REDUCTIONS.
//
// PHIST's builtin library computes V'W in double-double when the caller sets
// PHIST_ROBUST_REDUCTIONS (mvec_module.F90:2421-2747 dispatching to
// gemm_kernels_sC_prec.c): orthogrrB passes the flag to every Gram product
// it needs (phist_orthogrr_def.hpp:89,152,167), and orthog then aims at
// ||Q'Q - I|| < eps*sqrt(eps) (phist_orthog_def.hpp:42-43).
//
// Here each output C(r,j) = sum_i V(i,r) W(i,j) is accumulated with Dot2
// (Ogita, Rump and Oishi, "Accurate sum and dot product", SIAM J. Sci.
// Comput. 26(6), 2005): every product is split exactly into p + e by an FMA
// (TwoProduct), p is added to the running sum with TwoSum, and the rounding
// errors of both are collected in a second accumulator.
//
// Ten FP64 operations per product make the kernel bound by the FP64 pipe.
// A warp streams its own rows straight from global memory: lane (li, lj)
// owns, in each of MT tiles of 8 columns of V, column li against TJ columns
// of W, so a loaded value serves a whole tile and nothing is staged or
// synchronised (staging 32-row tiles through shared memory, one output per
// thread, took 84 us for 8 x 8 at n = 262,144, most of it waiting).  The
// (sum, error) pairs of warps and blocks are combined in fixed order with
// TwoSum, the blocks in two levels of about sqrt(blocks), so the result does
// not depend on the schedule.  Finally C = alpha*(s + c) + beta*C is
// evaluated in double-double and rounded once.
#pragma once
#include "pb_frag.cuh"

namespace pb {

__device__ __forceinline__ void dd_two_sum(double a, double b, double& s, double& e)
{
  s = a + b;
  const double z = s - a;
  e = (a - (s - z)) + (b - z);
}

// s + c += x*y (one Dot2 step)
__device__ __forceinline__ void dd_dot_step(double x, double y, double& s, double& c)
{
  const double p = x * y;
  const double ep = fma(x, y, -p);
  double t, et;
  dd_two_sum(s, p, t, et);
  s = t;
  c += ep + et;
}

// (s, c) += (s2, c2)
__device__ __forceinline__ void dd_add(double& s, double& c, double s2, double c2)
{
  double t, et;
  dd_two_sum(s, s2, t, et);
  s = t;
  c += c2 + et;
}

struct MvTmvPrecArgs {
  int64_t n;
  int m, k;           // columns of V (at most 64) and W (at most 8)
  const double* V;
  int64_t ldv;
  const double* W;
  int64_t ldw;
  double alpha, beta;
  double* C;          // C(i, j) at C[i*sr + j*sc]
  int64_t sr, sc;
  int mirror;         // W'W: outputs with i < mirror also go to
  double* Cm;         // Cm[j*sr + i*sc]
  double *mbox, *mboxm; int mr, mc;  // copies of C and Cm in mapped host memory (or NULL), strides mr, mc
  double* part;       // [blocks + groups][m*k][2]
  int gsz;
  unsigned int* counters;
};

// the two-level sum of frag_tree_sum on (sum, error) pairs
template <int NQ>
__device__ __forceinline__ bool prec_tree_sum(double* part, int nout, int gsz, unsigned int* counters, double (&s)[NQ],
                                              double (&c)[NQ])
{
  __shared__ int last;
  const int nb = gridDim.x, tid = threadIdx.x;
  const int grp = blockIdx.x / gsz, ngrp = (nb + gsz - 1) / gsz;
  const int b0 = grp * gsz, cnt = min(gsz, nb - b0);
  auto arrive = [&](unsigned int* ctr, int total) {
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      last = (atomicAdd(ctr, 1u) == (unsigned)total - 1);
      if (last) *ctr = 0u;  // ready for the next launch
      __threadfence();
    }
    __syncthreads();
    return last != 0;
  };
  constexpr int B = NQ == 1 ? 12 : 6;
  auto sum = [&](const double* p, int count) {
#pragma unroll
    for (int q = 0; q < NQ; q++) s[q] = c[q] = 0.0;
    for (int b = 0; b < count; b += B) {
      double2 v[NQ][B];
#pragma unroll
      for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int u = 0; u < B; u++) {
          const int o = tid + q * FRAG_BS;
          v[q][u] = make_double2(0.0, 0.0);
          if (b + u < count && o < nout)
            v[q][u] = __ldcg(reinterpret_cast<const double2*>(p) + (int64_t)(b + u) * nout + o);
        }
#pragma unroll
      for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int u = 0; u < B; u++) dd_add(s[q], c[q], v[q][u].x, v[q][u].y);
    }
  };
  auto put = [&](int64_t slot) {
#pragma unroll
    for (int q = 0; q < NQ; q++)
      if (tid + q * FRAG_BS < nout)
        reinterpret_cast<double2*>(part)[slot * nout + tid + q * FRAG_BS] = make_double2(s[q], c[q]);
  };
  put(blockIdx.x);
  if (!arrive(counters + 1 + grp, cnt)) return false;
  sum(part + 2 * (int64_t)b0 * nout, cnt);
  put(nb + grp);
  if (!arrive(counters, ngrp)) return false;
  sum(part + 2 * (int64_t)nb * nout, ngrp);
  return true;
}

template <int MT, int TJ>
__global__ void __launch_bounds__(FRAG_BS, 2) k_mvTmv_prec(const __grid_constant__ MvTmvPrecArgs a)
{
  pdl_begin();
  pdl_wait();
  constexpr int U = MT <= 2 ? 8 : MT <= 4 ? 4 : 2;  // rows of loads in flight
  constexpr int NO = MT * TJ * 32;                  // outputs, padded
  constexpr int NQ = (NO + FRAG_BS - 1) / FRAG_BS;
  constexpr int WB = NO <= 256 ? 8 : 4;             // warps combined at a time
  __shared__ double2 red[WB * NO];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int li = lane & 7, lj = lane >> 3;
  double s[MT][TJ], c[MT][TJ];
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int e = 0; e < TJ; e++) s[i][e] = c[i][e] = 0.0;
  // columns past the blocks' ends read a column inside (outputs not stored)
  int ci[MT], cj[TJ];
#pragma unroll
  for (int i = 0; i < MT; i++) ci[i] = min(8 * i + li, a.m - 1);
#pragma unroll
  for (int e = 0; e < TJ; e++) cj[e] = min(lj * TJ + e, a.k - 1);
  const int64_t nch = (a.n + U - 1) / U;
  const int64_t GW = gridDim.x * (int64_t)FRAG_NW;
  for (int64_t cc = blockIdx.x * (int64_t)FRAG_NW + w; cc < nch; cc += GW) {
    const int64_t ch = nch - 1 - cc;  // descending, as k_tn_frag
    double x[U][MT], y[U][TJ];
#pragma unroll
    for (int u = 0; u < U; u++) {
      // rows past the end repeat the last one, times zero
      const int64_t row = min(ch * U + u, a.n - 1);
#pragma unroll
      for (int i = 0; i < MT; i++) frag_ld1(a.V + row * a.ldv + ci[i], x[u][i]);
#pragma unroll
      for (int e = 0; e < TJ; e++) frag_ld1(a.W + row * a.ldw + cj[e], y[u][e]);
    }
    if ((ch + 1) * U > a.n)
#pragma unroll
      for (int u = 0; u < U; u++)
        if (ch * U + u >= a.n) {
#pragma unroll
          for (int i = 0; i < MT; i++) x[u][i] = 0.0;
#pragma unroll
          for (int e = 0; e < TJ; e++) y[u][e] = 0.0;
        }
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int i = 0; i < MT; i++)
#pragma unroll
        for (int e = 0; e < TJ; e++) dd_dot_step(x[u][i], y[u][e], s[i][e], c[i][e]);
  }
  // the warps in order; output (8i + li, lj*TJ + e) of the block at o = row + m*col
  const int nout = a.m * a.k;
  double ts[NQ], tc[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) ts[q] = tc[q] = 0.0;
#pragma unroll
  for (int w0 = 0; w0 < FRAG_NW; w0 += WB) {
    __syncthreads();
    if (w >= w0 && w < w0 + WB)
#pragma unroll
      for (int i = 0; i < MT; i++)
#pragma unroll
        for (int e = 0; e < TJ; e++)
          if (8 * i + li < a.m && lj * TJ + e < a.k)
            red[(w - w0) * NO + 8 * i + li + (lj * TJ + e) * a.m] = make_double2(s[i][e], c[i][e]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const int o = tid + q * FRAG_BS;
      if (o < nout)
#pragma unroll
        for (int b = 0; b < WB; b++) dd_add(ts[q], tc[q], red[b * NO + o].x, red[b * NO + o].y);
    }
  }
  if (!prec_tree_sum<NQ>(a.part, nout, a.gsz, a.counters, ts, tc)) return;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const int o = tid + q * FRAG_BS;
    if (o >= nout) continue;
    // alpha*(s + c) + beta*C in double-double, rounded once
    double* cp = a.C + (o % a.m) * a.sr + (o / a.m) * a.sc;
    const double p = a.alpha * ts[q];
    const double ep = fma(a.alpha, ts[q], -p) + a.alpha * tc[q];
    double qv = 0.0, eq = 0.0;
    if (a.beta != 0.0) {
      qv = a.beta * *cp;
      eq = fma(a.beta, *cp, -qv);
    }
    double t, et;
    dd_two_sum(p, qv, t, et);
    const double r = t + (et + ep + eq);
    *cp = r;
    if (a.mbox) a.mbox[(o % a.m) * a.mr + (o / a.m) * a.mc] = r;
    if (o % a.m < a.mirror) {
      a.Cm[(o / a.m) * a.sr + (o % a.m) * a.sc] = r;
      if (a.mboxm) a.mboxm[(o / a.m) * a.mr + (o % a.m) * a.mc] = r;
    }
  }
}

// C = alpha*V'W + beta*C with compensated sums (pb_frag.cu)
void launch_mvTmv_prec(int64_t n, int m, int k, double alpha, const double* V, int64_t ldv, const double* W,
                       int64_t ldw, double beta, double* C, int64_t ldc, double* mbox);

}  // namespace pb
