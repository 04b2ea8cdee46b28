// pb_spmmv_lz.cuh -- the SpMMV of a MINRES step with the step's first pass
// inside: W = (A - sigma I) V_j F_j together with Q'W and alpha = V_j'W.
//
// As separate kernels the dots read W and V_j again from HBM (268 MB of the
// 1.65 GB a step moved at n = 2,097,152, 8 systems FP64).  Here the new rows of
// a tile go through shared memory to the tensor pipe, where they meet the
// rows of Q loaded as fragments straight from global memory; V_j's own row is
// in registers already, for the shift.  The block that finishes last computes
// the Lanczos coefficients (kry_epilogue).
#pragma once
#include "pb_krylov.cuh"
#include "pb_spmmv_pf.cuh"

namespace pb {

constexpr int LZ_NT = FRAG_BS;
constexpr int LZ_MAXQ = 16;
// resident blocks handed to ptxas: 20 steps of 8 systems FP64 on 128^3 took
// 7,896 / 7,037 / 7,307 us with 2 / 3 / 4, 7,461 with the dots in a pass of their own
constexpr int LZ_MB = 3;

template <class T, int NV, int TPR>
struct EpiLanczos {
  static constexpr bool on = true, scale = true;
  static constexpr int RPB = LZ_NT / TPR, PY = NV + 1, VPT = NV / TPR;
  static constexpr int MQ = LZ_MAXQ / 8;
  static constexpr int STEPS = RPB / 4 / FRAG_NW;  // 4-row steps of a warp in a tile
  static constexpr int RED = (LZ_MAXQ + 2) * NV;   // a warp's sums
  static constexpr int BUF = RPB * PY > FRAG_NW * RED ? RPB * PY : FRAG_NW * RED;
  static_assert(RPB % (4 * FRAG_NW) == 0 && NV <= KRY_MAXC, "bad tile");
  static_assert(BUF >= KRY_MAXOUT + KRY_MAXC, "epilogue scratch of KE_LZ");
  const KryArgs<T>& a;
  T* ys;       // new rows of the tile
  int* rows;   // their row numbers, -1: none
  double* buf;
  double qa[MQ][2];
  T va[VPT];
  __device__ __forceinline__ EpiLanczos(const KryArgs<T>& args, double* b, int* r)
      : a(args), ys(reinterpret_cast<T*>(b)), rows(r), buf(b)
  {
#pragma unroll
    for (int i = 0; i < MQ; i++) qa[i][0] = qa[i][1] = 0.0;
#pragma unroll
    for (int i = 0; i < VPT; i++) va[i] = T(0);
  }
  __device__ __forceinline__ void clear(int lr)
  {
    const int s = threadIdx.x % TPR;
#pragma unroll
    for (int q = 0; q < VPT; q++) ys[lr * PY + s * VPT + q] = T(0);
    if (s == 0) rows[lr] = -1;
  }
  // VW columns from column c (vector v of the thread) of row i: y new, x of V_j
  template <int VW>
  __device__ __forceinline__ void put(int lr, int64_t i, int v, int c, const T* y, const T* x)
  {
#pragma unroll
    for (int w = 0; w < VW; w++) {
      ys[lr * PY + c + w] = y[w];
      va[v * VW + w] += x[w] * y[w];
    }
    if (c == 0) rows[lr] = (int)i;
  }
  __device__ __forceinline__ void tile()
  {
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    T qv[STEPS][MQ];
#pragma unroll
    for (int u = 0; u < STEPS; u++) {
      const int row = rows[4 * (w * STEPS + u) + t];
      const T* pq = a.Q + (int64_t)(row < 0 ? 0 : row) * a.ldq;
#pragma unroll
      for (int i = 0; i < MQ; i++) kry_ldp(pq + min(8 * i + g, a.nq - 1), row >= 0, qv[u][i]);
    }
#pragma unroll
    for (int u = 0; u < STEPS; u++) {
      const double b = (double)ys[(4 * (w * STEPS + u) + t) * PY + min(g, NV - 1)];
#pragma unroll
      for (int i = 0; i < MQ; i++) dmma_884(qa[i][0], qa[i][1], (double)qv[u][i], b);
    }
  }
  __device__ __forceinline__ void finish()
  {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    double vd[VPT];
#pragma unroll
    for (int q = 0; q < VPT; q++) {
      vd[q] = (double)va[q];
#pragma unroll
      for (int off = 16; off >= TPR; off >>= 1) vd[q] += __shfl_xor_sync(0xffffffffu, vd[q], off);
    }
    __syncthreads();  // the tile is no longer read
    double* red = buf + w * RED;
#pragma unroll
    for (int i = 0; i < MQ; i++)
#pragma unroll
      for (int e = 0; e < 2; e++)
        if (8 * i + g < a.nq && 2 * t + e < NV) red[(8 * i + g) * NV + 2 * t + e] = qa[i][e];
    if (lane < TPR) {
      // a thread's vectors are contiguous: VPT columns from lane * VPT
#pragma unroll
      for (int q = 0; q < VPT; q++) {
        red[a.nq * NV + lane * VPT + q] = vd[q];
        red[(a.nq + 1) * NV + lane * VPT + q] = 0.0;
      }
    }
    kry_totals<T, 1 << KE_LZ>(a, a.nq, 1, buf, RED, buf);
  }
};

template <class T, int NV, int TPR, int VB>
__global__ void __launch_bounds__(LZ_NT, LZ_MB) k_sell_spmmv_lz(const __grid_constant__ SellDev<T> A,
                                                            const __grid_constant__ SpmvArgs<T> p,
                                                            const __grid_constant__ KryArgs<T> a)
{
  typedef EpiLanczos<T, NV, TPR> Epi;
  static_assert((NV / TPR) * sizeof(T) == VB, "a thread's columns are one vector");
  __shared__ double buf[Epi::BUF];
  __shared__ int rows[Epi::RPB];
  Epi epi(a, buf, rows);
  sell_spmmv_pf<T, NV, TPR, LZ_NT, false, VB, false>(A, p, epi);
}

}  // namespace pb
