// pb_frag.cuh -- tall-skinny block products whose tensor-core fragments are
// loaded straight from global memory, for any width, stride and alignment.
//
//   k_tn_frag : C = alpha V'W + beta C     (mvecT_times_mvec)
//   k_nn_frag : W = alpha V C + beta W, or W(:,0:k) = W(:,0:m) C in place
//                                          (mvec_times_sdMat[_inplace])
//
// A fragment of mma.m8n8k4 in FP64 is one value per lane (lane l, g = l/4,
// t = l%4: a = A[g][t], b = B[t][g], d = D[g][2t..2t+1]), so a warp can read
// it from row-major blocks without any staging: V'W takes the row index as
// the k dimension (a = V(row t, column g), 4 rows of 64 bytes per load), V*C
// the row index as the m dimension (a = V(row g, column t)).  No shared
// memory, no block barrier and no alignment rule in the loop; every warp
// streams its own rows with U (or RT) steps of loads in flight.  Blocks whose
// rows start on even multiples of the element size take VEC: one load brings
// two columns, the fragments' column order being permuted to match.
//
// The products are bound by HBM at the widths a solver orthogonalises with
// (m <= 40 basis columns against k <= 8 new ones): the FP64 tensor pipe does
// 64 FMAs a cycle and SM, of which the padding of k to 8 uses a part.
//
// FP32 blocks are converted on load and their products formed and summed in
// FP64, rounded once at the end.
//
// Measured, n = 2,097,152, us with the L2 flushed, against the shared-memory
// kernels these replace (V'W | V*C with beta = 1; HBM floor in brackets):
//   FP64 37 x 5, odd offset, ld 47    850 -> 141 [106] | 884 -> 190 [119]
//   FP64 20 x 4 of ld 44              128 -> 115 [61]  | 200 -> 153 [71]
//   FP64 16 x 16                      110 -> 108 [81]  | 215 -> 127 [121]
//   FP64 32 x 32                      (staged kernel)  | 450 -> 260 [242]
//   FP64 64 x 64                      (staged kernel)  | 1,751 -> 641 [484]
//   FP64 W'W, 8 / 16 / 32 columns      56 -> 39, 71 -> 64, 171 -> 119
//   FP32 10 x 4                       260 -> 51 [18]   | 145 -> 46 [23]
// and back to back with a warm L2, FP32 V*C of 32 x 32 373 -> 212 (beta = 0: 156
// -> 170), of 64 x 64 1,020 -> 618 (516 -> 580, bound by the FP64 pipe).
// The launch bound is part of that: with the two blocks per SM named, ptxas
// keeps a whole chunk of loads in flight; without it 4 x 4 took 94 us, not 45.
#pragma once
#include "pb_dmma.cuh"

namespace pb {

constexpr int FRAG_BS = 256;
constexpr int FRAG_NW = FRAG_BS / 32;

template <class T>
struct FragTnArgs {
  int64_t n;
  int m, k;                     // V has m columns, W k (k <= m unless both fit one tile)
  const T* V; int64_t ldv;
  const T* W; int64_t ldw;
  T alpha, beta;
  T* C; int64_t sr, sc;         // C(i, j) at C[i*sr + j*sc] for V column i, W column j
  T* mbox; int mr, mc;          // copy of the result in mapped host memory (or NULL), strides mr, mc
  double* part;                 // (blocks + groups) x m*k partial sums
  int gsz;                      // blocks per group of the first reduction level
  unsigned int* counters;       // 1 + groups, zero between launches
};

template <class T>
struct FragNnArgs {
  int64_t n;
  int m, k;
  const T* V; int64_t ldv;
  T* W; int64_t ldw;
  const T* C; int64_t ldc;
  T alpha, beta;                // beta == 0: W is not read
};

// one or two consecutive elements.  Volatile, so that the loads of a chunk
// are issued in front of its products: left to itself the compiler sinks
// every load to its use, and a chunk then waits for memory once per step.
__device__ __forceinline__ void frag_ld1(const double* p, double& a)
{
  asm volatile("ld.global.f64 %0, [%1];\n" : "=d"(a) : "l"(p));
}
__device__ __forceinline__ void frag_ld1(const float* p, float& a)
{
  asm volatile("ld.global.f32 %0, [%1];\n" : "=f"(a) : "l"(p));
}
__device__ __forceinline__ void frag_ld2(const double* p, double& a, double& b)
{
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];\n" : "=d"(a), "=d"(b) : "l"(p));
}
__device__ __forceinline__ void frag_ld2(const float* p, float& a, float& b)
{
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];\n" : "=f"(a), "=f"(b) : "l"(p));
}
__device__ __forceinline__ void frag_st2(double* p, double a, double b)
{
  *reinterpret_cast<double2*>(p) = make_double2(a, b);
}
__device__ __forceinline__ void frag_st2(float* p, float a, float b)
{
  *reinterpret_cast<float2*>(p) = make_float2(a, b);
}

// Two-level sum of the blocks' partial outputs in a fixed order, inside the
// kernel: the last block of a group of gsz to arrive adds the group's
// partials in block order, the last group's block adds the group sums in
// group order.  Both levels are about sqrt(blocks) long, so two short rounds
// of independent loads replace one long one (a single last block) or a
// second launch.  True in the block that holds the totals: thread o (in
// steps of the block size NTH) has output o in tot[o / NTH].
template <int NQ, int NTH = FRAG_BS>
__device__ __forceinline__ bool frag_tree_sum(double* part, int nout, int gsz, unsigned int* counters, double (&tot)[NQ])
{
  __shared__ int last;
  const int nb = gridDim.x, tid = threadIdx.x;
  const int grp = blockIdx.x / gsz, ngrp = (nb + gsz - 1) / gsz;
  const int b0 = grp * gsz, cnt = min(gsz, nb - b0);
  // one thread's fence after the barrier covers the block's writes
  auto arrive = [&](unsigned int* c, int total) {
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      last = (atomicAdd(c, 1u) == (unsigned)total - 1);
      if (last) *c = 0u;  // ready for the next launch
      __threadfence();
    }
    __syncthreads();
    return last != 0;
  };
  // all outputs of a thread together, B partials of each in flight (a level is
  // 17 to 25 long: two rounds of loads)
  constexpr int B = NQ == 1 ? 16 : NQ == 2 ? 12 : 4;
  auto sum = [&](const double* p, int count) {
#pragma unroll
    for (int q = 0; q < NQ; q++) tot[q] = 0.0;
    for (int b = 0; b < count; b += B) {
      double v[NQ][B];
#pragma unroll
      for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int u = 0; u < B; u++) {
          const int o = tid + q * NTH;
          v[q][u] = (b + u < count && o < nout) ? __ldcg(p + (int64_t)(b + u) * nout + o) : 0.0;
        }
#pragma unroll
      for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int u = 0; u < B; u++) tot[q] += v[q][u];
    }
  };
  if (nout <= NTH && nout * nb <= 20 * NTH) {
    // few outputs: one level, the blocks of an output split over G threads
    // whose sums meet in a fixed tree
    if (!arrive(counters, nb)) return false;
    __shared__ double red1[NTH];
    const int G = NTH / nout, q = tid / nout, o = tid - q * nout;
    double s = 0.0;
    if (q < G)
      for (int b = q; b < nb; b += 8 * G) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = b + u * G < nb ? __ldcg(part + (int64_t)(b + u * G) * nout + o) : 0.0;
#pragma unroll
        for (int u = 0; u < 8; u++) s += v[u];
      }
    red1[tid] = s;
    __syncthreads();
    int P = 1;
    while (2 * P <= G) P *= 2;
    if (q < G - P) red1[tid] += red1[tid + P * nout];
    for (int h = P / 2; h >= 1; h >>= 1) {
      __syncthreads();
      if (q < h) red1[tid] += red1[tid + h * nout];
    }
    tot[0] = red1[tid];  // nout <= NTH: outputs o < nout are in thread o
    return true;
  }
  if (!arrive(counters + 1 + grp, cnt)) return false;
  sum(part + (int64_t)b0 * nout, cnt);
#pragma unroll
  for (int q = 0; q < NQ; q++)
    if (tid + q * NTH < nout) part[(int64_t)(nb + grp) * nout + tid + q * NTH] = tot[q];
  if (!arrive(counters, ngrp)) return false;
  sum(part + (int64_t)nb * nout, ngrp);
  return true;
}

// column of V (or W) held by fragment i of lane group g
template <int MT, bool VEC>
__device__ __forceinline__ int frag_col(int i, int g)
{
  return (VEC && i < (MT & ~1)) ? (i / 2) * 16 + 2 * g + (i & 1) : i * 8 + g;
}

// the fragments of one row: MT tiles of 8 columns, columns >= ncol read as a
// column inside the block (they only reach outputs that are not stored)
template <class T, int MT, bool VEC>
__device__ __forceinline__ void frag_row(const T* row, int ncol, int g, T* v)
{
  if (VEC) {
#pragma unroll
    for (int p = 0; p < MT / 2; p++) {
      int c = 16 * p + 2 * g;
      if (2 * p + 2 == MT) c = min(c, ncol - 2);
      frag_ld2(row + c, v[2 * p], v[2 * p + 1]);
    }
    if (MT & 1) frag_ld1(row + min(8 * (MT - 1) + g, ncol - 1), v[MT - 1]);
  } else {
#pragma unroll
    for (int i = 0; i < MT; i++) {
      int c = 8 * i + g;
      if (i == MT - 1) c = min(c, ncol - 1);
      frag_ld1(row + c, v[i]);
    }
  }
}

// shared memory of frag_finish: WB warps' outputs
template <int MT, int KT>
constexpr int frag_wb()
{
  return MT * KT <= 8 ? 8 : MT * KT <= 16 ? 4 : 2;
}
template <int MT, int KT>
constexpr int frag_red()
{
  return frag_wb<MT, KT>() * MT * KT * 64;
}

// The end of a V'W kernel: acc holds the warp's tiles (SYM: those on and above
// the diagonal); warps, then blocks are summed in fixed order and the block
// with the totals writes C = alpha V'W + beta C.  red: frag_red<MT, KT>()
// doubles, free on entry after a barrier.
template <class T, int MT, int KT, bool SYM, bool VEC, int NTILE>
__device__ __forceinline__ void frag_finish(const FragTnArgs<T>& a, const double (&acc)[NTILE][2], double* red)
{
  constexpr int NOUT = MT * KT * 64, WB = frag_wb<MT, KT>();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  // the warps' sums in warp order, WB warps at a time through shared memory
  const int nout = a.m * a.k;
  constexpr int NQ = (NOUT + FRAG_BS - 1) / FRAG_BS;
  double tot[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) tot[q] = 0.0;
#pragma unroll
  for (int s = 0; s < FRAG_NW; s += WB) {
    if (s > 0) __syncthreads();
    if (w >= s && w < s + WB) {
      double* rw = red + (w - s) * NOUT;
      int q = 0;
#pragma unroll
      for (int j = 0; j < KT; j++)
#pragma unroll
        for (int i = 0; i < (SYM ? j + 1 : MT); i++, q++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int row = frag_col<MT, VEC>(i, g), col = frag_col<KT, VEC>(j, 2 * t + e);
            rw[row + col * (MT * 8)] = acc[q][e];
            // the mirror image of a tile above the diagonal
            if (SYM && i < j) rw[col + row * (MT * 8)] = acc[q][e];
          }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const int o = tid + q * FRAG_BS;
      if (o < nout)
#pragma unroll
        for (int b = 0; b < WB; b++) tot[q] += red[b * NOUT + (o % a.m) + (o / a.m) * (MT * 8)];
    }
  }
#pragma unroll
  for (int q = 0; q < NQ; q++)
    if (tid + q * FRAG_BS < nout) a.part[(int64_t)blockIdx.x * nout + tid + q * FRAG_BS] = tot[q];
  if (!frag_tree_sum<NQ>(a.part, nout, a.gsz, a.counters, tot)) return;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const int o = tid + q * FRAG_BS;
    if (o < nout) {
      T* dst = a.C + (o % a.m) * a.sr + (o / a.m) * a.sc;
      const double s = (double)a.alpha * tot[q];
      const T r = (T)(a.beta == T(0) ? s : s + (double)a.beta * (double)*dst);
      *dst = r;
      if (a.mbox) a.mbox[(o % a.m) * a.mr + (o / a.m) * a.mc] = r;
    }
  }
}

// C = alpha V'W + beta C.  Warps take chunks of 4U rows in grid-stride
// order.  SYM: W is V, the fragments of V serve both operands and only the
// tiles on and above the diagonal are formed.
template <class T, int MT, int KT, bool SYM, bool VEC, int U>
__global__ void __launch_bounds__(FRAG_BS, 2) k_tn_frag(const __grid_constant__ FragTnArgs<T> a)
{
  pdl_begin();
  pdl_wait();
  static_assert(!SYM || MT == KT, "a symmetric product is square");
  constexpr int NTILE = SYM ? MT * (MT + 1) / 2 : MT * KT;
  __shared__ double red[frag_red<MT, KT>()];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  double acc[NTILE][2];
#pragma unroll
  for (int i = 0; i < NTILE; i++) acc[i][0] = acc[i][1] = 0.0;

  auto step = [&](const T* v, const T* wv) {
    int q = 0;
#pragma unroll
    for (int j = 0; j < KT; j++)
#pragma unroll
      for (int i = 0; i < (SYM ? j + 1 : MT); i++, q++)
        dmma_884(acc[q][0], acc[q][1], (double)v[i], (double)(SYM ? v[j] : wv[j]));
  };
  const int64_t nch = a.n / (4 * U);
  const int64_t gw = blockIdx.x * (int64_t)FRAG_NW + w, GW = gridDim.x * (int64_t)FRAG_NW;
  for (int64_t c = gw; c < nch; c += GW) {
    // from the last rows to the first: what the kernel before this one (rows
    // in ascending order) touched last is still in the L2
    const int64_t r = (nch - 1 - c) * (4 * U) + t;
    const T* pv = a.V + r * a.ldv;
    const T* pw = a.W + r * a.ldw;
    T v[U][MT], wv[U][KT];
#pragma unroll
    for (int u = 0; u < U; u++) {
      frag_row<T, MT, VEC>(pv + 4 * u * a.ldv, a.m, g, v[u]);
      if (!SYM) frag_row<T, KT, VEC>(pw + 4 * u * a.ldw, a.k, g, wv[u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) step(v[u], wv[u]);
  }
  if (gw == nch % GW) {
    // the last rows: steps past the block's end multiply zeros
    for (int64_t r0 = nch * (4 * U); r0 < a.n; r0 += 4) {
      const int64_t r = r0 + t;
      T v[MT], wv[KT];
#pragma unroll
      for (int i = 0; i < MT; i++) v[i] = T(0);
#pragma unroll
      for (int j = 0; j < KT; j++) wv[j] = T(0);
      if (r < a.n) {
        frag_row<T, MT, VEC>(a.V + r * a.ldv, a.m, g, v);
        if (!SYM) frag_row<T, KT, VEC>(a.W + r * a.ldw, a.k, g, wv);
      }
      step(v, wv);
    }
  }
  frag_finish<T, MT, KT, SYM, VEC>(a, acc, red);
}

// chunk ch of 8*RT rows: the fragments of V, and for beta != 0 the old W in
// the layout of the result
template <class T, int MC, int KT, bool VEC, int RT>
__device__ __forceinline__ void frag_nn_load(const FragNnArgs<T>& a, int64_t ch, int g, int t, T (&v)[RT][2 * MC],
                                             T (&wo)[RT][KT][2])
{
#pragma unroll
  for (int r = 0; r < RT; r++) {
    // rows past the end read the last row and are not stored
    const int64_t row = min(ch * (8 * RT) + 8 * r + g, a.n - 1);
    const T* pv = a.V + row * a.ldv;
#pragma unroll
    for (int q = 0; q < MC; q++) {
      // columns past m must not meet the zero rows of C as infinities
      const bool whole = q < MC - 1;
      if (VEC) {
        v[r][2 * q] = v[r][2 * q + 1] = T(0);
        if (whole || 8 * q + 2 * t < a.m) frag_ld2(pv + 8 * q + 2 * t, v[r][2 * q], v[r][2 * q + 1]);
      } else {
        v[r][2 * q] = v[r][2 * q + 1] = T(0);
        if (whole || 8 * q + t < a.m) frag_ld1(pv + 8 * q + t, v[r][2 * q]);
        if (whole || 8 * q + 4 + t < a.m) frag_ld1(pv + 8 * q + 4 + t, v[r][2 * q + 1]);
      }
    }
    if (a.beta != T(0)) {
      const T* pw = a.W + row * a.ldw;
#pragma unroll
      for (int j = 0; j < KT; j++) {
        const int c = 8 * j + 2 * t;
        wo[r][j][0] = wo[r][j][1] = T(0);
        if (VEC) {
          if (c < a.k) frag_ld2(pw + c, wo[r][j][0], wo[r][j][1]);
        } else {
          if (c < a.k) frag_ld1(pw + c, wo[r][j][0]);
          if (c + 1 < a.k) frag_ld1(pw + c + 1, wo[r][j][1]);
        }
      }
    }
  }
}

// W = alpha V C + beta W (V == W: in place).  A warp owns 8*RT rows: all its
// fragments of V are in registers before the first store, so the update in
// place needs no copy.  C sits in shared memory in fragment order.  WV: rows
// of W are stored two columns at a time.
template <class T, int MC, int KT, bool VEC, int RT>
__global__ void __launch_bounds__(FRAG_BS, 2) k_nn_frag(const __grid_constant__ FragNnArgs<T> a)
{
  pdl_begin();
  pdl_wait();
  constexpr int KS = 2 * MC;  // steps of 4 columns of V
  __shared__ double sC[KS * KT * 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  // column of V of step s in lane t
  auto vcol = [](int s, int tt) { return VEC ? 8 * (s / 2) + 2 * tt + (s & 1) : 4 * s + tt; };
  for (int q = tid; q < KS * KT * 32; q += FRAG_BS) {
    const int l = q & 31, j = (q >> 5) % KT, s = (q >> 5) / KT;
    const int i = vcol(s, l & 3), c = j * 8 + (l >> 2);
    sC[q] = (i < a.m && c < a.k) ? (double)a.C[i + (int64_t)c * a.ldc] : 0.0;
  }
  __syncthreads();
  const int64_t nch = (a.n + 8 * RT - 1) / (8 * RT);
  const int64_t GW = gridDim.x * (int64_t)FRAG_NW;
  for (int64_t ch = blockIdx.x * (int64_t)FRAG_NW + w; ch < nch; ch += GW) {
    T v[RT][KS], wo[RT][KT][2];
    frag_nn_load<T, MC, KT, VEC, RT>(a, ch, g, t, v, wo);
    double acc[RT][KT][2];
#pragma unroll
    for (int r = 0; r < RT; r++)
#pragma unroll
      for (int j = 0; j < KT; j++) acc[r][j][0] = acc[r][j][1] = 0.0;
#pragma unroll
    for (int s = 0; s < KS; s++)
#pragma unroll
      for (int j = 0; j < KT; j++) {
        const double b = sC[(s * KT + j) * 32 + lane];
#pragma unroll
        for (int r = 0; r < RT; r++) dmma_884(acc[r][j][0], acc[r][j][1], (double)v[r][s], b);
      }
#pragma unroll
    for (int r = 0; r < RT; r++) {
      const int64_t row = ch * (8 * RT) + 8 * r + g;
      if (row >= a.n) continue;
      T* pw = a.W + row * a.ldw;
#pragma unroll
      for (int j = 0; j < KT; j++) {
        const int c = 8 * j + 2 * t;
        double o[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          o[e] = (double)a.alpha * acc[r][j][e];
          if (a.beta != T(0)) o[e] += (double)a.beta * (double)wo[r][j][e];
        }
        if (VEC) {
          if (c < a.k) frag_st2(pw + c, (T)o[0], (T)o[1]);
        } else {
          if (c < a.k) pw[c] = (T)o[0];
          if (c + 1 < a.k) pw[c + 1] = (T)o[1];
        }
      }
    }
  }
}

// W = alpha V C + beta W (or in place) and G = galpha W'W + gbeta G of the new
// W in one pass (go.alpha, go.beta, go.C; go.m == go.k == a.k): the rows that
// a warp has just formed go through its own shared-memory tile from the
// result's fragment layout to the operands', and the tiles of W'W on and
// above the diagonal are accumulated at once, so W is not read again.
// RT row tiles in flight: 3 and one block per SM up to 16 columns, beyond (the
// accumulators of W'W take the registers) 1 and two blocks (n = 2,097,152, us:
// RT 1 / 2 / 3 at 8 columns 94 / 69 / 66, at 16 129 / 111 / 109, at 24 188 /
// 210 / 213, at 32 266 / 278 / 270)
template <int KT>
constexpr int nn_gram_rt()
{
  return KT <= 2 ? 3 : 1;
}
template <class T, int MC, int KT, bool VEC>
__global__ void __launch_bounds__(FRAG_BS, (KT <= 2 ? 1 : 2))
k_nn_gram_frag(const __grid_constant__ FragNnArgs<T> a, const __grid_constant__ FragTnArgs<T> go)
{
  pdl_begin();
  pdl_wait();
  constexpr int RT = nn_gram_rt<KT>();
  constexpr int KS = 2 * MC, P = KT * 8 + 4;
  constexpr int NC = KS * KT * 32, NTL = FRAG_NW * 8 * P, NRED = frag_red<KT, KT>();
  constexpr int NTILE = KT * (KT + 1) / 2;
  // the tile's pairs are stored 16 bytes at a time
  __shared__ __align__(16) double sm[NC + NTL > NRED ? NC + NTL : NRED];
  static_assert(NC % 2 == 0 && P % 2 == 0, "pairs of a tile start on 16 bytes");
  double* sC = sm;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  double* tile = sm + NC + w * 8 * P;
  for (int q = tid; q < NC; q += FRAG_BS) {
    const int l = q & 31, j = (q >> 5) % KT, s = (q >> 5) / KT;
    const int i = VEC ? 8 * (s / 2) + 2 * (l & 3) + (s & 1) : 4 * s + (l & 3), c = j * 8 + (l >> 2);
    sC[q] = (i < a.m && c < a.k) ? (double)a.C[i + (int64_t)c * a.ldc] : 0.0;
  }
  __syncthreads();
  double gacc[NTILE][2];
#pragma unroll
  for (int i = 0; i < NTILE; i++) gacc[i][0] = gacc[i][1] = 0.0;
  const int64_t nch = (a.n + 8 * RT - 1) / (8 * RT);
  const int64_t GW = gridDim.x * (int64_t)FRAG_NW;
  for (int64_t ch = blockIdx.x * (int64_t)FRAG_NW + w; ch < nch; ch += GW) {
    T v[RT][KS], wo[RT][KT][2];
    frag_nn_load<T, MC, KT, VEC, RT>(a, ch, g, t, v, wo);
    double acc[RT][KT][2];
#pragma unroll
    for (int r = 0; r < RT; r++)
#pragma unroll
      for (int j = 0; j < KT; j++) acc[r][j][0] = acc[r][j][1] = 0.0;
#pragma unroll
    for (int s = 0; s < KS; s++)
#pragma unroll
      for (int j = 0; j < KT; j++) {
        const double b = sC[(s * KT + j) * 32 + lane];
#pragma unroll
        for (int r = 0; r < RT; r++) dmma_884(acc[r][j][0], acc[r][j][1], (double)v[r][s], b);
      }
#pragma unroll
    for (int r = 0; r < RT; r++) {
      const int64_t row = ch * (8 * RT) + 8 * r + g;
      T* pw = a.W + row * a.ldw;
#pragma unroll
      for (int j = 0; j < KT; j++) {
        const int c = 8 * j + 2 * t;
        T o[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          double x = (double)a.alpha * acc[r][j][e];
          if (a.beta != T(0)) x += (double)a.beta * (double)wo[r][j][e];
          o[e] = row < a.n ? (T)x : T(0);
        }
        if (row < a.n) {
          if (VEC) {
            if (c < a.k) frag_st2(pw + c, o[0], o[1]);
          } else {
            if (c < a.k) pw[c] = o[0];
            if (c + 1 < a.k) pw[c + 1] = o[1];
          }
        }
        frag_st2(tile + g * P + c, (double)o[0], (double)o[1]);
      }
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; h++) {
        double f[KT];
#pragma unroll
        for (int j = 0; j < KT; j++) f[j] = tile[(4 * h + t) * P + 8 * j + g];
        int q = 0;
#pragma unroll
        for (int j = 0; j < KT; j++)
#pragma unroll
          for (int i = 0; i <= j; i++, q++) dmma_884(gacc[q][0], gacc[q][1], f[i], f[j]);
      }
      __syncwarp();
    }
  }
  __syncthreads();
  frag_finish<T, KT, KT, true, false>(go, gacc, sm);
}

// C = alpha V'W + beta C / W = alpha V C + beta W with the kernels above;
// false when the shape is not theirs (pb_frag.cu holds the rule).  mbox: C
// also goes there, dense and column-major (mapped host memory), or NULL.
template <class T>
bool frag_mvTmv(int64_t n, int m, int k, T alpha, const T* V, int64_t ldv, const T* W, int64_t ldw, T beta, T* C,
                int64_t ldc, T* mbox);
template <class T>
bool frag_mvsd(const RowGemmArgs<T>& a);
// the same with G = galpha W'W + gbeta G (a.Gd, a.ldg) of the new W in one
// pass; mbox as above
template <class T>
bool frag_mvsd_gram(const RowGemmArgs<T>& a, T* mbox);

}  // namespace pb
