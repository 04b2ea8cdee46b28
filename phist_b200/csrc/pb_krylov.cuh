// pb_krylov.cuh -- the passes over the basis of the device GMRES and MINRES
// (pb_gmres.cuh): all that happens between two SpMMVs, in one kernel body.
//
// The k systems are the k columns of every block: basis block V_i is n x k,
// contiguous.  The new direction W is the storage of the next block and
// stays unnormalised: v_i = F_i V_i with the factors F_i (one per system) on
// the device; the SpMMV multiplies by F_j, dots and coefficients carry F_i,
// so no pass is spent on scaling.
//
//   k_kry<MQ, MJ, UPD, DOTS> over the blocks V_0..V_{nb-1} it is given:
//     UPD : W -= Q cq + sum_i V_i hv_i          (cq: nq x k, hv: nb x k)
//     DOTS: Q'W (only without UPD) and V_i'W of every system
//     always ||W||^2 (after the update)
//
// The last block to finish holds the sums and goes on with the small dense
// work of the step (kry_epilogue): Lanczos or Gram-Schmidt coefficients, the
// column of H, rotations, residual estimate, convergence test, F_{j+1}.  A
// MINRES step is SpMMV + 2 launches, a GMRES step SpMMV + 3.
//
// More than 8 systems are split evenly into groups, gridDim.y of them, each
// with its own sums and epilogue; they run side by side over the same rows, so
// that Q and the lines that two groups share come from HBM once.  15 steps, nq
// = 32, us, a launch per group of 8 | so: GMRES FP64 32 systems, 24^3 2,871 | 907;
// 16 systems, 64^3 6,549 | 4,063; 12 systems, 100^3 18,548 | 13,628.
//
// A warp takes 32 rows at a time.  Q (row-major, any stride) meets W on the
// FP64 tensor pipe with fragments straight from global memory as in
// pb_frag.cuh; Q cq goes through a warp's own shared-memory tile into the
// layout of the basis part, where lane = (row, system) so that every load of
// V_i or W is one contiguous segment.  Bound by HBM, or for bases that fit it
// by the L2.
//
// Sums: lanes, warps and blocks in fixed order, FP64 from the lane sums on.
#pragma once
#include "pb_frag.cuh"

namespace pb {

constexpr int KRY_MAXQ = 32;  // projection columns of one launch
constexpr int KRY_MAXJ = 24;  // basis blocks of one launch
constexpr int KRY_MAXC = 8;   // most systems of one group (blockIdx.y) of a launch
constexpr int KRY_MAXOUT = (KRY_MAXQ + KRY_MAXJ + 1) * KRY_MAXC;

struct GmTol {
  double v[32];
};
struct GmIndex {
  int v[32];
};

// what the block holding the sums does
enum KryKind {
  KE_NONE = 0,    // nothing (the update alone)
  KE_START,       // beta = ||W||, g = beta e_1, F_0, g0
  KE_LZ,          // Lanczos coefficients of step j
  KE_GS,          // first Gram-Schmidt coefficients (blocks i0..), ||W|| before
  KE_GS2,         // second coefficients; with last also the decision on a second pass
  KE_STEP,        // rotations, residual estimate, convergence
  KE_NORM         // finv = 1/||W||
};

// H(:, :, s) at H[(i*m + j)*k + s]; per-system arrays have stride k and are
// indexed by the system number (c0 + the group's column); reorth, gflag and
// flags have one entry a group
template <class T>
struct KryEpi {
  int kind, last;             // last: last launch of a row of chunks (KE_GS2)
  int k, m, j, i0;
  int lanczos, first;
  double *H, *cs, *sn, *g, *bnorm;
  double *h1, *h2;            // [i*k + s] coefficients of the two Gram-Schmidt passes
  double *nrm0, *nf;          // ||W||^2 before the first pass; after the step
  T *F;                       // [i*k + s]
  T *cq, *hv, *hv2;           // coefficients for the update passes
  T *finv;
  int *conv, *jcount, *reorth;
  double eps_abs, h2_lim;
  GmTol tol;
  // Q'V_i = gam[i*k + s] g0 (nq values g0[l*k + s]); used while *gflag != 0
  double *g0, *gam, *dq;
  int* gflag;                 // NULL: no projection in the passes
  volatile unsigned long long* flags;  // mapped host memory: converged systems of the group << 32 | steps done
};

template <class T>
struct KryArgs {
  int64_t n;
  int k, per;                 // systems, the row stride of W and V_i; systems of a group (the last may have fewer)
  int nq; const T* Q; int64_t ldq;
  const T* V; int64_t vstep; int nb;   // blocks at V + i*vstep
  const T* Win;               // NULL: W starts from zero
  T* W;
  const T* cq; const T* hv;
  const int* skip;            // a group with skip[group] == 0 has nothing to do
  double* part; int gsz; unsigned int* counters;   // of group 0; the others' follow
  int64_t part_step; int cnt_step;                 // at these distances
  KryEpi<T> e;
  // KE_START: W = R(:, idx) (- W on a restart, converged systems zero)
  const T* R; int64_t ldr; GmIndex idx; int restart;
};

// the block's group: first system, systems, and that rounded up to a power of two
struct KryGrp {
  int c0, kc, kp;
  __device__ __forceinline__ KryGrp(int k, int per) : c0(blockIdx.y * per), kc(min(KRY_MAXC, min(per, k - c0)))
  {
    kp = kc <= 1 ? 1 : kc <= 2 ? 2 : kc <= 4 ? 4 : 8;
  }
};

__device__ __forceinline__ void kry_ldp(const double* p, bool ok, double& v)
{
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\nmov.f64 %0, 0d0000000000000000;\n@p ld.global.f64 %0, [%1];\n}\n"
               : "=d"(v)
               : "l"(p), "r"((int)ok));
}
__device__ __forceinline__ void kry_ldp(const float* p, bool ok, float& v)
{
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\nmov.f32 %0, 0f00000000;\n@p ld.global.f32 %0, [%1];\n}\n"
               : "=f"(v)
               : "l"(p), "r"((int)ok));
}

// Column j of every system's H is complete up to the new norm hn: apply the
// earlier rotations, zero h(j+1, j) with a new one, test for convergence.
// nrm: ||W||^2 per column of the launch; sm: shared scratch, 3*64*8 doubles.
// A Lanczos column is zero above j-1, so only the rotations from j-2 on act.
template <class T>
__device__ __forceinline__ void kry_step(const KryEpi<T>& e, int c0, int kc, const double* nrm, double* sm)
{
  const int tid = threadIdx.x, j = e.j, k = e.k, m = e.m;
  const int lo = e.lanczos ? max(0, j - 2) : 0;
  double* sh = sm;
  double* sc = sm + 64 * KRY_MAXC;
  double* ss = sc + 64 * KRY_MAXC;
  // what the chain of a system needs beside the rotations, loaded with them
  double gj = 0.0, bn = 0.0;
  int done = 0;
  if (tid < kc) {
    gj = __ldcg(&e.g[j * k + c0 + tid]);
    bn = __ldcg(&e.bnorm[c0 + tid]);
    done = __ldcg(&e.conv[c0 + tid]);
  }
  __syncthreads();
  for (int q = tid; q < (j + 1 - lo) * kc; q += FRAG_BS) {
    const int i = lo + q / kc, c = q % kc, s = c0 + c;
    sh[i * kc + c] = __ldcg(&e.H[((int64_t)i * m + j) * k + s]);
    if (i < j) {
      sc[i * kc + c] = __ldcg(&e.cs[i * k + s]);
      ss[i * kc + c] = __ldcg(&e.sn[i * k + s]);
    }
  }
  __syncthreads();
  if (tid < kc) {
    const int c = tid, s = c0 + c;
    const double n2 = fmax(nrm[c], 0.0), hn = sqrt(n2);
    double a = sh[lo * kc + c];
    for (int i = lo; i < j; i++) {
      const double b = sh[(i + 1) * kc + c], rc = sc[i * kc + c], rs = ss[i * kc + c];
      sh[i * kc + c] = rc * a + rs * b;
      a = -rs * a + rc * b;
    }
    double co = 1.0, si = 0.0;
    const double r = hypot(a, hn);
    if (r > 0.0) {
      co = a / r;
      si = hn / r;
    }
    sh[j * kc + c] = r;
    e.cs[j * k + s] = co;
    e.sn[j * k + s] = si;
    const double gn = -si * gj;
    e.g[j * k + s] = co * gj;
    e.g[(j + 1) * k + s] = gn;
    if (!done) {
      e.jcount[s] = j + 1;
      const double res = fabs(gn);
      if (res < e.eps_abs || (bn > 0.0 && res / bn < e.tol.v[s])) e.conv[s] = done = 1;
    }
    e.nf[s] = n2;
    e.F[(j + 1) * k + s] = (hn > 0.0) ? (T)(1.0 / hn) : T(0);
  }
  const int nconv = __syncthreads_count(tid < kc && done);
  for (int q = tid; q < (j + 1 - lo) * kc; q += FRAG_BS) {
    const int i = lo + q / kc, c = q % kc;
    e.H[((int64_t)i * m + j) * k + c0 + c] = sh[i * kc + c];
  }
  // step and count in one store: the host reads them together
  if (tid == 0) e.flags[blockIdx.y] = ((unsigned long long)(unsigned)nconv << 32) | (unsigned)(j + 1);
}

// The dots of a pass see W before the projection: V_i'W, where the step wants
// V_i'(P W) = V_i'W - (Q'V_i)'c with c = Q'W.  Q'V_i is rounding where the
// right-hand side is orthogonal to Q, but nothing demands that.  All vectors
// but V_0 come from the range of P, so Q'V_i is a multiple gam_i of g0 =
// Q'V_0, with V_{j+1} = P W - sum_i V_i hv_i: gam_{j+1} = -sum_i gam_i hv_i.
// The start takes g0 with the norms and sets *gflag where an entry is above
// rounding; the first coefficients then are F_i (V_i'W - gam_i d), d = g0'c.

// Warp w < kc: d (0 unless flagged) and ||c||^2 of system w in all lanes, for
// the c that the update subtracts
template <class T>
__device__ __forceinline__ void kry_proj_sums(const KryArgs<T>& a, int nqo, const double* out, bool flagged, double& d,
                                              double& c2)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const KryGrp gr(a.k, a.per);
  const bool on = w < gr.kc && lane < nqo;
  const double c = on ? (double)(T)out[lane * gr.kc + w] : 0.0;
  c2 = c * c;
  d = (on && flagged) ? __ldcg(&a.e.g0[lane * a.e.k + gr.c0 + w]) * c : 0.0;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    c2 += __shfl_xor_sync(0xffffffffu, c2, off);
    d += __shfl_xor_sync(0xffffffffu, d, off);
  }
}

// The kinds that a kernel can be asked for, as bits.  The last block runs this
// code once, from a cold instruction cache: with the kinds of all kernels in
// every kernel a pass of 20 us took 0.7 us more.
constexpr int kry_kinds(bool upd, bool dots)
{
  return upd ? (dots ? 1 << KE_GS2 : 1 << KE_STEP | 1 << KE_NORM) : 1 << KE_START | 1 << KE_LZ | 1 << KE_GS | 1 << KE_GS2;
}

// out: the sums in shared memory, [Q'W | V'W | ||W||^2] as nqo + nb + 1 rows
// of kc; sm: further shared scratch; flagged: *gflag
template <class T, int KINDS>
__device__ __forceinline__ void kry_epilogue(const KryArgs<T>& a, int nqo, int nbo, const double* out, double* sm,
                                             bool flagged)
{
  const KryEpi<T>& e = a.e;
  const KryGrp gr(a.k, a.per);
  const int tid = threadIdx.x, c0 = gr.c0, kc = gr.kc, k = e.k, j = e.j, m = e.m;
  const double* nrm = out + (nqo + nbo) * kc;
  auto is = [&](int kind) { return ((KINDS >> kind) & 1) && e.kind == kind; };
  if (is(KE_START)) {
    if (e.gflag) {
      int big = 0;
      for (int q = tid; q < nqo * kc; q += FRAG_BS) {
        const double v = out[q];
        const double eps = sizeof(T) == 8 ? 2.3e-16 : 1.2e-7;
        e.g0[(q / kc) * k + c0 + q % kc] = v;
        big |= v * v > 256.0 * eps * eps * nrm[q % kc];
      }
      big = __syncthreads_or(big);
      if (tid == 0) e.gflag[blockIdx.y] = big;
      if (tid < kc) e.gam[c0 + tid] = 1.0;
    }
    if (tid < kc) {
      const int s = c0 + tid;
      const double beta = sqrt(fmax(nrm[tid], 0.0));
      if (e.first) {
        e.bnorm[s] = beta;
        e.conv[s] = (beta < e.eps_abs) ? 1 : 0;
      }
      e.jcount[s] = 0;
      for (int i = 1; i <= m; i++) e.g[i * k + s] = 0.0;
      e.g[s] = e.conv[s] ? 0.0 : beta;
      e.F[s] = (beta > 0.0 && !e.conv[s]) ? (T)(1.0 / beta) : T(0);
    }
  } else if (is(KE_LZ)) {
    for (int q = tid; q < nqo * kc; q += FRAG_BS) e.cq[(q / kc) * k + c0 + q % kc] = (T)out[q];
    if (flagged) {
      double d, c2;
      kry_proj_sums<T>(a, nqo, out, true, d, c2);
      if ((tid & 31) == 0 && (tid >> 5) < kc) sm[tid >> 5] = d;
      __syncthreads();
    }
    if (tid < kc) {
      // alpha = v_j'w, beta = the previous step's norm; the update
      // subtracts V_j (F_j alpha), then V_{j-1} (F_{j-1} beta)
      const int s = c0 + tid;
      const double gj = flagged ? e.gam[j * k + s] : 0.0;
      const double alpha = (double)e.F[j * k + s] * (out[nqo * kc + tid] - (flagged ? gj * sm[tid] : 0.0));
      const double beta = j > 0 ? sqrt(e.nf[s]) : 0.0;
      for (int i = 0; i + 1 < j; i++) e.H[((int64_t)i * m + j) * k + s] = 0.0;
      if (j > 0) e.H[((int64_t)(j - 1) * m + j) * k + s] = beta;
      e.H[((int64_t)j * m + j) * k + s] = alpha;
      e.hv[s] = (T)((double)e.F[j * k + s] * alpha);
      e.hv[k + s] = j > 0 ? (T)((double)e.F[(j - 1) * k + s] * beta) : T(0);
      if (flagged)
        e.gam[(j + 1) * k + s] = -(gj * (double)e.hv[s] + (j > 0 ? e.gam[(j - 1) * k + s] * (double)e.hv[k + s] : 0.0));
    }
  } else if (is(KE_GS)) {
    for (int q = tid; q < nqo * kc; q += FRAG_BS) e.cq[(q / kc) * k + c0 + q % kc] = (T)out[q];
    if (e.i0 == 0) {
      // d, and ||P W||^2 = ||W||^2 - ||c||^2; where that is all cancellation
      // the larger ||W||^2, with which the second subtraction is made
      double d, c2;
      kry_proj_sums<T>(a, nqo, out, flagged, d, c2);
      const int w = tid >> 5;
      if ((tid & 31) == 0 && w < kc) {
        const double pw = nrm[w] - c2;
        e.nrm0[c0 + w] = pw > 1e-3 * nrm[w] ? pw : nrm[w];
        sm[w] = d;
        if (flagged) e.dq[c0 + w] = d;
      }
    } else if (flagged && tid < kc) {
      sm[tid] = __ldcg(&e.dq[c0 + tid]);
    }
    if (flagged) __syncthreads();
    for (int q = tid; q < nbo * kc; q += FRAG_BS) {
      const int p = (e.i0 + q / kc) * k + c0 + q % kc;
      const double h = (double)e.F[p] * (out[nqo * kc + q] - (flagged ? __ldcg(&e.gam[p]) * sm[q % kc] : 0.0));
      e.h1[p] = h;
      e.hv[p] = (T)((double)e.F[p] * h);
    }
  } else if (is(KE_GS2)) {
    // A second subtraction where some norm fell below 1/sqrt(2) of its value
    // before the pass ("twice is enough"), or where the first one has left
    // more than rounding along the basis: parts of V_i in the span of Q grow
    // from rounding as the steps go on, and Q may be orthonormal to less.
    int need = 0;
    for (int q = tid; q < nbo * kc; q += FRAG_BS) {
      const int p = (e.i0 + q / kc) * k + c0 + q % kc;
      const double h = (double)e.F[p] * out[nqo * kc + q];
      e.h2[p] = h;
      e.hv2[p] = (T)((double)e.F[p] * h);
      need |= h * h > e.h2_lim * nrm[q % kc];
    }
    if (!e.last) return;
    for (int q = tid; q < e.i0 * kc; q += FRAG_BS) {
      const double h = __ldcg(&e.h2[(q / kc) * k + c0 + q % kc]);
      need |= h * h > e.h2_lim * nrm[q % kc];
    }
    if (tid < kc) need |= nrm[tid] < 0.5 * e.nrm0[c0 + tid];
    __threadfence_block();
    const int any = __syncthreads_or(need);
    if (flagged && tid < kc) {
      const int s = c0 + tid;
      double gn = 0.0;
      for (int i = 0; i <= j; i++)
        gn -= __ldcg(&e.gam[i * k + s]) *
              ((double)__ldcg(&e.hv[i * k + s]) + (any ? (double)__ldcg(&e.hv2[i * k + s]) : 0.0));
      e.gam[(j + 1) * k + s] = gn;
    }
    for (int q = tid; q < (j + 1) * kc; q += FRAG_BS) {
      const int i = q / kc, s = c0 + q % kc;
      e.H[((int64_t)i * m + j) * k + s] = __ldcg(&e.h1[i * k + s]) + (any ? __ldcg(&e.h2[i * k + s]) : 0.0);
    }
    if (tid == 0) e.reorth[blockIdx.y] = any;
    __threadfence();
    if (!any) kry_step<T>(e, c0, kc, nrm, sm);
  } else if (is(KE_STEP)) {
    kry_step<T>(e, c0, kc, nrm, sm);
  } else if (is(KE_NORM)) {
    if (tid < kc) {
      const double nr = sqrt(fmax(nrm[tid], 0.0));
      e.finv[c0 + tid] = nr > 0.0 ? (T)(1.0 / nr) : T(0);
    }
  }
}

constexpr int KRY_RED = FRAG_NW * KRY_MAXOUT;
constexpr int KRY_TILE = 32 * 9;                                // a warp's Q cq tile
constexpr int KRY_SC = FRAG_NW * KRY_TILE;                      // coefficients of Q, fragment order
constexpr int KRY_SH = KRY_SC + 2 * (KRY_MAXQ / 8) * 32;        // coefficients of V
static_assert(KRY_SH + KRY_MAXJ * KRY_MAXC <= KRY_RED, "tiles fit the reduction buffer");
static_assert(KRY_MAXOUT + 3 * 64 * KRY_MAXC <= KRY_RED, "epilogue scratch fits the reduction buffer");

// red: the warps' sums, stride apart; from there the
// block's, the blocks' and, in the block that holds the totals, the epilogue
// (sm: shared scratch for it, may be red)
template <class T, int KINDS>
__device__ __forceinline__ void kry_totals(const KryArgs<T>& a, int nqo, int nbo, const double* red, int stride,
                                           double* sm)
{
  const int tid = threadIdx.x, nout = (nqo + nbo + 1) * KryGrp(a.k, a.per).kc;
  // loaded ahead of the sums, whose latency covers it
  constexpr bool uses = (KINDS & (1 << KE_LZ | 1 << KE_GS | 1 << KE_GS2)) != 0;
  const int flag = uses && a.e.gflag && a.e.kind != KE_START ? __ldcg(a.e.gflag + blockIdx.y) : 0;
  double* const part = a.part + blockIdx.y * a.part_step;
  unsigned int* const counters = a.counters + blockIdx.y * a.cnt_step;
  __syncthreads();
  double tot[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int o = tid + q * FRAG_BS;
    tot[q] = 0.0;
    if (o < nout) {
#pragma unroll
      for (int b = 0; b < FRAG_NW; b++) tot[q] += red[b * stride + o];
      part[(int64_t)blockIdx.x * nout + o] = tot[q];
    }
  }
  if (nout <= FRAG_BS) {
    double one[1] = {tot[0]};
    if (!frag_tree_sum<1>(part, nout, a.gsz, counters, one)) return;
    tot[0] = one[0];
  } else if (!frag_tree_sum<2>(part, nout, a.gsz, counters, tot)) {
    return;
  }
#pragma unroll
  for (int q = 0; q < 2; q++)
    if (tid + q * FRAG_BS < nout) sm[tid + q * FRAG_BS] = tot[q];
  __syncthreads();
  kry_epilogue<T, KINDS>(a, nqo, nbo, sm, sm + KRY_MAXOUT, flag != 0);
}

// after the row loop: the lanes' sums to the warps'
template <class T, int MQ, int MJ, int KINDS>
__device__ __forceinline__ void kry_finish(const KryArgs<T>& a, int nqo, int nbo, double (&qa)[MQ > 0 ? MQ : 1][2],
                                           T (&va)[MJ], T na, double* sm)
{
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
  if (a.e.kind == KE_NONE) return;  // the update alone
  const KryGrp gr(a.k, a.per);
  const int kc = gr.kc, kp = gr.kp, s = lane & (kp - 1);
  double nd = (double)na, vd[MJ];
#pragma unroll
  for (int i = 0; i < MJ; i++) vd[i] = i < nbo ? (double)va[i] : 0.0;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    if (off < kp) break;
#pragma unroll
    for (int i = 0; i < MJ; i++)
      if (i < nbo) vd[i] += __shfl_xor_sync(0xffffffffu, vd[i], off);
    nd += __shfl_xor_sync(0xffffffffu, nd, off);
  }
  __syncthreads();  // tiles and coefficients no longer read
  double* red = sm + w * KRY_MAXOUT;
  if (MQ > 0 && nqo > 0) {
#pragma unroll
    for (int i = 0; i < MQ; i++)
#pragma unroll
      for (int e = 0; e < 2; e++)
        if (i * 8 + g < nqo && 2 * t + e < kc) red[(i * 8 + g) * kc + 2 * t + e] = qa[i][e];
  }
  if (lane < kp && s < kc) {
#pragma unroll
    for (int i = 0; i < MJ; i++)
      if (i < nbo) red[(nqo + i) * kc + s] = vd[i];
    red[(nqo + nbo) * kc + s] = nd;
  }
  kry_totals<T, KINDS>(a, nqo, nbo, sm, KRY_MAXOUT, sm);
}

template <class T, int MQ, int MJ, bool UPD, bool DOTS>
__global__ void __launch_bounds__(FRAG_BS, 2) k_kry(const __grid_constant__ KryArgs<T> a)
{
  pdl_begin();
  pdl_wait();
  if (a.skip && a.skip[blockIdx.y] == 0) return;
  // packed steps, 4-row steps of Q'W and row tiles of Q cq with their loads in flight
  constexpr int UB = MJ <= 2 ? 4 : sizeof(T) == 4 ? (MJ <= 8 ? 4 : 2) : (MJ <= 8 ? 2 : 1);
  constexpr int QU = sizeof(T) == 4 ? 8 : 4;
  constexpr int MQ1 = MQ > 0 ? MQ : 1;
  constexpr int RTB = MQ <= 2 ? 4 : 2;
  __shared__ double sm[KRY_RED];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
  const KryGrp gr(a.k, a.per);
  const int c0 = gr.c0, kc = gr.kc, kp = gr.kp, k = a.k, nb = a.nb, nq = a.nq;
  const int s = lane & (kp - 1), rr = lane / kp, rs = 32 / kp;
  const bool mine = s < kc;
  double* sC = sm + KRY_SC;
  T* sH = reinterpret_cast<T*>(sm + KRY_SH);
  double* tile = sm + w * KRY_TILE;
  if (UPD) {
    for (int q = tid; q < 2 * MQ * 32; q += FRAG_BS) {
      const int l = q & 31, i = 4 * (q >> 5) + (l & 3), c = l >> 2;
      sC[q] = (i < nq && c < kc) ? (double)a.cq[i * k + c0 + c] : 0.0;
    }
    for (int q = tid; q < MJ * KRY_MAXC; q += FRAG_BS) {
      const int i = q / KRY_MAXC, c = q % KRY_MAXC;
      sH[q] = (i < nb && c < kc) ? a.hv[i * k + c0 + c] : T(0);
    }
    __syncthreads();
  }
  double qa[MQ1][2];
  T va[MJ], na = T(0);
#pragma unroll
  for (int i = 0; i < MQ1; i++) qa[i][0] = qa[i][1] = 0.0;
#pragma unroll
  for (int i = 0; i < MJ; i++) va[i] = T(0);
  const int64_t nch = (a.n + 31) / 32, GW = gridDim.x * (int64_t)FRAG_NW;
  for (int64_t ch = blockIdx.x * (int64_t)FRAG_NW + w; ch < nch; ch += GW) {
    // dots go from the last rows to the first, updates the other way: each
    // pass begins with the rows that the one before it left in the L2
    const int64_t r0 = (UPD ? ch : nch - 1 - ch) * 32;
    if (MQ > 0 && !UPD && DOTS) {
      // Q'W: 4-row steps
#pragma unroll
      for (int h = 0; h < 8; h += QU) {
        T qv[QU][MQ1], wv[QU];
#pragma unroll
        for (int u = 0; u < QU; u++) {
          const int64_t row = r0 + 4 * (h + u) + t;
          const bool ok = row < a.n;
          const T* pq = a.Q + (ok ? row : 0) * a.ldq;
#pragma unroll
          for (int i = 0; i < MQ; i++) kry_ldp(pq + min(8 * i + g, nq - 1), ok, qv[u][i]);
          kry_ldp(a.W + (ok ? row : 0) * k + c0 + min(g, kc - 1), ok, wv[u]);
        }
#pragma unroll
        for (int u = 0; u < QU; u++)
#pragma unroll
          for (int i = 0; i < MQ; i++) dmma_884(qa[i][0], qa[i][1], (double)qv[u][i], (double)wv[u]);
      }
    }
    if (MQ > 0 && UPD) {
      // Q cq of the chunk's rows, 8 rows per tensor tile, into the warp's tile
#pragma unroll
      for (int h = 0; h < 4; h += RTB) {
        T qv[RTB][2 * MQ1];
#pragma unroll
        for (int u = 0; u < RTB; u++) {
          const int64_t row = r0 + 8 * (h + u) + g;
          const T* pq = a.Q + (row < a.n ? row : 0) * a.ldq;
#pragma unroll
          for (int i = 0; i < 2 * MQ; i++) kry_ldp(pq + min(4 * i + t, nq - 1), row < a.n && 4 * i + t < nq, qv[u][i]);
        }
#pragma unroll
        for (int u = 0; u < RTB; u++) {
          double d0 = 0.0, d1 = 0.0;
#pragma unroll
          for (int i = 0; i < 2 * MQ; i++) dmma_884(d0, d1, (double)qv[u][i], sC[i * 32 + lane]);
          tile[(8 * (h + u) + g) * 9 + 2 * t] = d0;
          tile[(8 * (h + u) + g) * 9 + 2 * t + 1] = d1;
        }
      }
      __syncwarp();
    }
    // lane = (row, system)
    for (int u0 = 0; u0 < kp; u0 += UB) {
      T v[UB][MJ], wv[UB];
#pragma unroll
      for (int u = 0; u < UB; u++) {
        const int64_t row = r0 + (int64_t)(u0 + u) * rs + rr;
        const bool ok = mine && u0 + u < kp && row < a.n;
        const int64_t at = ok ? row * k + c0 + s : 0;
        kry_ldp(a.Win + at, ok && a.Win, wv[u]);
#pragma unroll
        for (int i = 0; i < MJ; i++) kry_ldp(a.V + i * a.vstep + at, ok && i < nb, v[u][i]);
      }
#pragma unroll
      for (int u = 0; u < UB; u++) {
        const int lr = (u0 + u) * rs + rr;
        const int64_t row = r0 + lr;
        const bool ok = mine && u0 + u < kp && row < a.n;
        T x = wv[u];
        if (UPD) {
          if (MQ > 0 && ok) x -= (T)tile[lr * 9 + s];
#pragma unroll
          for (int i = 0; i < MJ; i++) x -= v[u][i] * sH[i * KRY_MAXC + s];
          if (ok) a.W[row * k + c0 + s] = x;
          else x = T(0);
        }
        if (DOTS) {
#pragma unroll
          for (int i = 0; i < MJ; i++) va[i] += v[u][i] * x;
        }
        na += x * x;
      }
    }
    if (MQ > 0 && UPD) __syncwarp();
  }
  kry_finish<T, MQ, MJ, kry_kinds(UPD, DOTS)>(a, (DOTS && !UPD && MQ > 0) ? nq : 0, DOTS ? nb : 0, qa, va, na, sm);
}

// W = R(:, idx) at the start, W = R(:, idx) - W (0 for converged systems) on
// a restart, and the norms
template <class T>
__global__ void __launch_bounds__(FRAG_BS) k_kry_start(const __grid_constant__ KryArgs<T> a)
{
  pdl_begin();
  pdl_wait();
  __shared__ double sm[KRY_RED];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const KryGrp gr(a.k, a.per);
  const int c0 = gr.c0, kc = gr.kc, kp = gr.kp, k = a.k;
  const int s = lane & (kp - 1), rs = 32 / kp;
  T na = T(0);
  if (s < kc) {
    const int col = a.idx.v[c0 + s];
    const bool zero = a.restart && a.e.conv[c0 + s];
    const int64_t step = gridDim.x * (int64_t)FRAG_NW * rs;
#pragma unroll 4
    for (int64_t row = (blockIdx.x * (int64_t)FRAG_NW + w) * rs + lane / kp; row < a.n; row += step) {
      T x = a.R[row * a.ldr + col];
      if (a.restart) x = zero ? T(0) : x - a.W[row * k + c0 + s];
      a.W[row * k + c0 + s] = x;
      na += x * x;
    }
  }
  double qa[1][2];
  T va[1] = {T(0)};
  kry_finish<T, 0, 1, 1 << KE_START>(a, 0, 0, qa, va, na, sm);
}

}  // namespace pb
