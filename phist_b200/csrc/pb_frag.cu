// pb_frag.cu -- launches of the fragment kernels (pb_frag.cuh).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "pb_frag.cuh"
#include "pb_prec.cuh"

namespace pb {
namespace {

// resident blocks per SM of a kernel, taken once per instantiation
template <class K>
int frag_occ(K kern, std::atomic<int>& occ)
{
  int o = occ.load();
  if (o == 0) {
    PB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, FRAG_BS, 0));
    o = std::max(1, o);
    occ.store(o);
  }
  return o;
}

// row pairs of columns can be read with one load: two elements are aligned
template <class T>
bool pair_ok(const T* p, int64_t ld, int ncol)
{
  return ((uintptr_t)p) % (2 * sizeof(T)) == 0 && ld % 2 == 0 && ncol % 2 == 0;
}

// every row starts on a 16-byte boundary and is whole 16-byte pieces: the
// staged kernels (pb_dmma.cuh, pb_tile.cuh) take the block
template <class T>
bool rows16(const T* p, int64_t ld, int ncol)
{
  constexpr int vw = 16 / (int)sizeof(T);
  return ((uintptr_t)p) % 16 == 0 && ld % vw == 0 && ncol % vw == 0;
}

// every row starts on a 32-byte boundary
template <class T>
bool rows32(const T* p, int64_t ld)
{
  return ((uintptr_t)p) % 32 == 0 && ld * sizeof(T) % 32 == 0;
}

template <class T, int MT, int KT, bool SYM, bool VEC>
void tn_launch(FragTnArgs<T>& a)
{
  // rows in flight per warp: about 20 loads
  constexpr int NL = SYM ? MT : MT + KT;
  constexpr int U = 20 / NL > 8 ? 8 : 20 / NL;
  auto kern = k_tn_frag<T, MT, KT, SYM, VEC, U>;
  static std::atomic<int> occ{0};
  const int64_t want = ceil_div(a.n > 0 ? a.n : 1, 4 * U * FRAG_NW);
  const int grid = (int)std::min<int64_t>(want, (int64_t)rt().num_sms() * std::min(2, frag_occ(kern, occ)));
  // groups of about sqrt(grid) blocks; one counter each and one for the groups
  a.gsz = std::max((int)std::ceil(std::sqrt((double)grid)), (int)ceil_div(grid, 62));
  const int ngrp = (int)ceil_div(grid, a.gsz);
  a.part = (double*)rt().scratch(sizeof(double) * (size_t)(grid + ngrp) * a.m * a.k);
  a.counters = rt().counters();
  launch_pdl(kern, grid, FRAG_BS, 0, a);
  PB_LAUNCH_CHECK();
}

template <class T, int KT, bool VEC>
bool tn_mt(FragTnArgs<T>& a)
{
  switch ((a.m + 7) / 8) {
    case 1: tn_launch<T, 1, KT, false, VEC>(a); return true;
    case 2: tn_launch<T, 2, KT, false, VEC>(a); return true;
    case 3: tn_launch<T, 3, KT, false, VEC>(a); return true;
    case 4: tn_launch<T, 4, KT, false, VEC>(a); return true;
    case 5: tn_launch<T, 5, KT, false, VEC>(a); return true;
    case 6: tn_launch<T, 6, KT, false, VEC>(a); return true;
    case 7: tn_launch<T, 7, KT, false, VEC>(a); return true;
    case 8: tn_launch<T, 8, KT, false, VEC>(a); return true;
  }
  return false;
}

template <class T, bool VEC>
bool tn_sym(FragTnArgs<T>& a)
{
  switch ((a.m + 7) / 8) {
    case 1: tn_launch<T, 1, 1, true, VEC>(a); return true;
    case 2: tn_launch<T, 2, 2, true, VEC>(a); return true;
    case 3: tn_launch<T, 3, 3, true, VEC>(a); return true;
    case 4: tn_launch<T, 4, 4, true, VEC>(a); return true;
  }
  return false;
}

template <class T, int MC, int KT, bool VEC>
void nn_launch(const FragNnArgs<T>& a)
{
  constexpr int RT = MC <= 5 ? 2 : 1;
  auto kern = k_nn_frag<T, MC, KT, VEC, RT>;
  static std::atomic<int> occ{0};
  const int64_t want = ceil_div(a.n, 8 * RT * FRAG_NW);
  const int grid = (int)std::min<int64_t>(want, (int64_t)rt().num_sms() * frag_occ(kern, occ));
  launch_pdl(kern, grid, FRAG_BS, 0, a);
  PB_LAUNCH_CHECK();
}

template <class T, int KT, bool VEC>
bool nn_mc(const FragNnArgs<T>& a)
{
  switch ((a.m + 7) / 8) {
    case 1: nn_launch<T, 1, KT, VEC>(a); return true;
    case 2: nn_launch<T, 2, KT, VEC>(a); return true;
    case 3: nn_launch<T, 3, KT, VEC>(a); return true;
    case 4: nn_launch<T, 4, KT, VEC>(a); return true;
    case 5: nn_launch<T, 5, KT, VEC>(a); return true;
    case 6: nn_launch<T, 6, KT, VEC>(a); return true;
    case 7: nn_launch<T, 7, KT, VEC>(a); return true;
    case 8: nn_launch<T, 8, KT, VEC>(a); return true;
  }
  return false;
}

template <class T, int MC, int KT, bool VEC>
void nn_gram_launch(const FragNnArgs<T>& a, FragTnArgs<T>& go)
{
  constexpr int RT = nn_gram_rt<KT>();
  auto kern = k_nn_gram_frag<T, MC, KT, VEC>;
  static std::atomic<int> occ{0};
  const int64_t want = ceil_div(a.n, 8 * RT * FRAG_NW);
  const int grid = (int)std::min<int64_t>(want, (int64_t)rt().num_sms() * std::min(3, frag_occ(kern, occ)));
  go.gsz = std::max((int)std::ceil(std::sqrt((double)grid)), (int)ceil_div(grid, 62));
  go.part = (double*)rt().scratch(sizeof(double) * (size_t)(grid + ceil_div(grid, go.gsz)) * a.k * a.k);
  go.counters = rt().counters();
  launch_pdl(kern, grid, FRAG_BS, 0, a, go);
  PB_LAUNCH_CHECK();
}

template <class T, int KT, bool VEC>
void nn_gram_mc(const FragNnArgs<T>& a, FragTnArgs<T>& go)
{
  switch ((a.m + 7) / 8) {
    case 1: nn_gram_launch<T, 1, KT, VEC>(a, go); return;
    case 2: nn_gram_launch<T, 2, KT, VEC>(a, go); return;
    case 3: nn_gram_launch<T, 3, KT, VEC>(a, go); return;
    default: nn_gram_launch<T, 4, KT, VEC>(a, go); return;
  }
}

template <int MT, int TJ>
void prec_launch(MvTmvPrecArgs& a)
{
  constexpr int U = MT <= 2 ? 8 : MT <= 4 ? 4 : 2;
  const int64_t want = ceil_div(a.n > 0 ? a.n : 1, U * FRAG_NW);
  const int grid = (int)std::min<int64_t>(want, 2 * (int64_t)rt().num_sms());
  a.gsz = std::max((int)std::ceil(std::sqrt((double)grid)), (int)ceil_div(grid, 62));
  a.part = (double*)rt().scratch(2 * sizeof(double) * (size_t)(grid + ceil_div(grid, a.gsz)) * a.m * a.k);
  a.counters = rt().counters();
  launch_pdl(k_mvTmv_prec<MT, TJ>, grid, FRAG_BS, 0, a);
  PB_LAUNCH_CHECK();
}

template <int TJ>
void prec_mt(MvTmvPrecArgs& a)
{
  switch ((a.m + 7) / 8) {
    case 1: prec_launch<1, TJ>(a); return;
    case 2: prec_launch<2, TJ>(a); return;
    case 3: prec_launch<3, TJ>(a); return;
    case 4: prec_launch<4, TJ>(a); return;
    case 5: prec_launch<5, TJ>(a); return;
    case 6: prec_launch<6, TJ>(a); return;
    case 7: prec_launch<7, TJ>(a); return;
    default: prec_launch<8, TJ>(a); return;
  }
}

}  // namespace

// Up to 64 columns of the wider block against 8 of the other per launch.  W'W
// forms, for the columns j0.. of the result, only the rows up to j0 + 8 and
// mirrors them.
void launch_mvTmv_prec(int64_t n, int m, int k, double alpha, const double* V, int64_t ldv, const double* W,
                       int64_t ldw, double beta, double* C, int64_t ldc, double* mbox)
{
  const bool swap = k > m;
  const bool sym = V == W && ldv == ldw && m == k && m <= 64 && beta == 0.0;
  for (int i0 = 0; i0 < std::max(m, k); i0 += 64)
    for (int j0 = 0; j0 < std::min(m, k); j0 += 8) {
      MvTmvPrecArgs a;
      a.n = n;
      a.m = sym ? std::min(m, j0 + 8) : std::min(64, std::max(m, k) - i0);
      a.mirror = sym ? j0 : 0;
      a.Cm = C + j0;
      a.mr = swap ? m : 1; a.mc = swap ? 1 : m;
      a.mbox = mbox ? mbox + i0 * a.mr + j0 * a.mc : nullptr;
      a.mboxm = mbox ? mbox + j0 : nullptr;
      a.k = std::min(8, std::min(m, k) - j0);
      a.V = (swap ? W : V) + i0; a.ldv = swap ? ldw : ldv;
      a.W = (swap ? V : W) + j0; a.ldw = swap ? ldv : ldw;
      a.alpha = alpha; a.beta = beta;
      a.sr = swap ? ldc : 1; a.sc = swap ? 1 : ldc;
      a.C = C + i0 * a.sr + j0 * a.sc;
      if (a.k <= 4) prec_mt<1>(a);
      else prec_mt<2>(a);
    }
}

// Which products go here (us at n = 2,097,152, fragment | other kernel):
//   * thin ones (at most 4 columns against 4, FP32 8): up to a number of rows
//     the shorter cross-block sum decides, beyond it the row per thread of the
//     register kernels costs less.  FP64 against one column from 2^19 rows
//     (whole calls, back to back: 1 x 1 at 524,288 rows 17.9 | 18.0, at 1,048,576
//     20.6 | 19.0), else the fragments are as fast or faster (3 x 3 40.6 | 42.6,
//     W'W of 4 25.6 | 25.5) but for 4 x 4 in whole 32-byte rows (39.7 | 38.3).
//     FP32 from 2^20 (4 x 4 at 1,048,576 21.7 | 23.0, at 2,097,152 27.3 | 26.9; 4 x 2
//     21.3 | 21.6, 26.7 | 24.6), not with 5 to 8 columns against 2 to 4 (8 x 4 at
//     2,097,152 34.6 | 42.4), and against one column no earlier either, though it
//     would be faster from 2^19 on (4 x 1 18.0 | 17.4): the register kernel's
//     lanes sum in FP32;
//   * W'W up to 32 columns: half the tiles, one read (see pb_frag.cuh);
//   * blocks on 16-byte rows keep the TMA-staged kernels where those share
//     every row among many tiles: 64 x 8 207 | 202, 64 x 16 269 | 222,
//     32 x 16 160 | 152 (at 40 x 8 it is 148 | 149, at 32 x 8 129 | 128);
//   * everything else, whatever its alignment, up to 64 columns: there the
//     other kernels stage element by element (37 x 5 141 | 850).
template <class T>
bool frag_mvTmv(int64_t n, int m, int k, T alpha, const T* V, int64_t ldv, const T* W, int64_t ldw, T beta, T* C,
                int64_t ldc, T* mbox)
{
  if (n < 0 || m < 1 || k < 1 || m > 64 || k > 64) return false;
  const bool sym = V == W && ldv == ldw && m == k;
  const int big = std::max(m, k), small = std::min(m, k);
  const bool thin = small <= 4 && big <= (sizeof(T) == 4 ? 8 : 4);
  if (thin && n > (sizeof(T) == 8 && small == 1 ? 1 << 19 : 1 << 20) &&
      (small == 1 || (sizeof(T) == 4 ? big <= 4 : !sym && small == 4 && rows32(V, ldv) && rows32(W, ldw))))
    return false;
  const bool staged = rows16(V, ldv, m) && rows16(W, ldw, k);
  if (staged && (sym ? m > 32 : small > 8 ? big > 16 : big > 40)) return false;
  FragTnArgs<T> a;
  a.n = n;
  a.alpha = alpha;
  a.beta = beta;
  if (sym && m <= 32) {
    a.m = a.k = m;
    a.V = a.W = V; a.ldv = a.ldw = ldv;
    a.C = C; a.sr = 1; a.sc = ldc;
    a.mbox = mbox; a.mr = 1; a.mc = m;
    return pair_ok(V, ldv, m) ? tn_sym<T, true>(a) : tn_sym<T, false>(a);
  }
  // the wider block supplies the rows of the product, the narrower one at
  // most 16 columns at a time
  const bool swap = k > m;
  a.m = big;
  a.V = swap ? W : V; a.ldv = swap ? ldw : ldv;
  a.ldw = swap ? ldv : ldw;
  a.sr = swap ? ldc : 1; a.sc = swap ? 1 : ldc;
  a.mr = swap ? m : 1; a.mc = swap ? 1 : m;
  for (int j0 = 0; j0 < small; j0 += 16) {
    a.k = std::min(16, small - j0);
    a.W = (swap ? V : W) + j0;
    a.C = C + j0 * a.sc;
    a.mbox = mbox ? mbox + j0 * a.mc : nullptr;
    const bool vec = pair_ok(a.V, a.ldv, a.m) && pair_ok(a.W, a.ldw, a.k);
    if (a.k <= 8) vec ? tn_mt<T, 1, true>(a) : tn_mt<T, 1, false>(a);
    else vec ? tn_mt<T, 2, true>(a) : tn_mt<T, 2, false>(a);
  }
  return true;
}

// All products W = V C of up to 64 columns but the thin ones (FP32 3 x 3
// 41 | 23 us, FP64 40 | 39; see pb_frag.cuh for the others).
template <class T>
bool frag_mvsd(const RowGemmArgs<T>& r)
{
  const bool inplace = r.mode == RM_MVSDI;
  if (r.n < 1 || r.m < 1 || r.k < 1 || r.m > 64 || r.k > 64) return false;
  if (r.k <= 4 && r.m <= (sizeof(T) == 4 ? 8 : 4)) return false;
  FragNnArgs<T> a;
  a.n = r.n; a.m = r.m; a.k = r.k;
  a.V = inplace ? (const T*)r.W : r.V;
  a.ldv = inplace ? r.ldw : r.ldv;
  a.W = r.W; a.ldw = r.ldw;
  a.C = r.C; a.ldc = r.ldc;
  a.alpha = inplace ? T(1) : r.alpha;
  a.beta = inplace ? T(0) : r.beta;
  const bool vec = pair_ok(a.V, a.ldv, a.m) && pair_ok((const T*)a.W, a.ldw, a.k);
  if (a.k <= 8) return vec ? nn_mc<T, 1, true>(a) : nn_mc<T, 1, false>(a);
  if (a.k <= 16) return vec ? nn_mc<T, 2, true>(a) : nn_mc<T, 2, false>(a);
  if (a.k <= 32) return vec ? nn_mc<T, 4, true>(a) : nn_mc<T, 4, false>(a);
  return vec ? nn_mc<T, 8, true>(a) : nn_mc<T, 8, false>(a);
}

template <class T>
bool frag_mvsd_gram(const RowGemmArgs<T>& r, T* mbox)
{
  const bool inplace = r.mode == RM_MVSDI;
  if (r.n < 1 || r.m < 1 || r.k < 1 || r.m > 32 || r.k > 32) return false;
  FragNnArgs<T> a;
  a.n = r.n; a.m = r.m; a.k = r.k;
  a.V = inplace ? (const T*)r.W : r.V;
  a.ldv = inplace ? r.ldw : r.ldv;
  a.W = r.W; a.ldw = r.ldw;
  a.C = r.C; a.ldc = r.ldc;
  a.alpha = inplace ? T(1) : r.alpha;
  a.beta = inplace ? T(0) : r.beta;
  FragTnArgs<T> go;
  memset(&go, 0, sizeof(go));
  go.n = r.n; go.m = go.k = r.k;
  go.alpha = r.galpha; go.beta = r.gbeta;
  go.C = r.Gd; go.sr = 1; go.sc = r.ldg;
  go.mbox = mbox; go.mr = 1; go.mc = r.k;
  const bool vec = pair_ok(a.V, a.ldv, a.m) && pair_ok((const T*)a.W, a.ldw, a.k);
  switch ((a.k + 7) / 8) {
    case 1: vec ? nn_gram_mc<T, 1, true>(a, go) : nn_gram_mc<T, 1, false>(a, go); break;
    case 2: vec ? nn_gram_mc<T, 2, true>(a, go) : nn_gram_mc<T, 2, false>(a, go); break;
    case 3: vec ? nn_gram_mc<T, 3, true>(a, go) : nn_gram_mc<T, 3, false>(a, go); break;
    default: vec ? nn_gram_mc<T, 4, true>(a, go) : nn_gram_mc<T, 4, false>(a, go); break;
  }
  return true;
}

template bool frag_mvTmv<double>(int64_t, int, int, double, const double*, int64_t, const double*, int64_t, double,
                                 double*, int64_t, double*);
template bool frag_mvTmv<float>(int64_t, int, int, float, const float*, int64_t, const float*, int64_t, float, float*,
                                int64_t, float*);
template bool frag_mvsd<double>(const RowGemmArgs<double>&);
template bool frag_mvsd<float>(const RowGemmArgs<float>&);
template bool frag_mvsd_gram<double>(const RowGemmArgs<double>&, double*);
template bool frag_mvsd_gram<float>(const RowGemmArgs<float>&, float*);

}  // namespace pb
