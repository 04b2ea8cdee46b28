// pb_gmres_D.cu -- correction-equation solvers in FP64 (pb_gmres.cuh).
#include "pb_gmres.cuh"

extern "C" {

void phist_b200_DjadaCorrection_gmres(const void* A, const void* Q, const void* res, const int* resIndex, int k,
                                      const double* sigma, const double* tol, int maxIter, int maxBas, void* t,
                                      int* iflag)
{
  PB_API_BEGIN(iflag);
  const int u = pb::jada_gmres<double>(pb::SP<double>(A), Q ? pb::MV<double>(Q) : nullptr, pb::MV<double>(res), resIndex, k, sigma,
                                  tol, maxIter, maxBas, pb::MV<double>(t));
  *iflag = u;
  PB_API_END(iflag);
}

void phist_b200_DjadaCorrection_minres(const void* A, const void* Q, const void* res, const int* resIndex, int k,
                                       const double* sigma, const double* tol, int maxIter, int maxBas, void* t,
                                       int* iflag)
{
  PB_API_BEGIN(iflag);
  const int u = pb::jada_minres<double>(pb::SP<double>(A), Q ? pb::MV<double>(Q) : nullptr, pb::MV<double>(res), resIndex, k, sigma,
                                   tol, maxIter, maxBas, pb::MV<double>(t));
  *iflag = u;
  PB_API_END(iflag);
}

}  // extern "C"
