// pb_gmres_S.cu -- correction-equation solvers in FP32 (pb_gmres.cuh).
#include "pb_gmres.cuh"

extern "C" {

void phist_b200_SjadaCorrection_gmres(const void* A, const void* Q, const void* res, const int* resIndex, int k,
                                      const double* sigma, const double* tol, int maxIter, int maxBas, void* t,
                                      int* iflag)
{
  PB_API_BEGIN(iflag);
  const int u = pb::jada_gmres<float>(pb::SP<float>(A), Q ? pb::MV<float>(Q) : nullptr, pb::MV<float>(res), resIndex, k, sigma,
                                 tol, maxIter, maxBas, pb::MV<float>(t));
  *iflag = u;
  PB_API_END(iflag);
}

void phist_b200_SjadaCorrection_minres(const void* A, const void* Q, const void* res, const int* resIndex, int k,
                                       const double* sigma, const double* tol, int maxIter, int maxBas, void* t,
                                       int* iflag)
{
  PB_API_BEGIN(iflag);
  const int u = pb::jada_minres<float>(pb::SP<float>(A), Q ? pb::MV<float>(Q) : nullptr, pb::MV<float>(res), resIndex, k, sigma,
                                  tol, maxIter, maxBas, pb::MV<float>(t));
  *iflag = u;
  PB_API_END(iflag);
}

}  // extern "C"
