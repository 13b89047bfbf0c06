// The FP64 factors of a context, for test_gpu_factors.py.
#include "fp_internal.cuh"

extern "C" int factors(fp_ctx* c, double* lu, int32_t* piv) {
  if (cudaMemcpy2D(lu, c->N * sizeof(double), c->d_LU, c->ld * sizeof(double), c->N * sizeof(double), c->N,
                   cudaMemcpyDeviceToHost))
    return 1;
  return (int)cudaMemcpy(piv, c->d_ipiv, c->N * sizeof(int32_t), cudaMemcpyDeviceToHost);
}
