// The integer-pipe arithmetic of nsw6_soft.cuh on the device, one routine over an
// array (tests/test_gpu_softfp.py).
#include "nsw6_common.cuh"

using namespace nsw6;

enum { DIV, DIV_RN, RCP, SQRT, D2F, F2D, RCP_SEED, RSQRT_SEED };

__global__ void apply(int op, const double* a, const double* b, double* out, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double x = a[i], y = b[i];
    switch (op) {
      case DIV: out[i] = soft_div(x, y); break;
      case DIV_RN: out[i] = soft_div_rn(x, soft_divisor(y), y); break;
      case RCP: out[i] = soft_rcp(soft_divisor(y), y); break;
      case SQRT: out[i] = soft_sqrt(x); break;
      case D2F: out[i] = (double)soft_d2f(x); break;
      case F2D: out[i] = soft_f2d((float)x); break;
      case RCP_SEED: out[i] = (double)soft_rcp_seed((float)x); break;
      case RSQRT_SEED: out[i] = (double)soft_rsqrt_seed((float)x); break;
    }
  }
}

// device pointers of n doubles each; a CUDA error's number
extern "C" int softfp_apply(int op, const double* a, const double* b, double* out, long long n) {
  apply<<<1216, 256>>>(op, a, b, out, n);
  const cudaError_t e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
