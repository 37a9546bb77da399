// Errors of the FP32 edge arithmetic (csrc/common.cuh cutoff_fc, edge_length)
// against 64 bits, beside those of CUDA's own functions, over every float of the
// ranges that matter.  Driven by tests/test_gpu_edge_math.py through ctypes.
#include "common.cuh"

namespace {

enum { kMax, kSum, kSlots };   // per quantity: largest error, sum of squared errors

__device__ void add(double* acc, int quantity, double err)
{
  err = fabs(err);
  double sum = err * err;
  for (int o = 16; o > 0; o >>= 1) {
    err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(reinterpret_cast<unsigned long long*>(acc + quantity * kSlots + kMax),
              static_cast<unsigned long long>(__double_as_longlong(err)));
    atomicAdd(acc + quantity * kSlots + kSum, sum);
  }
}

// x = d / rc over the floats of [first, first + n): fc absolute, fc' relative,
// fc relative; engine then CUDA.
__global__ void k_cutoff(unsigned first, unsigned n, double* acc)
{
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
    const float x = __uint_as_float(first + k);
    float fc, fcp, s, c;
    nepx::cutoff_fc(1.0f, 1.0f, x, fc, fcp);
    sincospif(x, &s, &c);
    const double half = 0.5 * static_cast<double>(x);
    const double ref = cospi(half) * cospi(half);
    const double ref_p = -1.5707963267948966 * sinpi(static_cast<double>(x));
    const float cfc = 0.5f * c + 0.5f, cfcp = -1.5707963f * s;
    add(acc, 0, fc - ref);
    add(acc, 1, cfc - ref);
    add(acc, 2, fcp / ref_p - 1.0);
    add(acc, 3, cfcp / ref_p - 1.0);
    add(acc, 4, fc / ref - 1.0);
    add(acc, 5, cfc / ref - 1.0);
  }
}

// d^2 over the floats from `first`: the length and its reciprocal, relative
// errors; engine then CUDA; and the number of lengths that are not sqrtf's.
__global__ void k_length(unsigned first, unsigned n, double* acc)
{
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
    const float d2 = __uint_as_float(first + k);
    float d, dinv;
    nepx::edge_length<false>(d2, d, dinv);
    const float cd = sqrtf(d2), cdinv = 1.0f / cd;
    const double ref = sqrt(static_cast<double>(d2));
    add(acc, 0, d / ref - 1.0);
    add(acc, 1, cd / ref - 1.0);
    add(acc, 2, dinv * ref - 1.0);
    add(acc, 3, cdinv * ref - 1.0);
    add(acc, 4, d == cd ? 0.0 : 1.0);
  }
}

}  // namespace

// acc: 12 doubles, per quantity the largest error and the sum of the squared
// errors.  n is a multiple of 32 (whole warps).
extern "C" int edge_math(int which, unsigned first, unsigned n, double* out)
{
  double* acc = nullptr;
  if (n % 32 != 0 || cudaMalloc(&acc, 12 * sizeof(double)) != cudaSuccess) return 1;
  cudaMemset(acc, 0, 12 * sizeof(double));
  if (which == 0) k_cutoff<<<148 * 4, 256>>>(first, n, acc);
  else k_length<<<148 * 4, 256>>>(first, n, acc);
  const cudaError_t err = cudaMemcpy(out, acc, 12 * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(acc);
  return err == cudaSuccess ? 0 : 2;
}
