// rows.cu -- the float32 host calls' conversions on the device: the caller's
// float32 arrays widened for the double kernels, and the results written in the
// caller's row formats (volume files' {x, y, z, Ex, Ey, Ez} in float32 and
// {x, y, z, phi} in float16, CPET/utils/calculator.py:430-475).  Each value is
// rounded once from the double result, as numpy's astype does it on the host.
// Bound: launches; the arrays are a few hundred kilobytes.
#include <algorithm>
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.cuh"

namespace cpetgb {
namespace {

constexpr int kRowThreads = 256;

// Also clears the counters of the launch that follows (a memset of its own is one
// more operation on the stream).
__global__ void widen_kernel(int64_t n, const float* __restrict__ in, double* __restrict__ out,
                             int* __restrict__ zeroed, int64_t n_zero) {
  const int64_t i0 = blockIdx.x * int64_t(blockDim.x) + threadIdx.x, stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t i = i0; i < n_zero; i += stride) zeroed[i] = 0;
  for (int64_t i = i0; i < n; i += stride) out[i] = widen(in[i]);
}

// The device status word goes behind the rows, so that one copy brings both.
template <int FMT>
__global__ void rows_kernel(int64_t n, const float* __restrict__ pts, const double* __restrict__ val,
                            void* __restrict__ rows, const int* __restrict__ status, int* __restrict__ tail) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *tail = *status;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    if constexpr (FMT == kRowsPlain) {
      static_cast<float*>(rows)[i] = narrow(val[i]);
    } else if constexpr (FMT == kRowsField) {
      float2* r = static_cast<float2*>(rows) + 3 * i;
      r[0] = make_float2(pts[3 * i], pts[3 * i + 1]);
      r[1] = make_float2(pts[3 * i + 2], narrow(val[3 * i]));
      r[2] = make_float2(narrow(val[3 * i + 1]), narrow(val[3 * i + 2]));
    } else {
      __half2* r = static_cast<__half2*>(rows) + 2 * i;
      r[0] = __halves2half2(__float2half_rn(pts[3 * i]), __float2half_rn(pts[3 * i + 1]));
      r[1] = __halves2half2(__float2half_rn(pts[3 * i + 2]), __double2half(val[i]));
    }
  }
}

int blocks_of(int64_t n) { return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((n + kRowThreads - 1) / kRowThreads, 4096))); }

}  // namespace

cudaError_t launch_widen(int64_t n, const float* in, double* out, int* zeroed, int64_t n_zero, cudaStream_t s) {
  if (n <= 0 && n_zero <= 0) return cudaSuccess;
  widen_kernel<<<blocks_of(std::max(n, n_zero)), kRowThreads, 0, s>>>(n, in, out, zeroed, n_zero);
  return cudaGetLastError();
}

cudaError_t launch_rows(int fmt, int64_t n, const float* pts, const double* val, void* rows, const int* status,
                        int* tail, cudaStream_t s) {
  switch (fmt) {
    case kRowsField:
      rows_kernel<kRowsField><<<blocks_of(n), kRowThreads, 0, s>>>(n, pts, val, rows, status, tail);
      break;
    case kRowsEspHalf:
      rows_kernel<kRowsEspHalf><<<blocks_of(n), kRowThreads, 0, s>>>(n, pts, val, rows, status, tail);
      break;
    default:
      rows_kernel<kRowsPlain><<<blocks_of(n), kRowThreads, 0, s>>>(n, pts, val, rows, status, tail);
  }
  return cudaGetLastError();
}

cudaError_t preload_row_kernels() {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, widen_kernel);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, rows_kernel<kRowsPlain>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, rows_kernel<kRowsField>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, rows_kernel<kRowsEspHalf>);
  return e;
}

}  // namespace cpetgb
