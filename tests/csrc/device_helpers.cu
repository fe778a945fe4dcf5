// Kernels that call single device helpers of the library, and calls of its internal stages, for
// tests/test_gpu_device_helpers.py.
#include "common.cuh"
#include "gemm.cuh"
#include "kernels.h"

using namespace xtbeig;

__global__ void wait_kernel(int raise_to, int want, uint64_t limit_ns, DeviceStatus* st, int* result) {
  __shared__ int count;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  if (threadIdx.x < 32) {
    result[threadIdx.x] = wait_count(&count, want, st, limit_ns, 5) ? 1 : 0;
  } else if (threadIdx.x == 32) {
    *(volatile int*)&count = raise_to;
  }
}

// One warp waits for a counter that another raises to raise_to.  Returns the CUDA error.
extern "C" int run_wait(int raise_to, int want, long long limit_ns, int* status, int* result) {
  DeviceStatus* st = nullptr;
  int* r = nullptr;
  cudaError_t err = cudaMalloc(&st, sizeof(DeviceStatus));
  if (err == cudaSuccess) err = cudaMalloc(&r, 32 * sizeof(int));
  if (err == cudaSuccess) err = cudaMemset(st, 0, sizeof(DeviceStatus));
  if (err == cudaSuccess) {
    wait_kernel<<<1, 64>>>(raise_to, want, (uint64_t)limit_ns, st, r);
    err = cudaDeviceSynchronize();
  }
  if (err == cudaSuccess) err = cudaMemcpy(status, st, sizeof(DeviceStatus), cudaMemcpyDeviceToHost);
  if (err == cudaSuccess) err = cudaMemcpy(result, r, 32 * sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(st);
  cudaFree(r);
  return (int)err;
}

__global__ void divide_kernel(int n, const double* a, const double* x, double* rcp, double* quot, double* plain) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  rcp[i] = rcp_normal(x[i]);
  quot[i] = div_normal(a[i], x[i]);
  plain[i] = a[i] / x[i];
}

// 1 / x, a / x and the compiler's a / x for n pairs in device memory.
extern "C" int run_divide(int n, const double* a, const double* x, double* rcp, double* quot, double* plain) {
  divide_kernel<<<(n + 255) / 256, 256>>>(n, a, x, rcp, quot, plain);
  return (int)cudaDeviceSynchronize();
}

// A launch that the runtime refuses on the host (on the legacy stream while another stream captures): what the grouped
// GEMM's launcher returns.  The descriptors are empty problems, so a launch that went through would do nothing.
extern "C" int run_refused_gemm(int nprob) {
  cudaStream_t s = nullptr;
  cudaGraph_t graph = nullptr;
  GemmDesc<double>* empty = nullptr;
  const size_t bytes = (nprob + 1) * sizeof(*empty);
  cudaError_t err = cudaMalloc(&empty, bytes);
  if (err == cudaSuccess) err = cudaMemset(empty, 0, bytes);
  if (err == cudaSuccess) err = cudaDeviceSynchronize();
  if (err == cudaSuccess) err = cudaStreamCreate(&s);
  if (err == cudaSuccess) err = cudaStreamBeginCapture(s, cudaStreamCaptureModeGlobal);
  if (err != cudaSuccess) return -1;
  const int refused = (int)gemm_grouped_launch<double>(empty, nprob, 1, 64, nullptr);
  cudaStreamEndCapture(s, &graph);
  if (graph) cudaGraphDestroy(graph);
  cudaStreamDestroy(s);
  cudaGetLastError();
  cudaFree(empty);
  return refused;
}

// The divide and conquer stage on device buffers d (n), e (n - 1), z (ldz x n), with a status word that starts at `code`.
extern "C" int run_stedc(int n, double* d, double* e, double* z, int ldz, int m_cols, int leaf, int code, int* status) {
  void *work = nullptr, *plan = nullptr, *stage = nullptr;
  DeviceStatus* st = nullptr;
  const size_t wb = stedc_work_bytes(n), sb = (size_t)40 * n * sizeof(int) + 4 * (n + 8) * sizeof(GemmDesc<double>) + 4096;
  const DeviceStatus start{code, 0, 0, 0};
  cudaError_t err = cudaMalloc(&work, wb);
  if (err == cudaSuccess) err = cudaMalloc(&plan, stedc_plan_bytes(n));
  if (err == cudaSuccess) err = cudaMallocHost(&stage, sb);
  if (err == cudaSuccess) err = cudaMalloc(&st, sizeof(start));
  if (err == cudaSuccess) err = cudaMemcpy(st, &start, sizeof(start), cudaMemcpyHostToDevice);
  if (err == cudaSuccess) err = stedc_device(n, d, e, z, ldz, work, wb, plan, true, stage, sb, st, nullptr, m_cols, leaf);
  if (err == cudaSuccess) err = cudaDeviceSynchronize();
  if (err == cudaSuccess) err = cudaMemcpy(status, st, sizeof(start), cudaMemcpyDeviceToHost);
  cudaFree(st);
  cudaFreeHost(stage);
  cudaFree(plan);
  cudaFree(work);
  return (int)err;
}
