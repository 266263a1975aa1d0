// The two ends of a step, as kernels: between kernels the device's copy engine and a memset cost a step their change-over
// (9 us from the last kernel to the copy of the error code, 5 us each for the copies and the memset, 4 us to the next kernel:
// 28 us of a 640 us decode step; with these 10).
#include "common.cuh"

// The step's int arrays from pinned host memory to the device, and the counter of the chain kernels' barrier back to zero.
// Bound by the trip over PCIe, so every thread asks for all its words before it stores any.  No pdl_trigger: the kernels of
// the step read these arrays before their own pdl_wait, and must not begin before this one has ended.
__global__ void __launch_bounds__(256) step_begin_kernel(const int4* __restrict__ host, int4* __restrict__ dev, int n4, unsigned* barrier,
                                                         int n_barrier) {
  pdl_wait();
  constexpr int PER = 4;
  int4 v[PER];
  const int at = blockIdx.x * (256 * PER) + threadIdx.x;
#pragma unroll
  for (int i = 0; i < PER; ++i)
    if (at + i * 256 < n4) asm volatile("ld.volatile.global.v4.s32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v[i].x), "=r"(v[i].y), "=r"(v[i].z), "=r"(v[i].w) : "l"(host + at + i * 256));
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < n_barrier; i += 256) barrier[i] = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i)
    if (at + i * 256 < n4) dev[at + i * 256] = v[i];
}

// Behind a step's kernels: a code that one of them left is written where the host looks for it.
__global__ void step_end_kernel(const int* __restrict__ err, int* host) {
  pdl_trigger();
  pdl_wait();
  const int code = *err;
  if (code != 0) {
    *reinterpret_cast<volatile int*>(host) = code;
    __threadfence_system();
  }
}

// host: pinned memory, 16-byte aligned like dev; n_ints is rounded up to whole 16 bytes (both buffers have room for that).
Q25_EXPORT int q25_step_begin(const void* host, void* dev, int n_ints, void* barrier, int n_barrier, void* stream) {
  if (n_ints < 0 || n_barrier < 0 || ((uintptr_t)host & 15) || ((uintptr_t)dev & 15)) return (int)cudaErrorInvalidValue;
  const int n4 = (n_ints + 3) / 4, blocks = (n4 + 1023) / 1024;
  step_begin_kernel<<<blocks > 0 ? blocks : 1, 256, 0, (cudaStream_t)stream>>>((const int4*)host, (int4*)dev, n4, (unsigned*)barrier, n_barrier);
  return launch_status();
}

Q25_EXPORT int q25_step_end(const int* err, int* host, void* stream) {
  launch(step_end_kernel, dim3(1), dim3(1), 0, (cudaStream_t)stream, err, host);
  return launch_status();
}
