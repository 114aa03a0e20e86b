// Shared host/device helpers of libkascade_b200.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "kascade_b200.h"

namespace kb200 {

// thread-local error text returned by kb200_last_error()
void set_error(const char* fmt, ...);
bool initialised(int* device_out);
int check_on_current_device(const void* ptr, const char* what);

#define KB_ENTRY(first_ptr, what)                                                                 \
  do {                                                                                            \
    KB_REQUIRE(kb200::initialised(nullptr),                                                       \
               "kb200_init has not been called for the device that is current in this thread");  \
    if (kb200::check_on_current_device(first_ptr, what) != 0) return -1;                          \
  } while (0)

#define KB_REQUIRE(cond, ...)        \
  do {                               \
    if (!(cond)) {                   \
      kb200::set_error(__VA_ARGS__); \
      return -1;                     \
    }                                \
  } while (0)

#define KB_CUDA(expr)                                                            \
  do {                                                                           \
    cudaError_t e__ = (expr);                                                    \
    if (e__ != cudaSuccess) {                                                    \
      kb200::set_error("%s failed: %s", #expr, cudaGetErrorString(e__));         \
      return -1;                                                                 \
    }                                                                            \
  } while (0)

// The check of a kernel launch: KB_LAUNCH of one that returns its error, KB_CHECK_LAUNCH after one with <<<>>>.  A launch that
// the runtime refuses is also left behind as its last error; both take it back, so that the next launch check in this
// thread (PyTorch's, for one) does not report it a second time.
#define KB_LAUNCH(name, launch)                                                  \
  do {                                                                           \
    const cudaError_t launched__ = (launch);                                     \
    if (launched__ != cudaSuccess) {                                             \
      cudaGetLastError();                                                        \
      kb200::set_error("launch of %s failed: %s", name, cudaGetErrorString(launched__)); \
      return -1;                                                                 \
    }                                                                            \
  } while (0)

#define KB_CHECK_LAUNCH(name)                                                    \
  do {                                                                           \
    cudaError_t e__ = cudaGetLastError();                                        \
    if (e__ != cudaSuccess) {                                                    \
      kb200::set_error("launch of %s failed: %s", name, cudaGetErrorString(e__)); \
      return -1;                                                                 \
    }                                                                            \
  } while (0)

constexpr int kD = KB200_HEAD_DIM;       // head dimension
constexpr int kHg = KB200_GROUP_SIZE;    // query heads per KV head
constexpr int kTile = KB200_TILE;        // queries per prefill tile
constexpr float kLog2e = 1.4426950408889634f;

// Programmatic dependent launch.  Every kernel that is launched with launch_pdl starts with pdl_wait(): it waits until the
// kernel before it in the stream has completed and its writes are visible.  pdl_trigger() lets the kernel after it be set
// up; that one's launch, block scheduling and parameter loads so fall into this one's run time instead of a gap of
// 1.5-2 us after it.  (The other kernels of the library, kv_write and zero_padding among them, are plain launches: they
// wait for the one before them in full.)
// When to trigger: the next kernel's CTAs go to whichever SMs have room at that moment and wait there.  While a grid of
// fewer CTAs than SMs runs, that is the handful of idle SMs, and the whole next kernel then runs on those.  So the long
// kernels with such grids (decode attention, Top-k, pooling) trigger when they are nearly done, and the others at their
// start (pdl_begin).  With plain launches, every trigger at the start, and as it is now: decode steps of 4 layers, 9
// sequences of 16000 tokens in an FP8 cache 131 / 135 / 129 us, 8 of 48000 in fp16 401 / 399 / 389 us; 16 layers of one
// sequence of 4000 174 / 159 / 156 us.
// Nothing may touch global memory before the wait, and nothing may be read through the non-coherent path
// (__ldg, ld.global.nc, a `const T* __restrict__` parameter): that asks for memory which nobody writes while the kernel
// lives, and this kernel lives already while the one before it writes its inputs.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_wait();
  pdl_trigger();
}
// launches a kernel that begins with pdl_wait() or pdl_begin(), as a cluster of `cluster` CTAs along x if that is not 1
template <typename... P, typename... A>
static inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st,
                                     unsigned cluster, const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

int sm_count();

// per-module init hooks (raise dynamic shared memory limits); defined in the kernel files
int init_decode();
int init_prefill();
int init_topk();
int init_selftest();

}  // namespace kb200
