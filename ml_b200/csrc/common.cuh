// Shared device/host helpers for the sm_100a kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

#define MLB_API extern "C" __attribute__((visibility("default")))

// Error word shared by every kernel that can give up on a bounded wait (mbarrier, peer flag).
// 0 = ok.  Layout of a non-zero value: (code << 24) | detail.  Host reads it with mlb_get_error().
enum : int {
  MLB_ERR_NONE = 0,
  MLB_ERR_MBAR_TIMEOUT = 1,   // an mbarrier wait in a TMA/tcgen05 pipeline ran out
  MLB_ERR_FLAG_TIMEOUT = 2,   // a wait on a peer/host flag ran out
  MLB_ERR_BOUNDS = 3,         // a self-check found an index out of range
};
// Each translation unit owns one copy (no relocatable device code is used); MLB_DEFINE_ERROR_WORD(tag) also
// exports mlb_get_error_<tag>() / mlb_clear_error_<tag>() for the host.
#define MLB_DEFINE_ERROR_WORD(tag)                                             \
  MLB_API int mlb_get_error_##tag() {                                          \
    int v = 0;                                                                 \
    cudaMemcpyFromSymbol(&v, g_mlb_error, sizeof(int));                        \
    return v;                                                                  \
  }                                                                            \
  MLB_API void mlb_clear_error_##tag() {                                       \
    int v = 0;                                                                 \
    cudaMemcpyToSymbol(g_mlb_error, &v, sizeof(int));                          \
  }                                                                            \
  /* the word copied to (pinned) host memory behind the work already in `st`: no synchronisation of its own */ \
  MLB_API int mlb_read_error_async_##tag(int* host_dst, cudaStream_t st) {     \
    void* p = nullptr;                                                         \
    cudaError_t e = cudaGetSymbolAddress(&p, g_mlb_error);                     \
    if (e != cudaSuccess) return (int)e;                                       \
    return (int)cudaMemcpyAsync(host_dst, p, sizeof(int), cudaMemcpyDeviceToHost, st); \
  }
static __device__ int g_mlb_error = 0;

// ------------------------------------------------------------------ programmatic dependent launch
// Kernels started through mlb_launch() may become resident while the kernel before them in the stream is still
// draining: they run their own set-up, then mlb_pdl_sync() blocks until that kernel has completed and its writes are
// visible (and lets the kernel after this one start its set-up in turn).  Every global-memory access of such a
// kernel comes after the call.  Launched the ordinary way the instructions are no-ops.
__device__ __forceinline__ void mlb_pdl_sync() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#ifdef __CUDACC__
#include <atomic>
#include <cstdlib>
#include <utility>
// Which kernels start early, without MLB_PDL: all GEMMs, the persistent attention kernels of one wave (no more items than SMs), the split attention
// kernels up to a limit of their own (split_early), and element-wise kernels of no more threads than the machine holds (2048 an SM: one
// wave, or two where a kernel's registers allow half as many).  A chain of small kernels is bound by launch and set-up, which then run under the kernel before: step of
// the 4-layer / 128-wide decoder 637 -> 567 us, rotary copy and causal attention forward, 12 heads of 64, of 500 tokens 16.5 -> 15.2, of 8 x 256
// 14.6 -> 13.8, of 3 x 1000 31.6 -> 28.7 (in a captured graph, whose launches are closer anyway, 15.4 -> 14.8, 13.2 -> 13.6, 27.0 -> 26.8); GEMMs of any size gain 2 to 3 us of
// launch gap each (step of the 12-layer decoder 17.35 -> 17.11 ms, captured 16.40 -> 16.29).
// Larger ones stay out: their CTAs sit on the SMs while the kernel before still works there, and take registers and issue slots from
// it (every kernel early: attention at 16 x 1024 tokens 269 -> 283 us).
// A kernel that allocates tensor memory before its mlb_pdl_sync() may hold it while the kernel before has CTAs that are still to allocate only
// if both fit an SM; those that allocate after it (attention at head sizes 64 and 128) have more than 200 KB of shared memory and fit beside none.
// MLB_PDL=0: none; 1: all; 2: all element-wise ones.
enum { MLB_PDL_NONE = 0, MLB_PDL_ALL = 1, MLB_PDL_ELEMENTWISE = 2, MLB_PDL_BY_SIZE = 3 };
inline int mlb_pdl_mode() {
  static int mode = -1;
  if (mode < 0) {
    const char* e = getenv("MLB_PDL");
    mode = (e != nullptr && e[0] >= '0' && e[0] <= '2') ? e[0] - '0' : MLB_PDL_BY_SIZE;
  }
  return mode;
}
inline int mlb_sm_count() {
  static const int n = [] {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) cudaGetLastError();
    return sms > 0 ? sms : 148;
  }();
  return n;
}
// More than 48 KB of dynamic shared memory for `kern`, asked for once on each device (bit of `done`; beyond 64 devices each time)
template <typename K>
inline cudaError_t mlb_allow_smem(K kern, size_t bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
  if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return e;
}
template <typename... KArgs, typename... Args>
inline cudaError_t mlb_launch_attr(bool early, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t mlb_launch(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  const int mode = mlb_pdl_mode();
  const bool early = mode == MLB_PDL_BY_SIZE ? (long)grid.x * grid.y * grid.z * block.x <= 2048L * mlb_sm_count() : mode != MLB_PDL_NONE;
  return mlb_launch_attr(early, kern, grid, block, smem, st, std::forward<Args>(args)...);
}
// for kernels that allocate tensor memory (GEMMs, attention): `small`, of those that start early by size
inline bool mlb_pdl_tmem(bool small) { return mlb_pdl_mode() == MLB_PDL_ALL || (mlb_pdl_mode() == MLB_PDL_BY_SIZE && small); }
template <typename... KArgs, typename... Args>
inline cudaError_t mlb_launch_tmem(bool small, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  return mlb_launch_attr(mlb_pdl_tmem(small), kern, grid, block, smem, st, std::forward<Args>(args)...);
}
#endif

__device__ __forceinline__ void mlb_set_error(int code, int detail) {
  atomicCAS(&g_mlb_error, 0, (code << 24) | (detail & 0xFFFFFF));
}

static inline int ceil_div_i(long a, long b) { return (int)((a + b - 1) / b); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum for blockDim.x <= 1024 (multiple of 32). `red` needs 32 floats of shared memory.
__device__ __forceinline__ float block_sum(float v, float* red) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}
__device__ __forceinline__ float block_max(float v, float* red) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : -INFINITY;
  t = warp_max(t);
  return t;
}

struct __align__(16) bf16x8 { bf162 v[4]; };

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  bf162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&t);
}
