// Shared helpers for the sm_100a kernels of lightron_b200.
// Every entry point is extern "C", returns 0 or a negative code, and launches on the
// caller's stream.  Nothing here allocates device memory.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#define LB_OK 0
#define LB_ERR_ARG (-1)
#define LB_ERR_LAUNCH (-2)
#define LB_ERR_SHAPE (-3)
#define LB_ERR_DRIVER (-4)
#define LB_ERR_TMAP (-5)
#define LB_ERR_CAPACITY (-6)

extern int g_lb_last_cuda_error;
// Wall-time limit of every device-side wait on a flag that another GPU or CTA writes
// (lb_set_flag_wait_ns; kernels take it as a launch parameter).
extern unsigned long long g_lb_flag_wait_ns;
// Number of SMs of the current device (queried once per device).
int lb_num_sms();

#define LB_CHECK_LAUNCH()                                   \
  do {                                                      \
    cudaError_t e__ = cudaGetLastError();                   \
    if (e__ != cudaSuccess) {                               \
      g_lb_last_cuda_error = (int)e__;                      \
      return LB_ERR_LAUNCH;                                 \
    }                                                       \
  } while (0)

// ---- dependent launches --------------------------------------------------------------------------
// A kernel launched by lb_launch() may start as soon as every CTA of the kernel before it in the stream has called grid_go() or has ended:
// its launch, barriers, tensor memory and descriptors then run under the other's tail.  Its first access to memory that
// another kernel writes or reads comes behind grid_wait(), which returns when the kernels before it have completed and their writes are
// visible; every thread calls it, so that no bounded wait of a CTA's roles runs meanwhile.  A kernel that allocates tensor memory calls
// grid_go() behind the allocation: a later kernel's CTA could otherwise hold the columns for which an earlier one waits.  grid_wait() does nothing in a
// plain launch, but grid_go() does: whether the NEXT kernel starts early is that one's attribute.  So kernels that wait for other GPUs are launched
// plainly and do not call grid_go() either: the next kernel's CTAs would fill the SMs for as long as the peers take, and what runs on other streams, which a
// peer may be waiting for, would find no room.  Launched plainly, too, is one of very many short blocks (a block's grid_wait() takes
// some 0.3 us: 32000 of clear_kernel 31 instead of 23 us).  No grid_go() in kernels that fill an SM's shared memory or registers: the next one's
// CTAs would crowd into the SMs that are done first (1000 x 768 feed-forward, four launches, 76 instead of 74 us); for the same reason it does
// nothing in a grid of many blocks, whose own time is not that of a launch.
// (Host time of a launch, 700 bytes of parameters, plain / dependent: 3.05 / 2.48 us.)
__device__ __forceinline__ void grid_go() {
  if (gridDim.x <= 1024) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename T> struct lb_as_is { typedef T type; };      // (arguments convert to the kernel's parameter types)
// Launches `fn` on clusters of `cluster` CTAs; `dependent` as above.
template <typename... K>
inline int lb_launch_cluster(bool dependent, int cluster, void (*fn)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                             const typename lb_as_is<K>::type&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  unsigned n = 0;
  if (dependent) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = (unsigned)cluster; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
    n++;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  void* a[] = {const_cast<void*>(static_cast<const void*>(&args))...};
  const cudaError_t e = cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(fn), a);
  if (e != cudaSuccess) { cudaGetLastError(); g_lb_last_cuda_error = (int)e; return LB_ERR_LAUNCH; }
  return LB_OK;
}
template <typename... K>
inline int lb_launch(void (*fn)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const typename lb_as_is<K>::type&... args) {
  return lb_launch_cluster(true, 1, fn, grid, block, smem, s, args...);
}
#define LB_LAUNCH(...)                                      \
  do {                                                      \
    const int rc__ = lb_launch(__VA_ARGS__);                \
    if (rc__ != LB_OK) return rc__;                         \
  } while (0)

typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

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

// 8 bf16 <-> 8 floats through one 16-byte vector
struct __align__(16) bf16x8 {
  bf162 v[4];
};
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const bf162* p = reinterpret_cast<const bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 u;
  bf162* p = reinterpret_cast<bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// RoPE of 8 columns: pairs (a, b) to (a c - b s, a s + b c), with four cosines and four sines; `back`: by the opposite angle.  In each sum one product
// is rounded and the other is not.  Which one is written out, because the compiler chose differently from place to place, and 2e-5 of the bf16
// results then differed between the kernels: here as rope_kernel has always had it (the first pair, and every pair on the way back, round a s).
__device__ __forceinline__ void rope_rotate8(const float* cs, float* f, bool back = false) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float a = f[2 * i], b = f[2 * i + 1], c = cs[i], s = back ? -cs[4 + i] : cs[4 + i];
    f[2 * i] = __fmaf_rn(a, c, -__fmul_rn(b, s));
    f[2 * i + 1] = i == 0 || back ? __fmaf_rn(b, c, __fmul_rn(a, s)) : __fmaf_rn(a, s, __fmul_rn(b, c));
  }
}
