// Shared device helpers for the VecAttention kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "vecattn.h"

namespace va {

constexpr int kHeadDim = 128;

// ---- 16-bit element traits -------------------------------------------------------------------
template <int DT> struct Elem;
template <> struct Elem<VA_BF16> {
  using T = __nv_bfloat16;
  using T2 = __nv_bfloat162;
  static __device__ __forceinline__ float to_float(T x) { return __bfloat162float(x); }
  static __device__ __forceinline__ T from_float(float x) { return __float2bfloat16_rn(x); }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t w) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w));
  }
};
template <> struct Elem<VA_FP16> {
  using T = __half;
  using T2 = __half2;
  static __device__ __forceinline__ float to_float(T x) { return __half2float(x); }
  static __device__ __forceinline__ T from_float(float x) { return __float2half_rn(x); }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t w) {
    return __half22float2(*reinterpret_cast<__half2*>(&w));
  }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  int sz = valid ? 16 : 0;  // src-size 0 => 16 zero bytes are written
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(sz));
}
__device__ __forceinline__ void cp_async16_full(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// 2^x on the special-function unit (ex2.approx: 2 ulp, 2^-inf = 0)
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two fp32 values in one register pair, and arithmetic on both halves in one instruction (each half rounded as by the
// scalar instruction)
__device__ __forceinline__ uint64_t pair2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 halves(uint64_t x) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(x));
  return f;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// the largest of three, one instruction
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// 32-bit load that the compiler keeps where it is written (used to batch index loads)
__device__ __forceinline__ int load_here(const int32_t* p) {
  int v;
  asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// pull the 128-byte line at `p` into L2 (no register result, no wait)
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ---- errors of the runtime ------------------------------------------------------------------------
// A failed call's error stays with the thread until cudaGetLastError takes it, and the plain launches are checked with
// cudaGetLastError: a call that answers for itself takes its error back, or the next launch would be reported as failed.
inline bool succeeded(cudaError_t e) {
  if (e != cudaSuccess) cudaGetLastError();
  return e == cudaSuccess;
}

// ---- launches that overlap their predecessor's end -----------------------------------------------
// A kernel launched with launch_after may be scheduled while the kernel before it in the stream is still running, once
// every CTA of that one has let it (let_next_start) or ended.  It must not touch memory, not even read an argument's target, and
// no CTA of it may end before wait_for_previous, which returns when the kernel before has ended and its writes are visible:
// so the order of all effects is that of plain launches, also for the kernels after it.  What overlaps is the launch itself and, in the
// 64-row and the dense kernel, the setting up before the wait (barriers, tensor memory).
// Such a kernel reads global memory with coherent loads only: not with __ldg or ld.global.nc, which are for data that nobody writes
// while the kernel lives, and its life begins while the kernel before it is still writing.
// A call that is waited for: 4 heads x 2048 tokens 62.0 -> 57.2 us, 28/4 heads x 9001 360 -> 354, 20 011 around a vision span 817 -> 810;
// in a row of calls 34.2 -> 33.5 for the first, which the host limits.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... Params, typename... Args>
inline bool launch_after(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return succeeded(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
}

}  // namespace va
