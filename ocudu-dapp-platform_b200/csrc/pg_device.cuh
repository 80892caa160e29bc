// Device helpers shared by the pusch_b200 kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace pg {

// std::isnormal for device code: finite, non-zero and not subnormal.
__device__ __forceinline__ bool is_normal(float x)
{
  const float a = fabsf(x);
  return a >= 1.17549435e-38f && a <= 3.40282347e+38f;
}

// c(bit) .. c(bit + 31) of the TS 38.211 Section 5.2.1 Gold sequence with initialisation c_init
// (bit j of the result = c(bit + j)). tab holds 32 basis sequences of `words` words each, from
// position Nc = 1600: row 0 = x1 from (1, 0, ..., 0), row i + 1 = x2 from the unit state e_i; c is
// linear in c_init, so any sequence is x1 xor the rows of the set bits of c_init.
__device__ __forceinline__ uint32_t gold_word(const uint32_t* __restrict__ tab, uint32_t words, uint32_t c_init,
                                              uint32_t bit)
{
  const uint32_t w  = bit >> 5;
  const uint32_t sh = bit & 31u;
  uint32_t       lo = __ldg(tab + w), hi = __ldg(tab + w + 1);
#pragma unroll
  for (int i = 0; i < 31; ++i) {
    if ((c_init >> i) & 1u) {
      const uint32_t* b = tab + (size_t)(i + 1) * words;
      lo ^= __ldg(b + w);
      hi ^= __ldg(b + w + 1);
    }
  }
  return sh ? ((lo >> sh) | (hi << (32 - sh))) : lo;
}

// Programmatic dependent launch. launch_dependents: the next kernel of the stream, if launched to allow it
// (launch_overlapped), may start once every CTA of this grid has called it or exited. wait_prerequisites: until
// the kernels before this one have completed and their memory is visible; without such a launch it returns at
// once. Everything before it may touch only memory that no earlier kernel of the stream writes. What an earlier
// kernel does write is written while this one runs, so it is never read-only here: it is read after the wait and
// with load_written, not with __ldg, which may be served from a line cached before the write, nor with a plain load
// through const __restrict__, which the compiler may turn into the same and move ahead of the wait.
__device__ __forceinline__ void launch_dependents()
{
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_prerequisites()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Coherent loads, in order with the wait (both are volatile).
__device__ __forceinline__ int load_written(const int8_t* p)
{
  int v;
  asm volatile("ld.global.s8 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t load_written(const uint32_t* p)
{
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 load_written(const uint2* p)
{
  uint2 v;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 load_written(const float2* p)
{
  float2 v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}

// Launches a kernel that calls wait_prerequisites and may start before the kernel ahead of it has completed.
template <class... P, class... A>
inline cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args)
{
  cudaLaunchAttribute attr = {};
  attr.id                  = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim            = grid;
  cfg.blockDim           = block;
  cfg.dynamicSmemBytes   = smem;
  cfg.stream             = s;
  cfg.attrs              = &attr;
  cfg.numAttrs           = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

} // namespace pg
