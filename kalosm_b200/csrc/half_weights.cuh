// Quantised weights to fp16 operands, as the prompt products (qgemm.cu, qgemm_pair.cu) convert them.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

namespace {

__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 u2h(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// Four unsigned bytes -> four fp16 values ((1024 + byte) - centre) * scale + offset, as two half2.
__device__ __forceinline__ uint2 deq4(uint32_t w, __half2 centre, __half2 scale, __half2 offset) {
  const __half2 v01 = __hsub2(u2h(__byte_perm(w, 0x64646464u, 0x4140)), centre);
  const __half2 v23 = __hsub2(u2h(__byte_perm(w, 0x64646464u, 0x4342)), centre);
  return make_uint2(h2u(__hfma2(v01, scale, offset)), h2u(__hfma2(v23, scale, offset)));
}

}  // namespace
