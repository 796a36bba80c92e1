// Stores of FP32 results into a C of half or bfloat16 (rounded to nearest even).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "gemm_args.h"

namespace nmspmm {

__device__ __forceinline__ uint32_t round_pair(float lo, float hi, int dtype)
{
    if (dtype == kDtypeF16) {
        const __half2 h = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Four adjacent elements from element `at` of a 16-bit C on (C as GemmArgs holds it).
__device__ __forceinline__ void store_four_16(float* C, size_t at, float4 v, int dtype)
{
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(C) + at) = make_uint2(round_pair(v.x, v.y, dtype), round_pair(v.z, v.w, dtype));
}

}  // namespace nmspmm
