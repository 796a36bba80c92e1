// Row-major activations for the kernels that want A col-major, and operands kept in 16-bit
// storage (IEEE half, bfloat16).
//
// Every half and bfloat16 value is a TF32 value (at most 10 mantissa bits, exponent within
// FP32's), so widening loses nothing and the tensor-core path, which drops the low 13
// mantissa bits of its FP32 operands, multiplies widened 16-bit operands exactly; sums are
// FP32 on both paths.  The conversions therefore sit where the data is touched anyway:
// activations are widened by the kernel that transposes them into the multiply's col-major
// layout, weights once when they are compressed, and the result is rounded (to nearest even)
// by one pass over C.  All three are HBM-bound element-wise kernels.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"

namespace nmspmm {

template <typename T> __device__ __forceinline__ float widen(T v);
template <> __device__ __forceinline__ float widen<float>(float v) { return v; }
template <> __device__ __forceinline__ float widen<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float widen<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T narrow(float v);
template <> __device__ __forceinline__ __half narrow<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 narrow<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Four adjacent values, in one load where the row starts on a multiple of that load.
template <typename T>
__device__ __forceinline__ float4 load_four(const T* p, bool aligned)
{
    union { T v[4]; uint2 w2; uint4 w4; } x;
    if (aligned) {
        if constexpr (sizeof(T) == 4) x.w4 = __ldg(reinterpret_cast<const uint4*>(p));
        else x.w2 = __ldg(reinterpret_cast<const uint2*>(p));
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) x.v[i] = p[i];
    }
    return make_float4(widen<T>(x.v[0]), widen<T>(x.v[1]), widen<T>(x.v[2]), widen<T>(x.v[3]));
}

// Row-major activations [M][K] (K a multiple of 4) -> FP32 col-major [K][ld], ld a multiple of 4, columns
// M .. ld-1 zero.  HBM-bound: M K values in, 4 ld K bytes out.  A thread transposes 4 rows x 4 k in its
// registers; a warp covers 32 rows x 16 k, so that it writes whole 128-byte lines and reads whole
// 32-byte sectors, four independent loads per thread in flight.  32 x 32 patches through shared
// memory with 4-byte accesses took 21 us of a training pass at 2048 x 4096, this 12.
template <typename T>
__global__ void __launch_bounds__(256) transpose_rows_kernel(const T* __restrict__ in, float* __restrict__ out, int M, int K, int ld, int aligned)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = blockIdx.x * 128 + warp * 16 + (lane >> 3) * 4, m = (blockIdx.z * gridDim.y + blockIdx.y) * 32 + (lane & 7) * 4;
    grid_dependency_wait();
    if (k < K && m < ld) {
        float4 r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            r[j] = m + j < M ? load_four<T>(in + static_cast<size_t>(m + j) * K + k, aligned != 0) : make_float4(0.f, 0.f, 0.f, 0.f);
        grid_launch_dependents();
        float* o = out + static_cast<size_t>(k) * ld + m;
        *reinterpret_cast<float4*>(o) = make_float4(r[0].x, r[1].x, r[2].x, r[3].x);
        *reinterpret_cast<float4*>(o + ld) = make_float4(r[0].y, r[1].y, r[2].y, r[3].y);
        *reinterpret_cast<float4*>(o + 2 * static_cast<size_t>(ld)) = make_float4(r[0].z, r[1].z, r[2].z, r[3].z);
        *reinterpret_cast<float4*>(o + 3 * static_cast<size_t>(ld)) = make_float4(r[0].w, r[1].w, r[2].w, r[3].w);
    }
}

// n floats -> n 16-bit values, four per thread and step (n % 4 == 0, both 8-byte aligned).
template <typename T>
__global__ void __launch_bounds__(256) narrow_kernel(const float4* __restrict__ in, T* __restrict__ out, size_t n4)
{
    grid_dependency_wait();
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n4; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const float4 v = in[i];
        union { T h[4]; uint2 u; } w;
        w.h[0] = narrow<T>(v.x); w.h[1] = narrow<T>(v.y); w.h[2] = narrow<T>(v.z); w.h[3] = narrow<T>(v.w);
        reinterpret_cast<uint2*>(out)[i] = w.u;
    }
}

// n 16-bit values -> n floats (n % 4 == 0).
template <typename T>
__global__ void __launch_bounds__(256) widen_kernel(const T* __restrict__ in, float4* __restrict__ out, size_t n4)
{
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n4; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        union { T h[4]; uint2 u; } w;
        w.u = reinterpret_cast<const uint2*>(in)[i];
        out[i] = make_float4(widen<T>(w.h[0]), widen<T>(w.h[1]), widen<T>(w.h[2]), widen<T>(w.h[3]));
    }
}

static unsigned flat_grid(size_t n4)
{
    const size_t want = (n4 + 255) / 256;
    return static_cast<unsigned>(want < 1 ? 1 : (want > 148 * 16 ? 148 * 16 : want));     // grid-stride: a few CTAs per SM
}

template <typename T>
static cudaError_t launch_transpose(const void* in, float* out, int M, int K, int ld, cudaStream_t st)
{
    constexpr int kMaxY = 65535;                           // blocks of 32 rows along y; more of them (over 2097120 rows) go on along z
    const int blocks = (ld + 31) / 32;
    const dim3 grid((K + 127) / 128, blocks < kMaxY ? blocks : kMaxY, (blocks + kMaxY - 1) / kMaxY);
    const int aligned = reinterpret_cast<uintptr_t>(in) % (4 * sizeof(T)) == 0 ? 1 : 0;
    return launch_overlapped(transpose_rows_kernel<T>, grid, 256, 0, st, static_cast<const T*>(in), out, M, K, ld, aligned);
}

cudaError_t launch_transpose_rows(int dtype, const void* in, float* out, int M, int K, int ld, cudaStream_t st)
{
    if (dtype == kDtypeF32) return launch_transpose<float>(in, out, M, K, ld, st);
    if (dtype == kDtypeF16) return launch_transpose<__half>(in, out, M, K, ld, st);
    if (dtype == kDtypeBF16) return launch_transpose<__nv_bfloat16>(in, out, M, K, ld, st);
    return cudaErrorInvalidValue;
}

cudaError_t launch_narrow(int dtype, const float* in, void* out, size_t n, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (n % 4 != 0) return cudaErrorInvalidValue;
    if (dtype == kDtypeF16)
        return launch_overlapped(narrow_kernel<__half>, flat_grid(n / 4), 256, 0, st, reinterpret_cast<const float4*>(in), static_cast<__half*>(out), n / 4);
    if (dtype == kDtypeBF16)
        return launch_overlapped(narrow_kernel<__nv_bfloat16>, flat_grid(n / 4), 256, 0, st, reinterpret_cast<const float4*>(in), static_cast<__nv_bfloat16*>(out), n / 4);
    return cudaErrorInvalidValue;
}

cudaError_t launch_widen(int dtype, const void* in, float* out, size_t n, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (n % 4 != 0) return cudaErrorInvalidValue;
    if (dtype == kDtypeF16)
        widen_kernel<__half><<<flat_grid(n / 4), 256, 0, st>>>(static_cast<const __half*>(in), reinterpret_cast<float4*>(out), n / 4);
    else if (dtype == kDtypeBF16)
        widen_kernel<__nv_bfloat16><<<flat_grid(n / 4), 256, 0, st>>>(static_cast<const __nv_bfloat16*>(in), reinterpret_cast<float4*>(out), n / 4);
    else
        return cudaErrorInvalidValue;
    return cudaGetLastError();
}

}  // namespace nmspmm
