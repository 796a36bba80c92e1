// Vector-wise N:M magnitude pruning on the GPU: dense weight [K][N] -> compressed values
// BT [W][N] and window-local indices DT [W][Q], the inputs of the index packing and the
// multiply, so that a weight matrix never has to visit the host.
//
// Rule (the package's host generator formats.prune_magnitude states the same): in every
// window of 32 consecutive k rows and for every vector of vec_len (32 or 64) columns keep the
// n_keep rows with the largest sum of squares over the vector's columns, ties to the lower
// row; kept rows in ascending order.  The sum of squares is taken in double precision with
// eight interleaved partial sums combined pairwise -- the order numpy's float64 sum uses for
// a contiguous run of 32 or 64 values -- so the selection is bit-identical to the host's.
//
// One warp per (window, vector).  HBM-bound: K*N*4 bytes in, W*N*4 out.  The vector's 32 rows
// come into the warp's patch of shared memory by 16-byte asynchronous copies, eight (or sixteen)
// lanes per row, so that an instruction touches four (two) whole runs of 128 (256) bytes: with
// lane = row on the global loads every instruction touched 32 lines and the L1's tag look-ups were
// the bound (4096 x 11008, 4 of 32: 66 us, 2.8 TB/s of the 203 MB it moves).  Then lane = row: a lane
// adds up its row's squares, ranks them against the other 31 (broadcast shared loads), and the kept
// rows go out the way they came in.  A patch per warp and no register holds the tile, so that 32
// warps' copies are in flight on an SM.  Pruning and packing
// together, 4096 x 11008, 4 of 32: 75.8 us with the former loads, 41.1 with these (206 MB, 5.0 TB/s).
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "kernels.h"
#include "nmspmm_b200.h"

namespace nmspmm {

__device__ __forceinline__ void cp_async_16(uint32_t dst_smem, const void* src_gmem)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src_gmem) : "memory");
}

template <int VEC>
struct PruneCfg {
    static constexpr int WARPS = (VEC == 32) ? 8 : 4;
    static constexpr int PITCH = VEC * 4 + 16;               // lane = row reads 16 bytes per row without bank conflicts
    static constexpr int LANES = VEC / 4, ROWS = 32 / LANES; // lanes per row and rows per copy instruction
};

// PACK: what becomes of the indices.  0: DT as they are, one warp per unit wherever it falls.  Otherwise a CTA holds two windows
// of one index block of 128 columns and writes the packed indices itself (the packing kernels read nothing else): 1: re-tiled,
// [N / 128][W][4] (the 32-k formats); 2: the two windows' list of used columns to cinfo and every index's rank in it
// (the 64-k formats; preprocess.cu::preprocess_high_kernel).  4096 x 11008, 4 of 32, with a packing launch behind it 39.6 us
// (41.9 on another box), in one 38.3 (40.7).  What is left is this kernel's own 37 us from cold (the profiler's): 197 MB
// through DRAM at 5.3 TB/s, which is active 65 % of the time, beside the conversions to double, the ranking and
// the warps of a block that wait for one another.
template <int VEC, int PACK>
__global__ void __launch_bounds__((PruneCfg<VEC>::WARPS * 32), 5)      // shared memory has room for five, whose copies are in flight together
prune_magnitude_kernel(const float* __restrict__ dense, float* __restrict__ BT, int* __restrict__ DT, int* __restrict__ cinfo, int n_windows, int N,
                       int n_keep)
{
    using Cfg = PruneCfg<VEC>;
    constexpr int WARPS = Cfg::WARPS, PITCH = Cfg::PITCH, LANES = Cfg::LANES, ROWS = Cfg::ROWS;
    __shared__ __align__(16) unsigned char patches[WARPS][32 * PITCH];
    __shared__ __align__(16) double scores[WARPS][32];
    __shared__ int kept_rows[WARPS][32];
    __shared__ unsigned kept_masks[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nvec = N / VEC;
    constexpr int PER_BLOCK = 128 / VEC;                     // vectors per index block of 128 columns
    const int pair = blockIdx.x / (N / 128), blk = blockIdx.x - pair * (N / 128);      // (PACK)
    const long long unit = PACK ? static_cast<long long>(pair * 2 + warp / PER_BLOCK) * nvec + blk * PER_BLOCK + warp % PER_BLOCK
                                : static_cast<long long>(blockIdx.x) * WARPS + warp;
    grid_dependency_wait();
    if (unit >= static_cast<long long>(n_windows) * nvec) return;      // whole warps leave together (with lists: never)
    const int win = static_cast<int>(unit / nvec), v = static_cast<int>(unit - static_cast<long long>(win) * nvec);
    const uint32_t patch = smem_u32(patches[warp]);
    const int sub = lane / LANES, c4 = lane % LANES;
    {
        const float* src = dense + (static_cast<size_t>(win) * 32 + sub) * N + static_cast<size_t>(v) * VEC + c4 * 4;
#pragma unroll
        for (int r = 0; r < 32; r += ROWS) cp_async_16(patch + (r + sub) * PITCH + c4 * 16, src + static_cast<size_t>(r) * N);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
    // eight partial sums over elements j % 8, combined pairwise
    double r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = 0.0;
#pragma unroll
    for (int i = 0; i < VEC / 4; ++i) {
        const float4 x = lds_f4(patch + lane * PITCH + i * 16);
        const int b = (i & 1) * 4;
        r[b + 0] += static_cast<double>(x.x) * static_cast<double>(x.x);
        r[b + 1] += static_cast<double>(x.y) * static_cast<double>(x.y);
        r[b + 2] += static_cast<double>(x.z) * static_cast<double>(x.z);
        r[b + 3] += static_cast<double>(x.w) * static_cast<double>(x.w);
    }
    const double score = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
    scores[warp][lane] = score;
    __syncwarp();
    // rank among the window's 32 rows: rows with a larger score, or the same score and a lower row, come first
    int rank = 0;
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
        const double2 other = *reinterpret_cast<const double2*>(&scores[warp][j]);
        rank += (other.x > score || (other.x == score && j < lane)) ? 1 : 0;
        rank += (other.y > score || (other.y == score && j + 1 < lane)) ? 1 : 0;
    }
    const unsigned kept = __ballot_sync(0xffffffffu, rank < n_keep);
    const int pos = __popc(kept & ((1u << lane) - 1u));                // ascending row order
    // (a NaN score ranks itself first without pushing another row out: never more than n_keep rows all the same)
    const bool keep = ((kept >> lane) & 1u) && pos < n_keep;
    if (keep) {
        kept_rows[warp][pos] = lane;
        if constexpr (PACK == 0) {
            int* d = DT + (static_cast<size_t>(win) * n_keep + pos) * (N / 32) + static_cast<size_t>(v) * (VEC / 32);
#pragma unroll
            for (int h = 0; h < VEC / 32; ++h) d[h] = lane;             // one index per 32 columns (V = 64: the same twice)
        }
    }
    __syncwarp();
    const int n_out = min(__popc(kept), n_keep);
    float* dst = BT + static_cast<size_t>(win) * n_keep * N + static_cast<size_t>(v) * VEC + c4 * 4;
    for (int p = sub; p < n_out; p += ROWS)
        *reinterpret_cast<float4*>(dst + static_cast<size_t>(p) * N) = lds_f4(patch + kept_rows[warp][p] * PITCH + c4 * 16);
    // (the kept values are on their way before the warps of the block wait for one another)
    if constexpr (PACK != 0) {
        int k = lane;
        if constexpr (PACK == 2) {
            const unsigned mine = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) kept_masks[warp] = mine;
            __syncthreads();
            unsigned used[2] = { 0u, 0u };                              // of the block's vectors, per window
#pragma unroll
            for (int i = 0; i < WARPS; ++i) used[i / PER_BLOCK] |= kept_masks[i];
            const int second = warp / PER_BLOCK, first_n = __popc(used[0]);
            const unsigned below = (1u << lane) - 1u;
            k = __popc(used[second] & below) + (second ? first_n : 0);
            if (warp == 0) {
                int* list = cinfo + (static_cast<size_t>(blk) * (n_windows / 2) + pair) * 64;
                const int all = first_n + __popc(used[1]);
                if ((used[0] >> lane) & 1u) list[__popc(used[0] & below)] = lane;
                if ((used[1] >> lane) & 1u) list[first_n + __popc(used[1] & below)] = 32 + lane;
                if (lane >= all) list[lane] = -1;
                if (lane + 32 >= all) list[lane + 32] = -1;
                if (blockIdx.x == 0) {                                  // the extra window behind the last list: all -1
                    int* tail = cinfo + static_cast<size_t>(N / 128) * (n_windows / 2) * 64;
                    tail[lane] = tail[lane + 32] = -1;
                }
            }
        }
        if (keep) {
            int* d = DT + (static_cast<size_t>(blk) * n_windows * n_keep + static_cast<size_t>(win) * n_keep + pos) * 4 + (warp % PER_BLOCK) * (VEC / 32);
#pragma unroll
            for (int h = 0; h < VEC / 32; ++h) d[h] = k;
        }
    }
}

template <int VEC>
static cudaError_t launch_prune(const float* dense, float* BT, int* DT, int n_windows, int N, int n_keep, cudaStream_t st)
{
    constexpr int WARPS = PruneCfg<VEC>::WARPS;
    const long long blocks = (static_cast<long long>(n_windows) * (N / VEC) + WARPS - 1) / WARPS;
    return launch_overlapped(prune_magnitude_kernel<VEC, 0>, static_cast<unsigned>(blocks), WARPS * 32, 0, st, dense, BT, DT,
                             static_cast<int*>(nullptr), n_windows, N, n_keep);
}

template <int VEC, int PACK>
static cudaError_t launch_prune_pack(const float* dense, float* BT, int* D, int* cinfo, int n_windows, int N, int n_keep, cudaStream_t st)
{
    const unsigned blocks = static_cast<unsigned>((n_windows + 1) / 2) * static_cast<unsigned>(N / 128);
    return launch_overlapped(prune_magnitude_kernel<VEC, PACK>, blocks, PruneCfg<VEC>::WARPS * 32, 0, st, dense, BT, D, cinfo, n_windows, N, n_keep);
}

}  // namespace nmspmm

extern "C" int nmspmm_prune_device(const float* dense_dev, float* BT_dev, int* DT_dev, int K, int N, int n_keep, int vec_len,
                                   void* stream)
{
    if (!dense_dev || !BT_dev || !DT_dev) return NMSPMM_INVALID_ARGUMENT;
    if (K <= 0 || N <= 0 || K % 32 != 0 || (vec_len != 32 && vec_len != 64) || N % vec_len != 0) return NMSPMM_INVALID_ARGUMENT;
    if (n_keep < 1 || n_keep > 32) return NMSPMM_INVALID_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(dense_dev) | reinterpret_cast<uintptr_t>(BT_dev)) & 15u) return NMSPMM_INVALID_ARGUMENT;
    const long long units = static_cast<long long>(K / 32) * (N / vec_len);
    if ((units + 3) / 4 >= (1LL << 31)) return NMSPMM_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const cudaError_t e = vec_len == 32 ? nmspmm::launch_prune<32>(dense_dev, BT_dev, DT_dev, K / 32, N, n_keep, st)
                                        : nmspmm::launch_prune<64>(dense_dev, BT_dev, DT_dev, K / 32, N, n_keep, st);
    return e == cudaSuccess ? NMSPMM_OK : NMSPMM_CUDA_ERROR;
}

extern "C" int nmspmm_prune_pack_device(const float* dense_dev, float* BT_dev, int* D_dev, int* column_info_dev, int K, int N, int n_keep,
                                        int vec_len, int format, void* stream)
{
    if (!dense_dev || !BT_dev || !D_dev) return NMSPMM_INVALID_ARGUMENT;
    if (K <= 0 || N <= 0 || K % 32 != 0 || (vec_len != 32 && vec_len != 64) || N % 128 != 0) return NMSPMM_INVALID_ARGUMENT;
    if (n_keep < 1 || n_keep > 32 || (format != NMSPMM_FORMAT_LOW && format != NMSPMM_FORMAT_HIGH)) return NMSPMM_INVALID_ARGUMENT;
    if (format == NMSPMM_FORMAT_HIGH && (K % 64 != 0 || !column_info_dev)) return NMSPMM_INVALID_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(dense_dev) | reinterpret_cast<uintptr_t>(BT_dev)) & 15u) return NMSPMM_INVALID_ARGUMENT;
    if (static_cast<long long>((K / 32 + 1) / 2) * (N / 128) >= (1LL << 31)) return NMSPMM_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int n_windows = K / 32;
    cudaError_t e;
    if (format == NMSPMM_FORMAT_HIGH)
        e = vec_len == 32 ? nmspmm::launch_prune_pack<32, 2>(dense_dev, BT_dev, D_dev, column_info_dev, n_windows, N, n_keep, st)
                          : nmspmm::launch_prune_pack<64, 2>(dense_dev, BT_dev, D_dev, column_info_dev, n_windows, N, n_keep, st);
    else
        e = vec_len == 32 ? nmspmm::launch_prune_pack<32, 1>(dense_dev, BT_dev, D_dev, column_info_dev, n_windows, N, n_keep, st)
                          : nmspmm::launch_prune_pack<64, 1>(dense_dev, BT_dev, D_dev, column_info_dev, n_windows, N, n_keep, st);
    return e == cudaSuccess ? NMSPMM_OK : NMSPMM_CUDA_ERROR;
}
