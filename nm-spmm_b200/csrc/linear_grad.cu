// Backward of y = x . B for a vector-wise N:M sparse B, in FP32 like the exact forward path:
//
//     grad_B[w][n] = sum_m x[m][k(w, n/32)] grad_y[m][n]            (the kept positions only)
//     grad_x[m][k] = sum over the kept (w, n) with k(w, n/32) = k of grad_y[m][n] B[w][n]
//
// Both are 2 M N W useful FLOPs, n_keep / 32 of the dense products they replace (an expanded
// B or an M x K x N product of which most is thrown away), and both are bound by the FP32
// FMA pipe: 17.2 GFLOP at M = 2048, N = K = 4096, 8:32, against 0.1 GB of operands.  Measured
// there: grad_B 331 us (51.8 TFLOP/s of the 74 the pipe has), grad_x 372 us (46.2, two transposing passes
// included), against 1169 and 1136 us of the dense FP32 products (and 70 us of expanding B and picking the kept
// positions); at 16:32 647 and 709 us, at 4:32 207 and 235 us.
//
// The indices are the raw window-local ones, [W][N/32].  Every wait is bounded; one that
// gives up raises the device status word and nothing of its tile is stored.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"

namespace nmspmm {

struct GradArgs {
    const int* DT;          // [W][N/32] window-local k of every kept row
    const float* xq;        // grad_B: [M4/4][K][4], the rows of x in groups of four
    const float* B;         // grad_x: the launcher's (the kernel reads it through a tensor map)
    void* out;              // grad_B [W][N] float, or grad_x [M][K] of dtype
    float* partial;         // slots of split tiles
    int* status;
    int M, N, K, W;
    int tiles_x;            // tiles along the fast tile dimension
    int n_whole, slices;    // the first n_whole tiles are computed by one CTA each, the others in `slices` pieces
    int dtype;
};

template <typename T> __device__ __forceinline__ float to_float(T v);
template <> __device__ __forceinline__ float to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ void store_as(void* out, size_t at, float v, int dtype)
{
    if (dtype == kDtypeF32) static_cast<float*>(out)[at] = v;
    else if (dtype == kDtypeF16) static_cast<__half*>(out)[at] = __float2half_rn(v);
    else static_cast<__nv_bfloat16*>(out)[at] = __float2bfloat16_rn(v);
}

// Rows of x in groups of four: out[m / 4][k][m % 4], rows past M zero.  A thread reads one k of
// four rows (coalesced along k) and writes one float4 (coalesced): no shared memory.
template <typename T>
__global__ void __launch_bounds__(256) quad_rows_kernel(const T* __restrict__ x, float4* __restrict__ out, int M, int K)
{
    const size_t n = static_cast<size_t>((M + 3) / 4) * K;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int mq = static_cast<int>(i / K), k = static_cast<int>(i - static_cast<size_t>(mq) * K);
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = mq * 4 + j;
            v[j] = m < M ? to_float<T>(x[static_cast<size_t>(m) * K + k]) : 0.f;
        }
        out[i] = make_float4(v[0], v[1], v[2], v[3]);
    }
}

// ------------------------------------------------------------------------- grad of the kept values
// One CTA: RW kept rows x 128 columns (four vectors, a warp each) over a range of m.  Thread tile
// TW rows x 8 columns, eight row groups x four column groups.  A step stages MC rows of
// grad_y ([MC][128], TMA) and of x over the k range the rows come from ([MC/4][KT][4], bulk
// copies): a row's four m of one k are one 128-bit load at a k offset the thread keeps in a
// register for the whole launch, so the gather costs no index traffic.  Lanes: a 128-bit shared
// load takes one wavefront per eight lanes, and two such groups share one where lane i reads the
// address of lane i ^ 1 (the loads of x: lane bit 0 is a column bit) or of lane i ^ 2 (the loads of
// grad_y: bit 1 is a row bit).  A half warp then reads x at four unrelated k, which meet in a bank
// now and then: 2.7 wavefronts per load in all, the FMA pipe active 74 % of the time.
template <int NKEEP>
struct GradValuesCfg {
    static constexpr int TW = (NKEEP == 12) ? 6 : 8;
    static constexpr int RW = 8 * TW;
    static constexpr int KT = RW / NKEEP * 32;
    static constexpr int MC = (NKEEP == 4) ? 8 : 16;
    static constexpr int THREADS = 128;
    static constexpr int X_BYTES = MC * KT * 4, G_BYTES = MC * 128 * 4, STAGE_BYTES = X_BYTES + G_BYTES;
    static constexpr int STAGES = 3;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 128 + 128;
    static_assert(RW % NKEEP == 0, "whole windows");
};

template <int NKEEP>
__global__ void __launch_bounds__(128, 3)
nm_grad_values_kernel(const GradArgs a, const __grid_constant__ CUtensorMap map_g)
{
    using Cfg = GradValuesCfg<NKEEP>;
    constexpr int TW = Cfg::TW, RW = Cfg::RW, KT = Cfg::KT, MC = Cfg::MC, STAGES = Cfg::STAGES;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 127u) & ~127u;
    const uint32_t bars = ring + STAGES * Cfg::STAGE_BYTES, abort_word = bars + STAGES * 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ng = (lane & 1) | ((lane >> 1) & 2), wg = ((lane >> 1) & 1) | ((lane >> 2) & 6);      // see above

    const bool sliced = static_cast<int>(blockIdx.x) >= a.n_whole;
    const int S = sliced ? a.slices : 1, slot = static_cast<int>(blockIdx.x) - a.n_whole;
    const int tile = sliced ? a.n_whole + slot / S : static_cast<int>(blockIdx.x);
    const int tw = tile / a.tiles_x, tn = tile - tw * a.tiles_x;
    const int w0 = tw * RW, n0 = tn * 128, k0 = w0 / NKEEP * 32;
    const int n_steps_all = (a.M + MC - 1) / MC;
    int first, n_steps;
    slice_range(n_steps_all, S, sliced ? slot % S : 0, first, n_steps);
    const uint32_t row_bytes = static_cast<uint32_t>(min(KT, a.K - k0)) * 16u;      // one group of four m, the tile's k
    const int n_quads = (a.M + 3) / 4;

    if (tid == 0) {
        prefetch_tensor_map(&map_g);
        for (int s = 0; s < STAGES; ++s) mbar_init(bars + s * 8, 1);
        sts_volatile_s32(abort_word, 0);
        mbar_init_fence();
    }
    __syncthreads();
    grid_dependency_wait();

    auto fill = [&](int it) {                              // one thread
        const uint32_t dst = ring + (it % STAGES) * Cfg::STAGE_BYTES, full = bars + (it % STAGES) * 8;
        const int mq0 = (first + it) * (MC / 4), quads = min(MC / 4, n_quads - mq0);
        mbar_arrive_expect_tx(full, Cfg::G_BYTES + quads * row_bytes);
        for (int q = 0; q < quads; ++q)
            bulk_g2s(dst + q * (KT * 16), a.xq + (static_cast<size_t>(mq0 + q) * a.K + k0) * 4, row_bytes, full);
        tma_load_2d(dst + Cfg::X_BYTES, &map_g, n0, (first + it) * MC, full);       // rows past M arrive as zeros
    };
    if (tid == 0)
        for (int it = 0; it < STAGES - 1 && it < n_steps; ++it) fill(it);

    const int v = (n0 >> 5) + warp;                        // this warp's vector
    const bool live = v * 32 < a.N;
    int off[TW];
#pragma unroll
    for (int r = 0; r < TW; ++r) {
        const int w = w0 + wg * TW + r;
        const int k = (live && w < a.W) ? (__ldg(a.DT + static_cast<size_t>(w) * (a.N >> 5) + v) & 31) + (wg * TW + r) / NKEEP * 32 : 0;
        off[r] = k * 16;
    }
    float2 acc[TW][4];
#pragma unroll
    for (int r = 0; r < TW; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = make_float2(0.f, 0.f);

    bool alive = true;
    for (int it = 0; it < n_steps; ++it) {
        // the barrier frees the slot of the step before, which takes the step STAGES - 1 ahead
        __syncthreads();
        if (tid == 0 && it + STAGES - 1 < n_steps && alive) {
            fence_proxy_async();
            fill(it + STAGES - 1);
        }
        __syncwarp();
        const int s = it % STAGES;
        alive = __all_sync(0xffffffffu, mbar_wait_bounded(bars + s * 8, (it / STAGES) & 1, abort_word)) && alive;
        if (!live || !alive) continue;
        const uint32_t xs = ring + s * Cfg::STAGE_BYTES, gs = xs + Cfg::X_BYTES + warp * 128 + ng * 16;
        const int quads = min(MC / 4, n_quads - (first + it) * (MC / 4));       // the ragged last step holds fewer
#pragma unroll 1
        for (int q = 0; q < quads; ++q) {
            float4 x4[TW];
#pragma unroll
            for (int r = 0; r < TW; ++r) x4[r] = lds_f4(xs + q * (KT * 16) + off[r]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 g0 = lds_f4(gs + (q * 4 + j) * 512), g1 = lds_f4(gs + (q * 4 + j) * 512 + 64);
                const float2 p0 = make_float2(g0.x, g0.y), p1 = make_float2(g0.z, g0.w);
                const float2 p2 = make_float2(g1.x, g1.y), p3 = make_float2(g1.z, g1.w);
#pragma unroll
                for (int r = 0; r < TW; ++r) {
                    const float xv = j == 0 ? x4[r].x : (j == 1 ? x4[r].y : (j == 2 ? x4[r].z : x4[r].w));
                    const float2 xx = make_float2(xv, xv);
                    acc[r][0] = __ffma2_rn(xx, p0, acc[r][0]);
                    acc[r][1] = __ffma2_rn(xx, p1, acc[r][1]);
                    acc[r][2] = __ffma2_rn(xx, p2, acc[r][2]);
                    acc[r][3] = __ffma2_rn(xx, p3, acc[r][3]);
                }
            }
        }
    }
    __syncthreads();
    grid_launch_dependents();
    if (lds_volatile_s32(abort_word) != 0) {
        if (tid == 0) atomicMax(a.status, kDevTimeoutFull);
        return;
    }
    if (!live) return;
#pragma unroll
    for (int r = 0; r < TW; ++r) {
        const int w = wg * TW + r;
        if (w0 + w >= a.W) continue;
        float* p = sliced ? a.partial + (static_cast<size_t>(slot) * RW + w) * 128 + warp * 32 + ng * 4
                          : static_cast<float*>(a.out) + static_cast<size_t>(w0 + w) * a.N + n0 + warp * 32 + ng * 4;
        *reinterpret_cast<float4*>(p) = make_float4(acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y);
        *reinterpret_cast<float4*>(p + 16) = make_float4(acc[r][2].x, acc[r][2].y, acc[r][3].x, acc[r][3].y);
    }
}

// -------------------------------------------------------------------------------- grad of the input
// One CTA: MT rows x KT k of grad_x over a range of vectors.  A vector adds to n_keep of every 32
// k, a different set for every vector, so the accumulators that last are in shared memory
// ([KT][MT] floats, 128 KB) and the registers hold one vector's contribution: a warp multiplies
// 64 rows of grad_y by 32 (24) kept rows of B over the vector's 32 columns (thread tile 8 x 8, both
// operands read 128 bits along n, so the packed FMA takes its pairs from the loads as they are
// and sums even and odd columns apart), then adds the result to the rows of the accumulator
// that its index list names: 16 + 16 shared accesses of 128 bits after 1024 packed FMAs.
// Nothing is saturated: at M = 2048, N = K = 4096, 8:32 the FMA pipe is active 56 % of the time and half of the
// shared-memory wavefronts there are go by, on two warps per scheduler whose own fixed latencies are the
// largest stall.  (Thread tile 8 x 4 on sixteen warps took 481 us there.)
// A tile's last stores go out eight at a time per lane: as pairs of load and store, one after the other, they cost
// 5 % (2048 x 4096 x 4096, 4:32, 250 -> 235 us; 128 x 4096 x 4096, 8:32, 45.6 -> 42.2).
// The accumulator is what limits the warps: 32 KB of it per warp at 8:32.  At 8:32 and 4:32 two
// and four groups of warps therefore share it, each taking every second / fourth vector; a
// token per patch of the accumulator hands it from group to group in vector order, so that the
// sums have one order and the groups compute while others add.
template <int NKEEP>
struct GradInputCfg {
    static constexpr int MT = (NKEEP == 4) ? 64 : 128, KT = (NKEEP == 4) ? 512 : 256;
    static constexpr int WT = KT / 32 * NKEEP;             // kept rows under the tile
    static constexpr int TR = (NKEEP == 12) ? 6 : 8;       // kept rows per thread: a warp's 4 TR rows are whole windows
    static constexpr int MH = MT / 64, AREAS = MH * (WT / (4 * TR));
    static constexpr int GROUPS = 8 / AREAS;
    static constexpr int WARPS = AREAS * GROUPS, THREADS = WARPS * 32;
    static constexpr int G_BYTES = MT * 128, B_BYTES = WT * 128, STAGE_BYTES = G_BYTES + B_BYTES;
    static constexpr int ACC_BYTES = KT * MT * 4;
    static constexpr int STAGES = (227 * 1024 - 2048 - ACC_BYTES) / STAGE_BYTES;
    static constexpr int CTRL_BYTES = 512;
    static constexpr int SMEM_BYTES = ACC_BYTES + STAGES * STAGE_BYTES + CTRL_BYTES + 1024;
    static_assert(STAGES >= 3 && STAGES >= GROUPS, "a stage for every group at least");
    static_assert(STAGES * 12 + AREAS * GROUPS * 8 + 4 <= CTRL_BYTES, "control block");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
};

template <int NKEEP>
__global__ void __launch_bounds__((GradInputCfg<NKEEP>::THREADS), 1)
nm_grad_input_kernel(const GradArgs a, const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_b)
{
    using Cfg = GradInputCfg<NKEEP>;
    constexpr int MT = Cfg::MT, KT = Cfg::KT, MH = Cfg::MH, AREAS = Cfg::AREAS, GROUPS = Cfg::GROUPS, STAGES = Cfg::STAGES;
    constexpr int TR = Cfg::TR;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;       // 128-byte swizzle: 1024-byte alignment
    const uint32_t sums = ring + STAGES * Cfg::STAGE_BYTES;
    const uint32_t bars = sums + Cfg::ACC_BYTES, tokens = bars + STAGES * 8, reads = tokens + AREAS * GROUPS * 8;
    const uint32_t abort_word = reads + STAGES * 4;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mg = (lane >> 1) & 7, wg = (lane & 1) | ((lane >> 3) & 2);      // both operands' loads pair up (see grad_values)
    const int group = warp / AREAS, area = warp % AREAS, mh = area % MH, wq = area / MH;

    const bool sliced = static_cast<int>(blockIdx.x) >= a.n_whole;
    const int S = sliced ? a.slices : 1, slot = static_cast<int>(blockIdx.x) - a.n_whole;
    const int tile = sliced ? a.n_whole + slot / S : static_cast<int>(blockIdx.x);
    const int tm = tile / a.tiles_x, tk = tile - tm * a.tiles_x;
    const int m0 = tm * MT, k0 = tk * KT, w0 = k0 / 32 * NKEEP;
    int v0, T;                                             // this CTA's vectors: v0 .. v0 + T - 1
    slice_range(a.N >> 5, S, sliced ? slot % S : 0, v0, T);

    if (tid == 0) {
        prefetch_tensor_map(&map_g);
        prefetch_tensor_map(&map_b);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bars + s * 8, 1);
            sts_s32(reads + s * 4, 0);
        }
        for (int i = 0; i < AREAS * GROUPS; ++i) mbar_init(tokens + i * 8, 1);
        sts_volatile_s32(abort_word, 0);
        mbar_init_fence();
    }
    for (int o = tid * 16; o < Cfg::ACC_BYTES; o += Cfg::THREADS * 16) sts_f4(sums + o, make_float4(0.f, 0.f, 0.f, 0.f));
    __syncthreads();
    grid_dependency_wait();

    auto fill = [&](int t) {                               // one thread: vector v0 + t into stage t % STAGES
        const uint32_t dst = ring + (t % STAGES) * Cfg::STAGE_BYTES, full = bars + (t % STAGES) * 8;
        mbar_arrive_expect_tx(full, Cfg::STAGE_BYTES);     // rows past M or W arrive as zeros
        tma_load_2d(dst, &map_g, (v0 + t) * 32, m0, full);
        tma_load_2d(dst + Cfg::G_BYTES, &map_b, (v0 + t) * 32, w0, full);
    };
    if (tid == 0)
        for (int t = 0; t < STAGES && t < T; ++t) fill(t);

    // kept rows of this thread: wq * (4 * TR) + r * 4 + wg, so that the four row groups of a warp fall
    // into different 16-byte chunks of the swizzled rows; rows of grad_y: mh * 64 + i * 8 + mg.
    const int nv = a.N >> 5;
    const int* dt = a.DT + static_cast<size_t>(w0 + wq * (4 * TR) + wg) * nv + v0;
    auto index_of = [&](int t, int r) {                    // k within the window, -1: no such row
        return (w0 + wq * (4 * TR) + r * 4 + wg < a.W && t < T) ? (__ldg(dt + static_cast<size_t>(r * 4) * nv + t) & 31) : -1;
    };
    int k_next[TR];
#pragma unroll
    for (int r = 0; r < TR; ++r) k_next[r] = index_of(group, r);

    const uint32_t g_rel = (mh * 64 + mg) * 128, b_rel = Cfg::G_BYTES + (wq * (4 * TR) + wg) * 128;
    for (int t = group; t < T; t += GROUPS) {
        int k_of[TR];
#pragma unroll
        for (int r = 0; r < TR; ++r) {
            k_of[r] = k_next[r];
            k_next[r] = index_of(t + GROUPS, r);
        }
        const int s = t % STAGES;
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(bars + s * 8, (t / STAGES) & 1, abort_word))) break;
        const uint32_t gs = ring + s * Cfg::STAGE_BYTES + g_rel, bs = ring + s * Cfg::STAGE_BYTES + b_rel;
        float2 acc[8][TR];                                  // (even columns, odd columns)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int r = 0; r < TR; ++r) acc[i][r] = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 8; ++c) {                      // four columns at a time
            float4 b[TR];
#pragma unroll
            for (int r = 0; r < TR; ++r) b[r] = lds_f4(bs + r * 512 + ((c ^ (((wq * TR + r) & 1) * 4 + wg)) << 4));
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 g = lds_f4(gs + i * 1024 + ((c ^ mg) << 4));
#pragma unroll
                for (int r = 0; r < TR; ++r) acc[i][r] = __ffma2_rn(make_float2(g.x, g.y), make_float2(b[r].x, b[r].y), acc[i][r]);
#pragma unroll
                for (int r = 0; r < TR; ++r) acc[i][r] = __ffma2_rn(make_float2(g.z, g.w), make_float2(b[r].z, b[r].w), acc[i][r]);
            }
        }
        // the stage has been read by this warp; the last warp to say so refills it
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            unsigned old;
            asm volatile("atom.shared.add.u32 %0, [%1], 1;" : "=r"(old) : "r"(reads + s * 4) : "memory");
            if (old == static_cast<unsigned>(AREAS * (t / STAGES + 1) - 1) && t + STAGES < T) {
                __threadfence_block();
                fence_proxy_async();
                fill(t + STAGES);
            }
        }
        __syncwarp();
        // this patch of the accumulator, after the vector before has been added to it
        if (GROUPS > 1 && t > 0) {
            const int from = (t - 1) % GROUPS;
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(tokens + (area * GROUPS + from) * 8, ((t - 1) / GROUPS) & 1, abort_word))) break;
        }
        if (GROUPS == 1) __syncwarp();
#pragma unroll
        for (int r = 0; r < TR; ++r) {
            if (k_of[r] >= 0) {
                const int k = (wq * (4 * TR) + r * 4 + wg) / NKEEP * 32 + k_of[r];
                const uint32_t p = sums + k * (MT * 4) + mh * 256 + ((mg ^ (k & 7)) << 4);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float4 x = lds_f4(p + h * 128);
                    x.x += acc[4 * h][r].x + acc[4 * h][r].y;
                    x.y += acc[4 * h + 1][r].x + acc[4 * h + 1][r].y;
                    x.z += acc[4 * h + 2][r].x + acc[4 * h + 2][r].y;
                    x.w += acc[4 * h + 3][r].x + acc[4 * h + 3][r].y;
                    sts_f4(p + h * 128, x);
                }
            }
        }
        __syncwarp();
        if (GROUPS > 1 && lane == 0) mbar_arrive(tokens + (area * GROUPS + group) * 8);
    }
    __syncthreads();
    grid_launch_dependents();
    if (lds_volatile_s32(abort_word) != 0) {
        if (tid == 0) atomicMax(a.status, kDevTimeoutFull);
        return;
    }
    // a warp per row of the tile, lanes along k (four lanes of a load meet in a bank), eight loads in flight
    for (int m = warp; m < MT; m += Cfg::WARPS) {
        if (m0 + m >= a.M) continue;
        const int h = (m >> 5) & 1, x = (m >> 3) & 3;      // i = (m % 64) / 8 = 4 h + x
#pragma unroll 1
        for (int kk = 0; kk < KT; kk += 256) {
            float val[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int k = kk + lane + i * 32;
                val[i] = __uint_as_float(lds_u32(sums + k * (MT * 4) + (m >> 6) * 256 + h * 128 + (((m & 7) ^ (k & 7)) << 4) + x * 4));
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int k = kk + lane + i * 32;
                if (k0 + k >= a.K) break;
                if (sliced) a.partial[(static_cast<size_t>(slot) * MT + m) * KT + k] = val[i];
                else store_as(a.out, static_cast<size_t>(m0 + m) * a.K + k0 + k, val[i], a.dtype);
            }
        }
    }
}

// ------------------------------------------------------------- grad of the input, larger problems
// The same sum with the register tile of the exact forward path (gemm_ffma_wide.cuh): 16 rows x 8 (6) kept rows
// a thread, the packed FMA's pairs along m.  That wants both operands with n outermost, grad_y as
// [N][m] and B as [N][W]: two transposing passes ahead (20 us at M = 2048, N = K = 4096), after which a column of a
// vector costs six 128-bit shared loads per 64 packed FMAs (eight per 64 above, on half as many rows and kept rows).
// A warp multiplies 128 rows by 32 (24) kept rows over a vector's 32 columns and adds the result to the accumulator
// in shared memory, 64 accesses of 128 bits after 2048 packed FMAs (32 after 1024 above, a quarter of the vectors
// later: groups of warps take the vectors in turn and hand the accumulator on in vector order).  A warpgroup
// of 40 registers feeds each group through a ring of its own, sixteen columns a stage.
// Bound by the FMA pipe, active 72 % of the time, its shared loads and the hand-overs: M = 2048, N = K = 4096, 12:32 and 8:32,
// 672 and 455 us -> 552 and 372 with everything (340 of them this kernel at 8:32), 16:32 852 -> 709.
template <int NKEEP>
struct GradInputWideCfg {
    static constexpr int MT = 128, KT = 256, WT = KT / 32 * NKEEP;
    static constexpr int TR = (NKEEP == 12) ? 6 : 8, WROWS = 4 * TR;       // kept rows per thread / per warp: whole windows
    static constexpr int AREAS = WT / WROWS, GROUPS = 8 / AREAS;
    static constexpr int QN = 16, CHUNKS = 32 / QN;        // columns per stage
    static constexpr int A_BYTES = QN * MT * 4, B_BYTES = QN * WT * 4, STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int ACC_BYTES = KT * MT * 4;
    static constexpr int SPG = (227 * 1024 - 2048 - ACC_BYTES) / STAGE_BYTES / GROUPS;      // stages per group
    static constexpr int STAGES = SPG * GROUPS;
    static constexpr int CTRL_BYTES = 1024;
    static constexpr int SMEM_BYTES = ACC_BYTES + STAGES * STAGE_BYTES + CTRL_BYTES + 1024;
    static constexpr int THREADS = 384;
    static constexpr int LAUNCH_REGS = 168, COMPUTE_REGS = 232, FEED_REGS = 40;
    static_assert(2 * COMPUTE_REGS + FEED_REGS == 3 * LAUNCH_REGS, "the warpgroups share what the launch was given");
    static_assert(WT % WROWS == 0 && WROWS % NKEEP == 0 && AREAS * GROUPS == 8 && (GROUPS == 2 || GROUPS == 4) && SPG >= 2, "eight warps");
    static_assert(STAGES * 16 + 64 + 8 <= CTRL_BYTES && SMEM_BYTES <= 227 * 1024, "shared memory");
};

template <int NKEEP>
__global__ void __launch_bounds__((GradInputWideCfg<NKEEP>::THREADS), 1)
nm_grad_input_wide_kernel(const GradArgs a, const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_b)
{
    using Cfg = GradInputWideCfg<NKEEP>;
    constexpr int MT = Cfg::MT, KT = Cfg::KT, WT = Cfg::WT, TR = Cfg::TR, WROWS = Cfg::WROWS, AREAS = Cfg::AREAS, GROUPS = Cfg::GROUPS;
    constexpr int QN = Cfg::QN, CHUNKS = Cfg::CHUNKS, SPG = Cfg::SPG;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t sums = (smem_u32(smem_raw) + 1023u) & ~1023u, ring = sums + Cfg::ACC_BYTES;
    const uint32_t full = ring + Cfg::STAGES * Cfg::STAGE_BYTES, empty = full + Cfg::STAGES * 8, tokens = empty + Cfg::STAGES * 8;
    const uint32_t abort_word = tokens + 64;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const bool sliced = static_cast<int>(blockIdx.x) >= a.n_whole;
    const int S = sliced ? a.slices : 1, slot = static_cast<int>(blockIdx.x) - a.n_whole;
    const int tile = sliced ? a.n_whole + slot / S : static_cast<int>(blockIdx.x);
    const int tm = tile / a.tiles_x, tk = tile - tm * a.tiles_x;
    const int m0 = tm * MT, k0 = tk * KT, w0 = k0 / 32 * NKEEP;
    int v0, T;                                             // this CTA's vectors: v0 .. v0 + T - 1
    slice_range(a.N >> 5, S, sliced ? slot % S : 0, v0, T);

    if (tid == 0) {
        prefetch_tensor_map(&map_g);
        prefetch_tensor_map(&map_b);
        for (int s = 0; s < Cfg::STAGES; ++s) {
            mbar_init(full + s * 8, 1);
            mbar_init(empty + s * 8, AREAS);
        }
        for (int i = 0; i < 8; ++i) mbar_init(tokens + i * 8, 1);
        sts_volatile_s32(abort_word, 0);
        mbar_init_fence();
    }
    for (int o = tid * 16; o < Cfg::ACC_BYTES; o += Cfg::THREADS * 16) sts_f4(sums + o, make_float4(0.f, 0.f, 0.f, 0.f));
    __syncthreads();
    grid_dependency_wait();

    if (warp >= 8) {
        // ------------------------------------------------ copies: warp 8 + f feeds group f (of two or four)
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::FEED_REGS));
        if (elect_one()) {
            bool ok = true;
            for (int r = 0; ok && r * GROUPS < T; ++r) {
                for (int h = 0; ok && h < CHUNKS; ++h) {
                    const int g = warp - 8, t = r * GROUPS + g;
                    if (g >= GROUPS || t >= T) break;
                    const int c = r * CHUNKS + h, s = g * SPG + c % SPG;
                    if (c >= SPG) ok = mbar_sleep_bounded(empty + s * 8, (c / SPG - 1) & 1, abort_word);
                    if (!ok) break;
                    const uint32_t st = ring + s * Cfg::STAGE_BYTES;
                    mbar_arrive_expect_tx(full + s * 8, Cfg::STAGE_BYTES);         // rows past M or W arrive as zeros
                    tma_load_2d(st, &map_g, m0, (v0 + t) * 32 + h * QN, full + s * 8);
                    tma_load_2d(st + Cfg::A_BYTES, &map_b, w0, (v0 + t) * 32 + h * QN, full + s * 8);
                }
            }
            if (!ok) atomicMax(a.status, kDevTimeoutEmpty);
        }
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::COMPUTE_REGS));

    // Lanes as in gemm_ffma_wide.cuh: rows lm * 4 + 32 j .. + 3 (j < 4) of the tile, kept rows lw * 4 .. + 3 and 16 + lw * 4 .. + 3
    // (12:32: 16 + lw * 2, + 1) of the warp's.
    const int group = warp / AREAS, area = warp % AREAS;
    const int lm = (lane >> 1) & 7, lw = (lane & 1) | ((lane >> 3) & 2);
    const int nv = a.N >> 5;
    const uint32_t a_rel = lm * 16, b_rel = Cfg::A_BYTES + (area * WROWS + lw * 4) * 4;
    const uint32_t b_rel2 = (TR == 8) ? b_rel + 64 : Cfg::A_BYTES + (area * WROWS + 16 + lw * 2) * 4;
    // lane p keeps the place in the accumulator of the warp's p-th kept row, -1: there is none
    const int wp = w0 + area * WROWS + lane;
    const bool has = lane < WROWS && wp < a.W;
    const int* dt = a.DT + static_cast<size_t>(has ? wp : 0) * nv + v0;
    auto place_of = [&](int t) { return has && t < T ? (area * WROWS + lane) / NKEEP * 32 + (__ldg(dt + t) & 31) : -1; };

    float x[2][16], y[2][TR];
    auto load = [&](int buf, uint32_t st, int n) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 v = lds_f4(st + a_rel + n * (MT * 4) + j * 128);
            x[buf][4 * j] = v.x; x[buf][4 * j + 1] = v.y; x[buf][4 * j + 2] = v.z; x[buf][4 * j + 3] = v.w;
        }
        const float4 u = lds_f4(st + b_rel + n * (WT * 4));
        y[buf][0] = u.x; y[buf][1] = u.y; y[buf][2] = u.z; y[buf][3] = u.w;
        if constexpr (TR == 8) {
            const float4 w = lds_f4(st + b_rel2 + n * (WT * 4));
            y[buf][4] = w.x; y[buf][5] = w.y; y[buf][6] = w.z; y[buf][7] = w.w;
        } else {
            const float2 w = lds_f2(st + b_rel2 + n * (WT * 4));
            y[buf][4] = w.x; y[buf][5] = w.y;
        }
    };

    int s = 0;                                             // stage of the group's ring, and the parity of its next wait
    uint32_t parity = 0;
    int next = place_of(group);
    bool alive = true;
    auto wait_full = [&]() { return __all_sync(0xffffffffu, mbar_wait_bounded(full + (group * SPG + s) * 8, parity, abort_word)) != 0; };
    for (int t = group; alive && t < T; t += GROUPS) {
        const int place = next;
        next = place_of(t + GROUPS);
        float2 acc[8][TR];                                 // (rows 2 i, 2 i + 1) x kept row
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int r = 0; r < TR; ++r) acc[i][r] = make_float2(0.f, 0.f);
        alive = wait_full();
        if (!alive) break;
        load(0, ring + (group * SPG + s) * Cfg::STAGE_BYTES, 0);
#pragma unroll 1
        for (int h = 0; h < CHUNKS; ++h) {
            const int sc = s;
            const uint32_t st = ring + (group * SPG + sc) * Cfg::STAGE_BYTES;
            if (++s == SPG) { s = 0; parity ^= 1; }
#pragma unroll
            for (int n = 0; n < QN; ++n) {
                if (n == QN - 2 && h + 1 < CHUNKS) alive = wait_full() && alive;
                if (n + 1 < QN) load((n + 1) & 1, st, n + 1);
                else load(0, ring + (group * SPG + s) * Cfg::STAGE_BYTES, 0);      // (after the last chunk: read once, not used)
#pragma unroll
                for (int r = 0; r < TR; ++r) {
                    const float2 yy = make_float2(y[n & 1][r], y[n & 1][r]);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int q = (r & 1) ? 7 - i : i;
                        acc[q][r] = __ffma2_rn(make_float2(x[n & 1][2 * q], x[n & 1][2 * q + 1]), yy, acc[q][r]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + (group * SPG + sc) * 8);
        }
        // this patch of the accumulator, after the vector before has been added to it
        if (t > 0)
            alive = __all_sync(0xffffffffu, mbar_wait_bounded(tokens + (area * GROUPS + (t - 1) % GROUPS) * 8, ((t - 1) / GROUPS) & 1, abort_word)) && alive;
        if (!alive) break;
#pragma unroll
        for (int r0 = 0; r0 < TR; r0 += 2) {               // two kept rows at a time: eight loads in flight
            float4 v[2][4];
            uint32_t p[2];
            bool there[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int r = r0 + q, k = __shfl_sync(0xffffffffu, place, r < 4 ? lw * 4 + r : (TR == 8 ? 16 + lw * 4 + r - 4 : 16 + lw * 2 + r - 4));
                there[q] = k >= 0;
                p[q] = sums + (there[q] ? k : 0) * (MT * 4) + ((lm ^ (k & 7)) << 4);
#pragma unroll
                for (int j = 0; j < 4; ++j) v[q][j] = lds_f4(p[q] + j * 128);
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (there[q]) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 lo = acc[2 * j][r0 + q], hi = acc[2 * j + 1][r0 + q];
                        sts_f4(p[q] + j * 128, make_float4(v[q][j].x + lo.x, v[q][j].y + lo.y, v[q][j].z + hi.x, v[q][j].w + hi.y));
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(tokens + (area * GROUPS + group) * 8);
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    grid_launch_dependents();
    if (lds_volatile_s32(abort_word) != 0) {
        if (tid == 0) atomicMax(a.status, kDevTimeoutFull);
        return;
    }
    // a warp per row of the tile, lanes along k (four lanes of a load meet in a bank), eight loads in flight
    for (int m = warp; m < MT; m += 8) {
        if (m0 + m >= a.M) continue;
        float val[KT / 32];
#pragma unroll
        for (int i = 0; i < KT / 32; ++i) {
            const int k = lane + i * 32;
            val[i] = __uint_as_float(lds_u32(sums + k * (MT * 4) + (m >> 5) * 128 + ((((m >> 2) & 7) ^ (k & 7)) << 4) + (m & 3) * 4));
        }
#pragma unroll
        for (int i = 0; i < KT / 32; ++i) {
            const int k = lane + i * 32;
            if (k0 + k >= a.K) break;
            if (sliced) a.partial[(static_cast<size_t>(slot) * MT + m) * KT + k] = val[i];
            else store_as(a.out, static_cast<size_t>(m0 + m) * a.K + k0 + k, val[i], a.dtype);
        }
    }
}

// Adds the slices of split tiles (slots of rows x cols floats, one after the other) in order and
// writes the elements that exist.  One float4 per thread.
__global__ void __launch_bounds__(256) nm_grad_reduce_kernel(const GradArgs a, int rows, int cols, int out_rows, int out_cols)
{
    const int per_row = cols / 4, ctas = (rows * per_row + 255) / 256;
    const int i = blockIdx.x / ctas, e = (blockIdx.x - i * ctas) * 256 + threadIdx.x;
    const int tile = a.n_whole + i, ty = tile / a.tiles_x, tx = tile - ty * a.tiles_x;
    const int r = e / per_row, c = (e - r * per_row) * 4;
    grid_dependency_wait();
    if (*reinterpret_cast<volatile int*>(a.status) != 0) return;       // a wait gave up: the slices are incomplete
    if (r >= rows || ty * rows + r >= out_rows || tx * cols + c >= out_cols) return;
    const float4* src = reinterpret_cast<const float4*>(a.partial + (static_cast<size_t>(i) * a.slices * rows + r) * cols + c);
    const size_t step = static_cast<size_t>(rows) * cols / 4;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int z = 0; z < a.slices; z += 4) {
        float4 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (z + u < a.slices) x[u] = __ldcg(src + (z + u) * step);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (z + u < a.slices) { sum.x += x[u].x; sum.y += x[u].y; sum.z += x[u].z; sum.w += x[u].w; }
    }
    const size_t at = static_cast<size_t>(ty * rows + r) * out_cols + tx * cols + c;
    if (a.dtype == kDtypeF32) {
        *reinterpret_cast<float4*>(static_cast<float*>(a.out) + at) = sum;
    } else {
        store_as(a.out, at, sum.x, a.dtype);
        store_as(a.out, at + 1, sum.y, a.dtype);
        store_as(a.out, at + 2, sum.z, a.dtype);
        store_as(a.out, at + 3, sum.w, a.dtype);
    }
}

// ---------------------------------------------------------------------------------------- host side
// How a grid of equal tiles over `steps` contraction steps is cut: whole tiles while they fill
// rounds of `slots` CTAs, the rest in S slices each.  S minimises the rounds of the rest, in
// units of a whole tile, plus what a slice costs besides (its scratch slot written and read back
// by the reduction: `slot_cost`, as a share of a tile's time).
static void cut_tiles(int tiles, int slots, int steps, int least_steps, double slot_cost, int* whole, int* slices)
{
    *whole = tiles / slots * slots;
    const int rest = tiles - *whole;
    *slices = 1;
    if (rest == 0) return;
    double best = 1.0;
    for (int s = 2; s <= 32 && steps / s >= least_steps; ++s) {
        const long long ctas = static_cast<long long>(rest) * s;
        const double cost = static_cast<double>((ctas + slots - 1) / slots) / s + slot_cost * (static_cast<double>(ctas) / slots);
        if (cost < best * 0.98) {
            best = cost;
            *slices = s;
        }
    }
    if (*slices == 1) *whole = tiles;
}

struct GradPlan {
    int tiles_x = 0, tiles = 0, whole = 0, slices = 1, rows = 0, cols = 0;
    size_t partial_floats() const { return slices > 1 ? static_cast<size_t>(tiles - whole) * slices * rows * cols : 0; }
    int ctas() const { return whole + (tiles - whole) * slices; }
};

template <int NKEEP>
static GradPlan plan_values(int M, int N, int W, int sms)
{
    using Cfg = GradValuesCfg<NKEEP>;
    GradPlan p;
    p.rows = Cfg::RW;
    p.cols = 128;
    p.tiles_x = (N + 127) / 128;
    p.tiles = p.tiles_x * ((W + Cfg::RW - 1) / Cfg::RW);
    cut_tiles(p.tiles, sms * 3, (M + Cfg::MC - 1) / Cfg::MC, 4, 10.0 / (M > 10 ? M : 10), &p.whole, &p.slices);
    return p;
}

template <int NKEEP>
static GradPlan plan_input(int M, int N, int K, int sms)
{
    using Cfg = GradInputCfg<NKEEP>;
    GradPlan p;
    p.rows = Cfg::MT;
    p.cols = Cfg::KT;
    p.tiles_x = (K + Cfg::KT - 1) / Cfg::KT;
    p.tiles = p.tiles_x * ((M + Cfg::MT - 1) / Cfg::MT);
    cut_tiles(p.tiles, sms, N / 32, 4, 4.0 / (N / 32 > 4 ? N / 32 : 4), &p.whole, &p.slices);
    return p;
}

template <int NKEEP>
static GradPlan plan_input_wide(int M, int N, int K, int sms)
{
    using Cfg = GradInputWideCfg<NKEEP>;
    GradPlan p;
    p.rows = Cfg::MT;
    p.cols = Cfg::KT;
    p.tiles_x = (K + Cfg::KT - 1) / Cfg::KT;
    p.tiles = p.tiles_x * ((M + Cfg::MT - 1) / Cfg::MT);
    cut_tiles(p.tiles, sms, N / 32, 8, 4.0 / (N / 32 > 4 ? N / 32 : 4), &p.whole, &p.slices);
    return p;
}

// About how long the input's gradient takes on a plan, in microseconds: the launches, the products of the busiest SM (at
// the FMA peak of one, 128 a cycle at 1.965 GHz, times what the kernel takes of it: 55 % / 68 %), the slices' way through
// scratch and, for the larger register tiles, the two transposing passes.
static double input_us(const GradPlan& p, bool wide, int M, int N, int K, int n_keep, int sms)
{
    const long long cut = static_cast<long long>(p.tiles - p.whole) * p.slices;
    const double rounds = (p.whole + sms - 1) / sms + (p.tiles > p.whole ? static_cast<double>((cut + sms - 1) / sms) / p.slices : 0.0);
    const double slowdown = wide ? 1.47 : (n_keep == 8 ? 1.83 : (n_keep == 12 ? 1.74 : 1.75));
    double us = (wide ? 17.3 : 12.1) + slowdown * rounds * (p.cols / 32 * n_keep) * N * p.rows / (128 * 1965.0);
    if (p.slices > 1) us += (wide ? 0.5 : 1.9) + 0.16e-6 * 8.0 * cut * p.rows * p.cols;
    if (wide) us += 0.107e-6 * 8.0 * N * (M + K / 32 * static_cast<double>(n_keep));
    return us;
}

// Whether the input's gradient takes the larger register tiles and the two transposing passes ahead of them: not at
// 4:32, where one warp holds a vector's kept rows and eight in turn on one patch of the accumulator wait for one
// another (2048 x 4096 x 4096: 250 -> 275 us), and elsewhere where they are 2 % under the smaller tiles by the times
// above: least squares over 120 shapes measured both ways (64 to 8192 rows, 20 to 850 us, each time within 11 %).  On 120
// other shapes it takes 71, which are 1.10 times as fast in the mean, the slowest of them 0.974; the best of those it leaves would be
// 1.013.  Few rows lose what transposing B costs (100 x 4224 x 4992, 12:32, 69.6 -> 74.8 us; 128 x 17792 x 9920, 16:32, 591 -> 630).
static bool wide_input_pays(int M, int N, int K, int n_keep, int sms)
{
    switch (n_keep) {
    case 16: return 1.02 * input_us(plan_input_wide<16>(M, N, K, sms), true, M, N, K, 16, sms) < input_us(plan_input<16>(M, N, K, sms), false, M, N, K, 16, sms);
    case 12: return 1.02 * input_us(plan_input_wide<12>(M, N, K, sms), true, M, N, K, 12, sms) < input_us(plan_input<12>(M, N, K, sms), false, M, N, K, 12, sms);
    case 8: return 1.02 * input_us(plan_input_wide<8>(M, N, K, sms), true, M, N, K, 8, sms) < input_us(plan_input<8>(M, N, K, sms), false, M, N, K, 8, sms);
    default: return false;
    }
}

static size_t transposed_floats(int rows, int cols) { return static_cast<size_t>((rows + 3) / 4 * 4) * cols; }     // [cols][rows up to a multiple of 4]

// Once per device: the kernel's shared memory and, where its warpgroups share out registers, that the launch is given
// as many a thread as the shares add up to (less of it and they would wait).
template <typename Kernel>
static cudaError_t allow_smem(Kernel kernel, int bytes, bool* configured, int launch_regs = 0)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev >= 64 || configured[dev]) return e;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && launch_regs > 0) {
        cudaFuncAttributes fa;
        e = cudaFuncGetAttributes(&fa, kernel);
        if (e == cudaSuccess && fa.numRegs < launch_regs) e = cudaErrorInvalidKernelImage;
    }
    if (e == cudaSuccess) configured[dev] = true;
    return e;
}

static cudaError_t launch_quad_rows(int dtype, const void* x, float* out, int M, int K, cudaStream_t st)
{
    const size_t n = static_cast<size_t>((M + 3) / 4) * K, want = (n + 255) / 256;
    const unsigned blocks = static_cast<unsigned>(want < 148 * 32 ? want : 148 * 32);
    float4* o = reinterpret_cast<float4*>(out);
    if (dtype == kDtypeF32) quad_rows_kernel<float><<<blocks, 256, 0, st>>>(static_cast<const float*>(x), o, M, K);
    else if (dtype == kDtypeF16) quad_rows_kernel<__half><<<blocks, 256, 0, st>>>(static_cast<const __half*>(x), o, M, K);
    else quad_rows_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(x), o, M, K);
    return cudaGetLastError();
}

static cudaError_t launch_grad_reduce(const GradArgs& a, const GradPlan& p, int out_rows, int out_cols, cudaStream_t st)
{
    const int ctas = (p.rows * p.cols / 4 + 255) / 256;
    return launch_overlapped(nm_grad_reduce_kernel, (p.tiles - p.whole) * ctas, 256, 0, st, a, p.rows, p.cols, out_rows, out_cols);
}

template <int NKEEP>
static cudaError_t launch_values(GradArgs a, const GradPlan& p, const float* grad_y, cudaStream_t st)
{
    using Cfg = GradValuesCfg<NKEEP>;
    static bool configured[64] = {};
    cudaError_t e = allow_smem(nm_grad_values_kernel<NKEEP>, Cfg::SMEM_BYTES, configured);
    if (e != cudaSuccess) return e;
    CUtensorMap map_g;
    e = encode_tensor_map_2d(&map_g, grad_y, a.N, a.M, 128, Cfg::MC, 0);
    if (e != cudaSuccess) return e;
    a.tiles_x = p.tiles_x;
    a.n_whole = p.whole;
    a.slices = p.slices;
    a.dtype = kDtypeF32;
    e = launch_overlapped(nm_grad_values_kernel<NKEEP>, p.ctas(), Cfg::THREADS, Cfg::SMEM_BYTES, st, a, map_g);
    if (e == cudaSuccess && p.slices > 1) e = launch_grad_reduce(a, p, a.W, a.N, st);
    return e;
}

template <int NKEEP>
static cudaError_t launch_input(GradArgs a, const GradPlan& p, const float* grad_y, cudaStream_t st)
{
    using Cfg = GradInputCfg<NKEEP>;
    static bool configured[64] = {};
    cudaError_t e = allow_smem(nm_grad_input_kernel<NKEEP>, Cfg::SMEM_BYTES, configured);
    if (e != cudaSuccess) return e;
    CUtensorMap map_g, map_b;
    e = encode_tensor_map_2d(&map_g, grad_y, a.N, a.M, 32, Cfg::MT, 2);
    if (e != cudaSuccess) return e;
    e = encode_tensor_map_2d(&map_b, a.B, a.N, a.W, 32, Cfg::WT, 2);
    if (e != cudaSuccess) return e;
    a.tiles_x = p.tiles_x;
    a.n_whole = p.whole;
    a.slices = p.slices;
    e = launch_overlapped(nm_grad_input_kernel<NKEEP>, p.ctas(), Cfg::THREADS, Cfg::SMEM_BYTES, st, a, map_g, map_b);
    if (e == cudaSuccess && p.slices > 1) e = launch_grad_reduce(a, p, a.M, a.K, st);
    return e;
}

template <int NKEEP>
static cudaError_t launch_input_wide(GradArgs a, const GradPlan& p, const float* grad_y, float* scratch, cudaStream_t st)
{
    using Cfg = GradInputWideCfg<NKEEP>;
    static bool configured[64] = {};
    cudaError_t e = allow_smem(nm_grad_input_wide_kernel<NKEEP>, Cfg::SMEM_BYTES, configured, Cfg::LAUNCH_REGS);
    if (e != cudaSuccess) return e;
    const int ldm = (a.M + 3) / 4 * 4, ldw = (a.W + 3) / 4 * 4;
    float* g_cols = scratch;
    float* b_cols = g_cols + transposed_floats(a.M, a.N);
    a.partial = b_cols + transposed_floats(a.W, a.N);
    e = launch_transpose_rows(kDtypeF32, grad_y, g_cols, a.M, a.N, ldm, st);
    if (e == cudaSuccess) e = launch_transpose_rows(kDtypeF32, a.B, b_cols, a.W, a.N, ldw, st);
    if (e != cudaSuccess) return e;
    CUtensorMap map_g, map_b;
    e = encode_tensor_map_2d(&map_g, g_cols, ldm, a.N, Cfg::MT, Cfg::QN);
    if (e != cudaSuccess) return e;
    e = encode_tensor_map_2d(&map_b, b_cols, ldw, a.N, Cfg::WT, Cfg::QN);
    if (e != cudaSuccess) return e;
    a.tiles_x = p.tiles_x;
    a.n_whole = p.whole;
    a.slices = p.slices;
    e = launch_overlapped(nm_grad_input_wide_kernel<NKEEP>, p.ctas(), Cfg::THREADS, Cfg::SMEM_BYTES, st, a, map_g, map_b);
    if (e == cudaSuccess && p.slices > 1) e = launch_grad_reduce(a, p, a.M, a.K, st);
    return e;
}

#define NMSPMM_BY_RATIO(call)                       \
    switch (n_keep) {                               \
    case 16: return call(16);                       \
    case 12: return call(12);                       \
    case 8: return call(8);                         \
    case 4: return call(4);                         \
    default: break;                                 \
    }

bool linear_grad_supported(int n_keep) { return n_keep == 16 || n_keep == 12 || n_keep == 8 || n_keep == 4; }

size_t grad_values_scratch_bytes(int M, int N, int K, int n_keep, int sms)
{
    const size_t quads = static_cast<size_t>((M + 3) / 4) * 4 * K;
    const int W = K / 32 * n_keep;
#define NMSPMM_CALL(R) (quads + plan_values<R>(M, N, W, sms).partial_floats()) * sizeof(float)
    NMSPMM_BY_RATIO(NMSPMM_CALL)
#undef NMSPMM_CALL
    return 0;
}

size_t grad_input_scratch_bytes(int M, int N, int K, int n_keep, int sms)
{
    if (wide_input_pays(M, N, K, n_keep, sms)) {
        const GradPlan p = n_keep == 16 ? plan_input_wide<16>(M, N, K, sms) : (n_keep == 12 ? plan_input_wide<12>(M, N, K, sms) : plan_input_wide<8>(M, N, K, sms));
        return (transposed_floats(M, N) + transposed_floats(K / 32 * n_keep, N) + p.partial_floats()) * sizeof(float);
    }
#define NMSPMM_CALL(R) plan_input<R>(M, N, K, sms).partial_floats() * sizeof(float)
    NMSPMM_BY_RATIO(NMSPMM_CALL)
#undef NMSPMM_CALL
    return 0;
}

cudaError_t launch_grad_values(int dtype, const void* x, const float* grad_y, const int* DT, float* grad_B, int M, int N, int K,
                               int n_keep, int sms, float* scratch, int* status, cudaStream_t st)
{
    cudaError_t e = launch_quad_rows(dtype, x, scratch, M, K, st);
    if (e != cudaSuccess) return e;
    GradArgs a {};
    a.DT = DT;
    a.xq = scratch;
    a.out = grad_B;
    a.partial = scratch + static_cast<size_t>((M + 3) / 4) * 4 * K;
    a.status = status;
    a.M = M; a.N = N; a.K = K; a.W = K / 32 * n_keep;
#define NMSPMM_CALL(R) launch_values<R>(a, plan_values<R>(M, N, a.W, sms), grad_y, st)
    NMSPMM_BY_RATIO(NMSPMM_CALL)
#undef NMSPMM_CALL
    return cudaErrorInvalidValue;
}

cudaError_t launch_grad_input(int dtype, const float* grad_y, const float* B, const int* DT, void* grad_x, int M, int N, int K,
                              int n_keep, int sms, float* scratch, int* status, cudaStream_t st)
{
    GradArgs a {};
    a.DT = DT;
    a.B = B;
    a.out = grad_x;
    a.partial = scratch;
    a.status = status;
    a.dtype = dtype;
    a.M = M; a.N = N; a.K = K; a.W = K / 32 * n_keep;
    if (wide_input_pays(M, N, K, n_keep, sms)) {
        switch (n_keep) {
        case 16: return launch_input_wide<16>(a, plan_input_wide<16>(M, N, K, sms), grad_y, scratch, st);
        case 12: return launch_input_wide<12>(a, plan_input_wide<12>(M, N, K, sms), grad_y, scratch, st);
        case 8: return launch_input_wide<8>(a, plan_input_wide<8>(M, N, K, sms), grad_y, scratch, st);
        default: return cudaErrorInvalidValue;
        }
    }
#define NMSPMM_CALL(R) launch_input<R>(a, plan_input<R>(M, N, K, sms), grad_y, st)
    NMSPMM_BY_RATIO(NMSPMM_CALL)
#undef NMSPMM_CALL
    return cudaErrorInvalidValue;
}

}  // namespace nmspmm
