// Exact-FP32 vector-wise N:M sparse GEMM for sm_100a, large tiles: one CTA per SM, eight
// compute warps of 16 x 8 register tiles and a warpgroup that feeds them.
//
// The schedule (units, ranges, pieces, scratch slots) is that of gemm_args.h, as in
// gemm_ffma.cuh; what differs is how a window gets through the SM:
//   * A warp's tile is 128 rows x one 32-column vector, or 64 rows x two vectors: a thread
//     holds 16 rows x 8 columns (128 accumulators), so a kept row costs six 128-bit shared
//     loads per 64 packed FMAs instead of four per 32, and the packed FMA takes its pairs along
//     m, straight out of the loads of A, with the eight values of B duplicated (pairs along n,
//     sixteen values of A duplicated: 4 - 6 % slower).
//   * No CTA barrier in the loop.  Every stage has a barrier that says it is full and one that
//     says every compute warp has read it; a warp reaches into its next window -- waits for
//     it, fetches its first rows and operands -- while it multiplies the last kept
//     rows of this one, so nothing of a window's start is exposed.
//   * One warp issues the copies, three resolve the window's indices (through column_info
//     on the 64-k format) to shared addresses of rows of A, [vector][kept row]; a compute warp
//     reads four of them per 128-bit load.  Their warpgroup gives its registers up to the
//     compute warps: 168 a thread at launch, 40 and 232 from then on.  They share the
//     schedulers with compute warps: with a division per window and one resolving warp the
//     same multiply took 3 % longer.
// Bound by the FMA pipe.  The 128 x 128 kernel loses the time of about four kept rows per window to its
// barrier, waits and look-ups (82 / 78 / 75 / 62 % of the 74.1 TFLOP/s peak at 16 / 12 / 8 / 4 of 32, 4096 cubed); this one runs
// at 85 / 82 / 82 / 74 %, of the 88 % that the inner loop reaches alone (its loads take register
// ports from the FMAs).  What is left between the two is the waits and loop ends of a window (6 % at 8:32)
// and the copies' writes to shared memory; at 4:32 half as many rows carry each, and the compute warps read two or
// three spilled registers per window (every variant spills 8 to 24 bytes; at 8:32 none of it is in the window loop).  Measured, us: 4096 cubed, 8:32, 620 -> 564; 128 x 1024 x 131072, 4:32, 107 -> 84;
// 777 x 5760 x 2080, 12:32, row-major, 164 -> 153; 64 x 11008 x 4096, 8:32, 42.2 -> 40.3; 2368 x 4096 x 4096, 16:32, 671 -> 661.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "gemm_args.h"
#include "kernels.h"

namespace nmspmm {

// WR x WV warps; a warp's tile is WM rows x VPW vectors (WM 128: one, 64: two).
template <int WR_, int WV_, int WM_, int WS_, int KS_, int MODE>
struct WideCfg {
    static constexpr int WR = WR_, WV = WV_, WM = WM_, WS = WS_, KS = KS_;
    static constexpr int VPW = 128 / WM;
    static constexpr int MS = WR * WM, QT = WV * VPW, NS = QT * kVecLen;
    static constexpr int NCW = WR * WV, NCT = NCW * 32, THREADS = NCT + 128;
    static constexpr int LAUNCH_REGS = 168, COMPUTE_REGS = 232, FEED_REGS = 40;
    static_assert(2 * COMPUTE_REGS + FEED_REGS == 3 * LAUNCH_REGS, "the warpgroups share what the launch was given");
    static constexpr int A_BYTES = KS * MS * 4, B_BYTES = WS * NS * 4;
    static constexpr int B_BOX = NS > 256 ? 256 : NS;            // columns per copy of B (a box is at most 256 wide)
    static constexpr int D_BYTES = (WS * QT * 4 + 127) / 128 * 128;
    static constexpr int CI_BYTES = (MODE == kModeHigh) ? QT * 256 : 0;
    static constexpr int O_BYTES = D_BYTES;                      // resolved offsets, [QT][WS]
    static constexpr int BAR_REL = A_BYTES + B_BYTES + D_BYTES + CI_BYTES + O_BYTES;     // the stage's three barriers
    static constexpr int STAGE_BYTES = BAR_REL + 128;
    static constexpr int RESOLVERS = 3;
    static constexpr int CTRL_BYTES = 128;
    static constexpr int ST0 = (227 * 1024 - 128 - CTRL_BYTES) / STAGE_BYTES;
    static constexpr int STAGES = ST0 > 8 ? 8 : ST0;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + CTRL_BYTES + 128;
    static_assert(NCW == 8 && (WM == 128 || WM == 64) && QT >= 4, "warp tiles");
    static_assert(WS % 4 == 0 && STAGES >= 2, "stages");
    static_assert(WS * NS * 4 % 128 == 0 && KS * MS * 4 % 128 == 0, "operands start on 128 bytes");
};

// What a compute thread holds of its CTA's tile.
// Lanes: a 128-bit shared load takes one wavefront per eight lanes, and two such groups share
// one where lane i reads the address of lane i ^ 1 (A: bit 0 is a column bit) or of lane
// i ^ 2 (B: bit 1 is a row bit).  With two vectors per warp bit 3 tells them apart; their
// rows of A and columns of B meet in the same banks, so the second vector's lanes take the
// halves of both in the other order.
template <int WR, int WV, int WM>
struct WideLane {
    static constexpr int VPW = 128 / WM, NCT = WR * WV * 32;
    static constexpr int RSTEP = (VPW == 2) ? 16 : 32;     // rows between a thread's groups of four
    int vec;                                               // vector of the tile
    int r0, r1;                                            // first rows of its groups 0 and 1; 2 and 3 follow 2 RSTEP on
    int c0, c1;                                            // first columns of its two groups of four, within the vector
    __device__ __forceinline__ explicit WideLane(int tid)
    {
        const int lane = tid & 31, warp = tid >> 5, vsel = (VPW == 2) ? (lane >> 3) & 1 : 0;
        const int lm = (VPW == 2) ? (lane >> 1) & 3 : (lane >> 1) & 7;
        vec = warp % WV * VPW + vsel;
        r0 = warp / WV * WM + lm * 4 + vsel * RSTEP;
        r1 = warp / WV * WM + lm * 4 + (RSTEP - vsel * RSTEP);
        c0 = (lane >> 4) * 8 + (lane & 1) * 4 + vsel * 16;
        c1 = c0 ^ 16;
    }
    __device__ __forceinline__ int row(int i) const { return ((i & 4) ? r1 : r0) + (i >> 3) * 2 * RSTEP + (i & 3); }     // i-th of sixteen
};

template <int WR, int WV, int WM, int WS, int KS, int MODE, bool MULTI>
__device__ __forceinline__ void nm_gemm_wide_body(const GemmArgs& g, const CUtensorMap& map_a, const CUtensorMap& map_b,
                                                  const GemmOutputs& outs)
{
    using Cfg = WideCfg<WR, WV, WM, WS, KS, MODE>;
    constexpr int MS = Cfg::MS, NS = Cfg::NS, QT = Cfg::QT, VPW = Cfg::VPW, STAGES = Cfg::STAGES, NCT = Cfg::NCT;
    constexpr int B_REL = Cfg::A_BYTES, D_REL = B_REL + Cfg::B_BYTES, CI_REL = D_REL + Cfg::D_BYTES, O_REL = CI_REL + Cfg::CI_BYTES;

    extern __shared__ unsigned char smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 127u) & ~127u;
    constexpr int FULL = Cfg::BAR_REL, IDX = FULL + 8, EMPTY = FULL + 16;     // operands landed and offsets resolved; indices landed; read by every compute warp
    const uint32_t ring_end = ring + STAGES * Cfg::STAGE_BYTES, abort_word = ring_end;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        prefetch_tensor_map(&map_a);
        prefetch_tensor_map(&map_b);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(ring + s * Cfg::STAGE_BYTES + FULL, 1 + Cfg::RESOLVERS);     // the copies' bytes, the resolving warps
            mbar_init(ring + s * Cfg::STAGE_BYTES + IDX, 1);
            mbar_init(ring + s * Cfg::STAGE_BYTES + EMPTY, Cfg::NCW);
        }
        sts_volatile_s32(abort_word, 0);
        mbar_init_fence();
    }
    // the compute warps read ahead without asking whether there is a next window: what they find is always a row
    for (int e = tid; e < STAGES * QT * WS; e += Cfg::THREADS) sts_s32(ring + e / (QT * WS) * Cfg::STAGE_BYTES + O_REL + e % (QT * WS) * 4, ring);
    __syncthreads();
    grid_dependency_wait();                                // everything above overlapped the tail of the kernel ahead

    int u_begin, n_units;                                  // this CTA's range
    {
        long long u0, u1;
        virtual_range(g.sched, blockIdx.x, u0, u1);
        u_begin = static_cast<int>(u0);
        n_units = static_cast<int>(u1 - u0);
    }
    const int n_win = g.sched.n_win, tiles_y = (g.M + MS - 1) / MS;
    const int qs_shift = g.qs_shift;                       // log2(vectors per packed index block)

    if (warp >= Cfg::NCW) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::FEED_REGS));
        const int d_chunk = WS << qs_shift;                // ints of one index block's window
        const uint32_t d_bytes = static_cast<uint32_t>(d_chunk) * 4u;
        bool alive = true;
        // (These warps share the schedulers with compute warps that wait for none of them to spare: no
        // division per window, and the index work spread over three of them.)
        int tile = u_begin / n_win, win = u_begin - tile * n_win;
        uint32_t st = ring, parity = 0;
        auto advance = [&]() {                             // true: on to the next tile
            st += Cfg::STAGE_BYTES;
            if (st == ring_end) {
                st = ring;
                parity ^= 1;
            }
            if (++win < n_win) return false;
            win = 0;
            ++tile;
            return true;
        };
        if (warp == Cfg::NCW) {
            // ------------------------------------------------ copies
            int bi, bj, nlb;                               // the tile, and the index blocks under it
            const int* d_src;                              // this lane's index block at window `win`, and its list
            const int* ci_src = nullptr;
            auto enter_tile = [&]() {
                int ty, tx;
                tile_coords(tile, g.tiles_x, tiles_y, ty, tx);
                bi = ty * MS;
                bj = tx * NS;
                const int q0 = tx * QT, lb0 = q0 >> qs_shift;
                nlb = ((min(q0 + QT, g.N >> 5) - 1) >> qs_shift) - lb0 + 1;
                d_src = g.D + ((static_cast<size_t>(lb0 + lane) * g.W) << qs_shift) + static_cast<size_t>(win) * d_chunk;
                if constexpr (MODE == kModeHigh) ci_src = g.cinfo + (static_cast<size_t>(lb0 + lane) * n_win + win) * 64;
            };
            enter_tile();
            for (int j = 0; j < n_units; ++j) {
                if (j >= STAGES) {
                    alive = __all_sync(0xffffffffu, mbar_sleep_bounded(st + EMPTY, parity ^ 1, abort_word));
                    if (!alive) break;
                }
                const uint32_t idx = st + IDX, full = st + FULL;
                if (elect_one()) {
                    mbar_arrive_expect_tx(idx, nlb * (d_bytes + (MODE == kModeHigh ? 256u : 0u)));
                    mbar_arrive_expect_tx(full, Cfg::A_BYTES + Cfg::B_BYTES);
                    tma_load_2d(st, &map_a, bi, win * KS, full);         // rows / columns past the tensor arrive as zeros
                    for (int c = 0; c < NS; c += Cfg::B_BOX) tma_load_2d(st + B_REL + c * (WS * 4), &map_b, bj + c, win * WS, full);
                }
                __syncwarp();
                if (lane < nlb) {
                    bulk_g2s(st + D_REL + lane * d_bytes, d_src, d_bytes, idx);
                    if constexpr (MODE == kModeHigh) bulk_g2s(st + CI_REL + lane * 256, ci_src, 256, idx);
                }
                d_src += d_chunk;
                if constexpr (MODE == kModeHigh) ci_src += 64;
                if (advance()) enter_tile();
            }
        } else {
            // ------------------------------------------------ indices -> offsets
            constexpr int PER = (QT * WS + Cfg::RESOLVERS * 32 - 1) / (Cfg::RESOLVERS * 32);
            const int e0 = (warp - Cfg::NCW - 1) * 32 + lane;
            uint32_t d_rel[PER], ci_rel[PER];              // this lane's entries: vector (e / WS), kept row e % WS
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int e = e0 + i * (Cfg::RESOLVERS * 32), v = e / WS, p = e - v * WS, lb = v >> qs_shift;     // (a tile starts on an index block)
                d_rel[i] = D_REL + (lb * d_chunk + (p << qs_shift) + (v & ((1 << qs_shift) - 1))) * 4;
                ci_rel[i] = CI_REL + lb * 256;
            }
            int live = 0;                                  // entries of the tile's vectors that exist
            auto enter_tile = [&]() {
                int ty, tx;
                tile_coords(tile, g.tiles_x, tiles_y, ty, tx);
                live = min(QT, (g.N >> 5) - tx * QT) * WS;
            };
            enter_tile();
            for (int j = 0; j < n_units; ++j) {
                alive = __all_sync(0xffffffffu, mbar_sleep_bounded(st + IDX, parity, abort_word));
                if (!alive) break;
                int k[PER];
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int e = e0 + i * (Cfg::RESOLVERS * 32);
                    k[i] = 0;                              // vectors past N: any row of A, against zeros of B
                    if (e < live) k[i] = lds_s32(st + d_rel[i]);
                }
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int e = e0 + i * (Cfg::RESOLVERS * 32);
                    if (MODE == kModeHigh && e < live) k[i] = lds_s32(st + ci_rel[i] + k[i] * 4);
                    if (e < QT * WS) sts_s32(st + O_REL + e * 4, static_cast<int>(st) + k[i] * (MS * 4));
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(st + FULL);
                if (advance()) enter_tile();
            }
        }
        if (!alive && lane == 0) atomicMax(g.status, kDevTimeoutEmpty);
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::COMPUTE_REGS));

    // ---------------------------------------------------------------------- compute warps
    using Lane = WideLane<WR, WV, WM>;
    constexpr int RSTEP = Lane::RSTEP;
    const Lane me(tid);
    const uint32_t a0_rel = me.r0 * 4, a1_rel = me.r1 * 4;
    constexpr int BROW = Cfg::B_BOX * 4;                   // bytes of a row of B in shared memory
    const uint32_t b0_rel = B_REL + (me.vec * kVecLen / Cfg::B_BOX) * (WS * BROW) + (me.vec * kVecLen % Cfg::B_BOX + me.c0) * 4;
    const uint32_t b1_rel = (me.c1 - me.c0) * 4;
    const uint32_t o_rel = O_REL + me.vec * (WS * 4);

    float a[2][16];
    float4 b[2][2];
    auto load = [&](int buf, uint32_t bs, int p, int row) {        // bs: the stage's rows of B (+ b0_rel), row: address of the row of A
        const uint32_t x0 = row + a0_rel, x1 = (VPW == 1) ? x0 + RSTEP * 4 : row + a1_rel;
        const float4 v0 = lds_f4(x0), v1 = lds_f4(x1), v2 = lds_f4(x0 + 2 * RSTEP * 4), v3 = lds_f4(x1 + 2 * RSTEP * 4);
        a[buf][0] = v0.x; a[buf][1] = v0.y; a[buf][2] = v0.z; a[buf][3] = v0.w;
        a[buf][4] = v1.x; a[buf][5] = v1.y; a[buf][6] = v1.z; a[buf][7] = v1.w;
        a[buf][8] = v2.x; a[buf][9] = v2.y; a[buf][10] = v2.z; a[buf][11] = v2.w;
        a[buf][12] = v3.x; a[buf][13] = v3.y; a[buf][14] = v3.z; a[buf][15] = v3.w;
        b[buf][0] = lds_f4(bs + p * BROW);
        b[buf][1] = lds_f4((VPW == 1 ? bs + 64 : bs + b1_rel) + p * BROW);
    };

    uint32_t st = ring, parity = 0;                        // stage of the window to wait for next, and the parity of that wait
    // A wait that gives up raises the CTA's abort word and the device's status: nothing is stored from then on.
    bool alive = true;
    auto wait_full = [&]() { return __all_sync(0xffffffffu, mbar_wait_bounded(st + FULL, parity, abort_word)) != 0; };
    auto advance = [&]() {
        st += Cfg::STAGE_BYTES;
        if (st == ring_end) {
            st = ring;
            parity ^= 1;
        }
    };

    for (int cu = u_begin, u_end = u_begin + n_units; alive && cu < u_end;) {
        int windows;                                       // of this piece
        bool warp_live;                                    // some column of this warp exists
        {
            const int tile = cu / n_win;
            windows = min((tile + 1) * n_win, u_end) - cu;
            int ty, tx;
            tile_coords(tile, g.tiles_x, tiles_y, ty, tx);
            warp_live = tx * NS + warp % WV * (VPW * kVecLen) < g.N;
        }

        float2 acc[8][8];                                  // (rows 2 i, 2 i + 1) x column
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[i][c] = make_float2(0.0f, 0.0f);

        alive = wait_full();
        if (!warp_live) {                                  // vectors past N: keep the ring moving
            for (int w = 1; alive; ++w) {
                if (lane == 0) mbar_arrive(st + EMPTY);
                advance();
                if (w == windows) break;
                alive = wait_full();
            }
        } else if (alive) {
            int4 o_first = lds_i4(st + o_rel);             // row offsets of the window's first four kept rows
            load(0, st + b0_rel, 0, o_first.x);
            for (int w = windows; w > 0; --w) {
                const uint32_t sc = st, bs = st + b0_rel;
                int4 o[WS / 4];
                o[0] = o_first;
                advance();
#pragma unroll
                for (int p = 0; p < WS; ++p) {
                    if (p % 4 == 1 && p / 4 + 1 < WS / 4) o[p / 4 + 1] = lds_i4(sc + o_rel + (p / 4 + 1) * 16);
                    if (p == WS - 2) {                     // the next window: its rows of A are known before this one's last products
                        if (w > 1) alive = wait_full();
                        o_first = lds_i4(st + o_rel);
                    }
                    if (p + 1 < WS) {
                        const int4& q = o[(p + 1) / 4];
                        load((p + 1) & 1, bs, p + 1, (p + 1) % 4 == 0 ? q.x : ((p + 1) % 4 == 1 ? q.y : ((p + 1) % 4 == 2 ? q.z : q.w)));
                    } else {
                        load(0, st + b0_rel, 0, o_first.x);
                    }
                    const float4 b0 = b[p & 1][0], b1 = b[p & 1][1];
                    const float bv[8] = { b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w };
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float2 bb = make_float2(bv[c], bv[c]);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int r = (c & 1) ? 7 - i : i;
                            acc[r][c] = __ffma2_rn(make_float2(a[p & 1][2 * r], a[p & 1][2 * r + 1]), bb, acc[r][c]);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(sc + EMPTY);
                if (!alive) break;
            }
        }

        // -------------------------------------------------------------- end of the piece
        // (what only this part needs is worked out again from here: the loop above has no register to spare)
        int tid_e, cu_e = cu;
        asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid_e));
        asm volatile("" : "+r"(cu_e));
        const Lane own(tid_e);
        const int tile = cu_e / n_win, piece_n = min((tile + 1) * n_win, u_end) - cu_e;
        int ty, tx;
        tile_coords(tile, g.tiles_x, tiles_y, ty, tx);
        const int bj = tx * NS, bi = ty * MS;
        if (cu_e + piece_n >= u_end) grid_launch_dependents();     // last piece: only stores are left
        auto store_tile = [&]() {
            if (own.vec * kVecLen >= g.N - bj) return;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int r = bi + own.row(i);
                if (r < g.M) {
                    auto val = [&](int c) { return (i & 1) ? acc[i >> 1][c].y : acc[i >> 1][c].x; };
                    const float4 x = make_float4(val(0), val(1), val(2), val(3)), y = make_float4(val(4), val(5), val(6), val(7));
                    if constexpr (MULTI) {
                        const size_t at = static_cast<size_t>(r) * outs.ldc + outs.col0 + bj + own.vec * kVecLen;
                        for (int o = 0; o < outs.n_out; ++o) {
                            float* cp = output_of(g, outs, o) + at;
                            *reinterpret_cast<float4*>(cp + own.c0) = x;
                            *reinterpret_cast<float4*>(cp + own.c1) = y;
                        }
                    } else {
                        float* cp = g.C + static_cast<size_t>(r) * g.N + bj + own.vec * kVecLen;
                        *reinterpret_cast<float4*>(cp + own.c0) = x;
                        *reinterpret_cast<float4*>(cp + own.c1) = y;
                    }
                }
            }
        };
        if (piece_n == n_win) {
            if (alive) store_tile();                       // the whole tile was computed here
        } else {
            // A piece of the tile goes to this range's scratch slot: the reduction kernel adds them.  (Added by the last
            // to arrive, as on the smaller tiles, 256 x 11008 x 4096, 8:32 took 114.3 us instead of 112.0, 4096 cubed 574.7 instead of 573.0.)
            float4* slots = reinterpret_cast<float4*>(g.partial);
            constexpr size_t kSlot = static_cast<size_t>(32) * NCT;            // float4 words per slot
            {
                float4* mine = slots + static_cast<size_t>(piece_slot(g.sched, blockIdx.x, tile)) * kSlot + tid_e;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    auto val = [&](int c) { return (i & 1) ? acc[i >> 1][c].y : acc[i >> 1][c].x; };
                    __stcg(mine + (2 * i) * NCT, make_float4(val(0), val(1), val(2), val(3)));
                    __stcg(mine + (2 * i + 1) * NCT, make_float4(val(4), val(5), val(6), val(7)));
                }
            }
        }
        cu = cu_e + piece_n;
    }
    if (!alive && lane == 0) atomicMax(g.status, kDevTimeoutFull);
}

template <int WR, int WV, int WM, int WS, int KS, int MODE>
__global__ void __launch_bounds__((WideCfg<WR, WV, WM, WS, KS, MODE>::THREADS), 1)
nm_gemm_wide_kernel(const GemmArgs g, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b)
{
    nm_gemm_wide_body<WR, WV, WM, WS, KS, MODE, false>(g, map_a, map_b, GemmOutputs {});
}

template <int WR, int WV, int WM, int WS, int KS, int MODE>
__global__ void __launch_bounds__((WideCfg<WR, WV, WM, WS, KS, MODE>::THREADS), 1)
nm_gemm_wide_multi_kernel(const GemmArgs g, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                          const __grid_constant__ GemmOutputs outs)
{
    nm_gemm_wide_body<WR, WV, WM, WS, KS, MODE, true>(g, map_a, map_b, outs);
}

template <int WR, int WV, int WM, int WS, int KS, int MODE, bool MULTI>
cudaError_t launch_wide(const GemmArgs& a, const GemmOutputs& outs, int grid, cudaStream_t st)
{
    using Cfg = WideCfg<WR, WV, WM, WS, KS, MODE>;
    static bool configured[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && !configured[dev]) {
        if (MULTI)
            e = cudaFuncSetAttribute(nm_gemm_wide_multi_kernel<WR, WV, WM, WS, KS, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     Cfg::SMEM_BYTES);
        else
            e = cudaFuncSetAttribute(nm_gemm_wide_kernel<WR, WV, WM, WS, KS, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        // the compute warps' share comes out of what the launch is given: less of it and they would wait
        cudaFuncAttributes fa;
        if (MULTI) e = cudaFuncGetAttributes(&fa, nm_gemm_wide_multi_kernel<WR, WV, WM, WS, KS, MODE>);
        else e = cudaFuncGetAttributes(&fa, nm_gemm_wide_kernel<WR, WV, WM, WS, KS, MODE>);
        if (e != cudaSuccess) return e;
        if (fa.numRegs < Cfg::LAUNCH_REGS) return cudaErrorInvalidKernelImage;
        configured[dev] = true;
    }
    CUtensorMap map_a, map_b;
    e = encode_tensor_map_2d(&map_a, a.A, outs.lda ? outs.lda : a.M, a.sched.n_win * KS, Cfg::MS, KS);
    if (e != cudaSuccess) return e;
    e = encode_tensor_map_2d(&map_b, a.B, a.N, a.W, Cfg::B_BOX, WS - (g_test_short_fill ? 1 : 0));     // (test hook, see kernels.h)
    if (e != cudaSuccess) return e;
    if (MULTI)
        return launch_overlapped(nm_gemm_wide_multi_kernel<WR, WV, WM, WS, KS, MODE>, grid, Cfg::THREADS, Cfg::SMEM_BYTES, st, a, map_a, map_b,
                                 outs);
    return launch_overlapped(nm_gemm_wide_kernel<WR, WV, WM, WS, KS, MODE>, grid, Cfg::THREADS, Cfg::SMEM_BYTES, st, a, map_a, map_b);
}

#define NMSPMM_WIDE_VARIANT(ID, NKEEP, WR, WV, WM, WS, KS, MODE)                                                        \
    FfmaVariant { ID, WideCfg<WR, WV, WM, WS, KS, MODE>::MS, WideCfg<WR, WV, WM, WS, KS, MODE>::NS, NKEEP, WS, KS, MODE,  \
                  WideCfg<WR, WV, WM, WS, KS, MODE>::THREADS, WideCfg<WR, WV, WM, WS, KS, MODE>::SMEM_BYTES,              \
                  WideCfg<WR, WV, WM, WS, KS, MODE>::STAGES, 1, &launch_wide<WR, WV, WM, WS, KS, MODE, false>,            \
                  &launch_wide<WR, WV, WM, WS, KS, MODE, true> }

// The wide tiles for one (kept rows per 32-window, B rows per stage, A rows per stage, MODE).
#define NMSPMM_WIDE_TILES(NKEEP, WS, KS, MODE)                               \
    NMSPMM_WIDE_VARIANT(kTile128x256, NKEEP, 1, 8, 128, WS, KS, MODE),       \
    NMSPMM_WIDE_VARIANT(kTile256x128, NKEEP, 2, 4, 128, WS, KS, MODE),       \
    NMSPMM_WIDE_VARIANT(kTile64x512, NKEEP, 1, 8, 64, WS, KS, MODE)

}  // namespace nmspmm
