// TF32 tensor-core path of the vector-wise N:M sparse GEMM (tcgen05, accumulators in TMEM).
//
// One CTA computes a 128 x NS tile of C (QT = NS / 32 vectors of 32 columns; NS = 256, 192 or 128) over its k steps.
// A step is one 32-k window (one 64-k merged window for 4:32) with WS kept rows of B.  The
// contraction is per vector, C[128 x 32] += A_gathered[128 x WS] . B[WS x 32], and A_gathered
// (the WS columns of the step's A window that the vector's index list names) differs for
// every vector.  The gather itself is done by the tensor core:
//
//     G[128 x QT*WS] = A_window[128 x KW] . P[KW x QT*WS]
//
// where column (v, j) of P is one-hot at the k that vector v's j-th index names.  Products
// with 1.0 and sums with 0.0 are exact, so G holds exactly the (TF32-truncated) gathered
// values -- in Tensor Memory, lane = tile row, column = (v, j): the layout of a TMEM A
// operand.  The second instruction group then multiplies, per vector, G's WS columns by the
// vector's WS x 32 block of B.  Nothing of A goes through registers; the only generic-proxy
// shared-memory traffic of the main loop is two 4-byte stores per index (clear the old
// one-hot entry, set the new one).  Tensor work is twice the useful work for every ratio.
// A non-finite value anywhere in a row of the A window reaches every gathered column of that
// row (0 x inf), not only the vectors that select it: this path wants finite A.
//
//   warp 0      TMA producer: per step one tiled copy of the A window and one of the B rows,
//               both as blocks of 32 floats along m / n with 32-byte chunks swizzled within
//               128-byte rows (the one legal layout of an MN-major TF32 operand).
//   warp 1      (and 2 where a step is short) one elected thread issues the gathers (tcgen05.mma kind::tf32, A and P from
//               shared memory, M128 N=QT*WS, KW/8 instructions per step) into a ring of
//               result buffers in TMEM, each followed by a tcgen05.commit to the buffer's
//               mbarrier.
//   next two    one elected thread each issues the products of half the tile's vectors
//               (A = G from TMEM, B from shared memory, M128 N32 K8 each) once the gather's
//               mbarrier has completed, and commits to the mbarrier that frees the stage and
//               the result buffer.  Measured alone (instruction chains, cycles): a product takes the pipe
//               16 / 32 at N = 32 / 64, its arithmetic and no more; a gather 40 / 48 / 64 at N = 32 / 64 / 128,
//               in TF32 (K = 8) and 16 bits (K = 16) alike; one thread issues an instruction every 27.
//               Issuers are one elected thread each, from first wait to last commit, operand
//               descriptors by addition: with a warp-wide wait, a vote and descriptors built anew
//               per instruction a step of 8:32 took 600 cycles on the issuers' side alone (2048 x 9472 x 4096, 8:32,
//               186 -> 138 us; 256 x 11008 x 4096, bfloat16, 42 -> 31.5, and 28.0 with what GATHER_WARPS, PAIRS and 192 columns add).
//   the others  (eight; four on the 128-column tile, at 16:32 and 12:32 with 32-wide vectors, and at 32:32) one
//               thread per (vector, kept row) and turn: loads its index two to four turns ahead
//               into registers (through column_info on the 64-k format), keeps P's one-hot
//               entry current, and after the last step reads the accumulators (tcgen05.ld),
//               transposes them through shared memory and stores C in 128-byte row pieces.
//
// What bounds a step now is what feeds it: a tiled copy takes the SM about 2.1 cycles per row of its
// box (128 bytes or fewer): 128 rows of A and 64 of B, 400 cycles, at 8:32, for FP32 and 16-bit
// activations alike -- without any tensor-core instruction the kernel takes 126 us where it takes 138 (FP32)
// and 125 (bfloat16) with them.  16:32 and 12:32 with 32-wide vectors have room for two gather results only, and
// a result's way to its products and back, about 500 cycles each, is exposed (780 cycles a step with everything else left out;
// at 4096 cubed the tensor pipe is active 59 % of an 8:32 call's cycles and 62 % of a 16:32 call's).  Long runs are also
// under the power cap: 1.68 to 1.72 GHz there, 1.57 at 8192 x 28672 x 8192 (2817 us after a pause, 3242 back to back).
// n_keep = 32 (nothing pruned) has the identity as its index list and multiplies A_window by
// the B rows directly.  12:32 gathers 16 columns per vector of which 4 are zero (P has no
// entry for them), and loads 16 rows of B per vector of which the last 4 meet those zeros.
//
// Row-major A (activations as a layer has them) is read as it lies in memory: a window is 128 rows x
// KW columns, a K-major operand.  FP32 rows change nothing else.  Half and bfloat16 rows are
// gathered in their own type (kind::f16, one-hot P of that type, FP32 result: exact), K = 16 per
// instruction: half as many gather instructions per step and half of A's bytes, no transposing and
// widening launch ahead of the multiply, and C is stored in the activations' type.
// 256 x 11008 x 4096, bfloat16, 8:32: 59.5 us with a transposing and a rounding launch, 28.0 now.
// Every wait is bounded; a wait that gives up raises the device status word.
#include <cuda.h>

#include "common.cuh"
#include "gemm_args.h"
#include "kernels.h"
#include "tcgen05.cuh"
#include "tf32_epilogue.cuh"

namespace nmspmm {

// Diagnostic target, not part of the shipped library: built with
//     NMSPMM_NVCC_EXTRA=-DNMSPMM_TF32_PROFILE NMSPMM_BUILD_DIR=<dir> NMSPMM_BUILD_LIB=<file.so> python nm-spmm_b200/build.py
// the kernel adds up, per role, the cycles (clock64) spent waiting and issuing, and
// nmspmm_debug_tf32_profile (exported by that build only) reads and clears the sixteen sums:
//   0 producer waits for a free stage, 1 producer total, 2 / 3 / 4 / 5 gather issuer: wait for the
//   stage, wait for a result buffer, issue, total, 6 / 7 / 15 product issuer: wait for the gather,
//   issue, total, 8 CTAs, 9 steps, 13 / 14 epilogue: wait for the accumulators, run.  The
//   issuers of steps in pairs (Cfg::PAIRS) count nothing: 2 to 9 and 15 stay zero there.
// Without the macro every TF_* below expands to nothing.
#ifdef NMSPMM_TF32_PROFILE
__device__ unsigned long long g_tf32_profile[16];
#define TF_DECL(...) long long __VA_ARGS__
#define TF_T(name) const long long name = clock64()
#define TF_ADD(acc, since) acc += clock64() - (since)
#define TF_OUT(i, v) atomicAdd(&g_tf32_profile[i], (unsigned long long)(v))
#else
#define TF_DECL(...)
#define TF_T(name)
#define TF_ADD(acc, since)
#define TF_OUT(i, v)
#endif

// How A is read: col-major FP32, or row-major FP32 / 16-bit values (half or bfloat16 by launch).
enum { kTf32Cols = 0, kTf32Rows32 = 1, kTf32Rows16 = 2 };

template <int NKEEP, int KW_, int MODE, int QT_, int VL_ = 32, int SRC_ = kTf32Cols>
struct Tf32Cfg {
    static constexpr int SRC = SRC_;
    static constexpr int EB = (SRC == kTf32Rows16) ? 2 : 4;  // bytes of a value of A and of P
    static constexpr int MS = 128, QT = QT_, NS = QT * 32;   // QT = 8 and 6: one CTA per SM; QT = 4: two
    static constexpr int KW = KW_;                           // k per step
    static constexpr int WS = NKEEP * (KW / 32);             // rows of B per step
    static constexpr int WSP = (WS + 7) / 8 * 8;             // gathered columns per vector (K of the products)
    static constexpr bool DIRECT = (NKEEP == 32);            // identity index list: no gather
    static constexpr int G = WSP / 8;                        // product instructions per vector and step
    static constexpr int NKS = KW * EB / 32;                 // gather instructions per step (32 bytes of K each)
    static constexpr int VL = VL_;                           // columns that share an index list: 32, or 64 (two adjacent equal lists)
    static constexpr int QV = NS / VL;                       // vectors per tile
    static constexpr int N1 = QV * WSP;                      // gathered columns per step
    static_assert(VL == 32 || (VL == 64 && NKEEP != 32), "vectors of 32 or 64 columns");
    static constexpr int NT = (N1 + 31) / 32 * 32;           // threads that keep them, whole warps; columns of P's 32-bit layout
    static_assert(DIRECT || (N1 <= 128 && N1 % 16 == 0), "one builder thread per gathered column");
    static_assert(MODE == kModeHigh || KW == 32, "only the 64-k format has merged windows");
    static_assert(!(DIRECT && SRC == kTf32Rows16), "the direct product multiplies A by FP32 rows of B");
    static constexpr int A_BYTES = 128 * KW * EB;            // col-major: [4 blocks of 32 rows of the tile][KW][32]; rows: [128][<= 128 bytes], blocks of 32 k if FP32
    static constexpr int B_BYTES = QT * WSP * 128;           // [QT][WSP][32]
    static constexpr int P_BYTES = DIRECT ? 0 : (EB == 2 ? N1 : NT) * KW * EB;      // [NT / 32][KW][32]; 16 bits: K-major, [N1][KW]
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES + P_BYTES;
    static_assert(A_BYTES % 1024 == 0 && B_BYTES % 1024 == 0 && P_BYTES % 1024 == 0, "swizzle atoms stay aligned");
    static constexpr int CTAS_PER_SM = (QT > 4) ? 1 : 2;
    static constexpr int TMEM_COLS = 512 / CTAS_PER_SM;      // each resident CTA allocates its share
    static constexpr int PD = 2;                             // index prefetch distance, in turns, per look-up
    // One thread keeps one gathered column; the builder warps form GROUPS groups of N1 threads that take
    // turns with the steps.  A step is a chain of some 600 cycles for the warp that builds it (index
    // arrived, stage free, old entry, new entry, proxy fence, arrival): with one group that chain,
    // not the tensor pipe, was part of what an 8:32 step waited for: 4096 x 4096 x 11008, 8:32, 417 -> 404 us,
    // with bfloat16 activations 444 -> 405; 4096 x 28672 x 2048 with 64-wide vectors 667 -> 636 and 632 -> 578.
    // (16:32 and 12:32 with 32-wide vectors fill one group of 128: a second one gained nothing there, their steps are longer.)
    static constexpr int BUILDERS = (QT > 4 && N1 < 128) ? 256 : 128;
    static constexpr int GROUP_WARPS = NT / 32;
    static constexpr int PRODUCT_WARPS = 2;
    // A wait costs the thread that issues some 150 to 190 cycles even when it is over already, and a gather
    // has two of them ahead of it: where a step takes less, two threads take turns with the gathers (2048 x 9472 x 4096,
    // bfloat16, 8:32, 125 -> 116 us, 64-wide vectors 121 -> 107, and in FP32 131 -> 125; FP32 8:32 with 32-wide vectors and 4:32 lose 2 - 4 %
    // on 256 columns: the second gather only crowds the products).
    static constexpr int GATHER_WARPS = (!DIRECT && KW == 32 && N1 <= 96 && (EB == 2 || VL == 64 || QT == 6)) ? 2 : 1;
    static constexpr int THREADS = (1 + GATHER_WARPS + PRODUCT_WARPS) * 32 + BUILDERS;
    // Every stage counts (2048 x 9472 x 4096, 8:32, six / eight stages: 145 / 138 us, 64-wide vectors 141 / 130; 4096 cubed, 4:32,
    // three / four: 142 / 121).
    static constexpr int MAX_STAGES = 8;
    static constexpr int AUX_BYTES = MAX_STAGES * 128;       // previous one-hot per stage and column (a byte each)
    static constexpr int CTRL_BYTES = 256;
    static constexpr int SMEM_LIMIT = (CTAS_PER_SM == 1 ? 227 : 113) * 1024;
    static constexpr int ST0 = (SMEM_LIMIT - 1024 - AUX_BYTES - CTRL_BYTES) / STAGE_BYTES;
    static constexpr int STAGES = ST0 > MAX_STAGES ? MAX_STAGES : ST0;
    static_assert(STAGES >= 2, "at least two stages");
    // A group that has built step i - GROUPS knows that step i - GROUPS - STAGES has been consumed; its
    // wait for the stage of step i tells one phase from the next only if step i - 2 STAGES has been.
    static constexpr int GROUPS = DIRECT ? 1 : (BUILDERS / NT < STAGES ? BUILDERS / NT : STAGES);
    static_assert(GROUPS >= 1 && GROUPS <= STAGES, "see above");
    // Ring of gather results beside the accumulators.  A gather's result is complete (and its
    // commit arrives) some hundreds of cycles after issue, and the products that free the
    // buffer again take as long: the loop gather -> products -> gather is latency-bound
    // unless several steps are in flight, so the ring is as deep as Tensor Memory allows.
    static constexpr int NBUF0 = DIRECT ? 1 : (TMEM_COLS - NS) / N1;
    static constexpr int NBUF1 = NBUF0 > 4 ? 4 : NBUF0;
    static constexpr int NBUF = NBUF1 > STAGES ? STAGES : NBUF1;     // (the barrier that frees a step's stage frees its buffer too)
    static_assert(NBUF >= 1, "no room for a gather result beside the accumulators");
    // 16-bit activations: pairs of steps share one commit and one wait between gather and products where Tensor
    // Memory holds three pairs of results or more -- their steps are the shortest, and the products' issuers spend
    // them waiting (256 x 11008 x 4096, 8:32, 28.4 -> 27.8 us, 25.4 with the weights in L2; 2048 x 9472 x 4096, 64-wide vectors, 107 -> 102; in FP32 125 -> 127).
    // The buffers of a pair are free when the stage of its second step is; that stage's next phase may not end
    // before they are asked for; and a stage's last step is done by then, so that the wait on it is unmistakable.
    static constexpr int NP0 = DIRECT ? 0 : (TMEM_COLS - NS) / (2 * N1);
    static constexpr int NP1 = NP0 > 4 ? 4 : NP0;
    static constexpr int NP = NP1 > STAGES / 2 ? STAGES / 2 : NP1;
    static constexpr bool PAIRS = EB == 2 && NP >= 3;
    static constexpr int EPI_BYTES = BUILDERS / 32 * kTf32PatchBytes;    // the builder warps' transposition patches
    static_assert(EPI_BYTES <= STAGES * STAGE_BYTES, "the epilogue reuses the stage ring");
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + AUX_BYTES + CTRL_BYTES + 1024;   // + alignment slack
    static constexpr int ACOL0 = NS;                         // first gather-result column
};

// Byte offset of P[k][n] (n = gathered column) inside a stage's P region.
template <int KW>
__device__ __forceinline__ uint32_t p_offset(int n, int k)
{
    const int nb = n >> 5, c = n & 31;
    return static_cast<uint32_t>(nb * (KW * 128) + k * 128 + ((((c >> 3) ^ (k & 3)) << 5) | ((c & 7) << 2)));
}

// The same for a P of 16-bit values (K-major, [N1][KW], 16-byte chunks swizzled within the rows).
template <int KW>
__device__ __forceinline__ uint32_t p16_offset(int n, int k)
{
    return static_cast<uint32_t>(n * (KW * 2) + (((k >> 3) ^ (KW == 64 ? (n & 7) : ((n >> 1) & 3))) << 4) + (k & 7) * 2);
}
__device__ __forceinline__ void sts_u16(uint32_t addr, unsigned v)
{
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"(static_cast<unsigned short>(v)) : "memory");
}

__device__ __forceinline__ int lds_s8(uint32_t addr)
{
    int v;
    asm volatile("ld.shared.s8 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts_s8(uint32_t addr, int v) { asm volatile("st.shared.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }

// C16: C is stored in 16 bits (a parameter: see gemm_tf32_few_rows.cu).
template <int NKEEP, int KW_, int MODE, int QT_, int VL_, int SRC_, bool C16>
__global__ void __launch_bounds__((Tf32Cfg<NKEEP, KW_, MODE, QT_, VL_, SRC_>::THREADS), (Tf32Cfg<NKEEP, KW_, MODE, QT_, VL_, SRC_>::CTAS_PER_SM))
nm_gemm_tf32_kernel(const GemmArgs g, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const GemmOutputs outs, const int a_form)     // col-major: 1 where the rows of A are whole blocks of 32; 16 bits: the type
{
    using Cfg = Tf32Cfg<NKEEP, KW_, MODE, QT_, VL_, SRC_>;
    constexpr int MS = Cfg::MS, NS = Cfg::NS, QT = Cfg::QT, KW = Cfg::KW, WS = Cfg::WS, WSP = Cfg::WSP;
    constexpr int VL = Cfg::VL, QV = Cfg::QV, BPV = VL / 32;              // 32-column blocks per vector
    constexpr int STAGES = Cfg::STAGES, NBUF = Cfg::NBUF, PD = Cfg::PD;
    constexpr bool DIRECT = Cfg::DIRECT;
    constexpr int GW = Cfg::GATHER_WARPS, FIRST_PRODUCT = 1 + GW, FIRST_BUILDER = FIRST_PRODUCT + Cfg::PRODUCT_WARPS;

    extern __shared__ unsigned char smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;          // swizzle atoms want 1024-byte alignment
    const uint32_t prev_k = ring + STAGES * Cfg::STAGE_BYTES;             // [STAGES][128] one-hot entry of each column now set in the stage
    const uint32_t bars = ring + STAGES * Cfg::STAGE_BYTES + Cfg::AUX_BYTES;
    const uint32_t bar_full = bars, bar_empty = bars + STAGES * 8;
    const uint32_t bar_gdone = bar_empty + STAGES * 8, bar_acc = bar_gdone + 4 * 8;
    const uint32_t tmem_word = bar_acc + 8, abort_word = tmem_word + 4;
    static_assert((2 * Cfg::MAX_STAGES + 4 + 1) * 8 + 8 <= Cfg::CTRL_BYTES, "control block");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // The first n_dp CTAs take one whole tile each.  The remaining tiles (the partial last
    // wave of a large problem, or all tiles of a small one) are cut into split_k K slices,
    // one CTA each: a slice's accumulators go to its scratch slot and the reduction kernel
    // adds the slots.
    const int n_dp = g.sched.n_dp;
    const bool sliced = static_cast<int>(blockIdx.x) >= n_dp;
    const int n_slices = sliced ? g.sched.split_k : 1;
    const int slot = static_cast<int>(blockIdx.x) - n_dp;  // scratch slot of a sliced CTA
    const int tile = sliced ? n_dp + slot / n_slices : static_cast<int>(blockIdx.x);
    int ty, tx;
    tile_coords(tile, g.tiles_x, (g.M + MS - 1) / MS, ty, tx);
    const int bi = ty * MS, bj = tx * NS;
    int win0, n_win;                                       // this CTA's steps: win0 .. win0 + n_win - 1
    slice_range(g.sched.n_win, n_slices, sliced ? slot % n_slices : 0, win0, n_win);
    const int live_vecs = min(QT, (g.N - bj) / 32);        // vectors of the tile that exist

    if (tid == 0) {
        prefetch_tensor_map(&map_a);
        prefetch_tensor_map(&map_b);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bar_full + s * 8, DIRECT ? 1 : 1 + Cfg::GROUP_WARPS);     // the TMA bytes + the warps that build the step
            mbar_init(bar_empty + s * 8, DIRECT ? 1 : Cfg::PRODUCT_WARPS);      // the commits behind the step's products
        }
        for (int b = 0; b < 4; ++b) mbar_init(bar_gdone + b * 8, 1);            // the commit behind a gather
        mbar_init(bar_acc, DIRECT ? 1 : Cfg::PRODUCT_WARPS);
        sts_volatile_s32(abort_word, 0);
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(tmem_word, Cfg::TMEM_COLS);
    if (!DIRECT) {
        for (int o = tid * 4; o < Cfg::MAX_STAGES * 128; o += Cfg::THREADS * 4) sts_s32(prev_k + o, -1);
        // P starts as all zeros; 12:32 also wants the never-set columns of every vector zero
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s = 0; s < STAGES; ++s)
            for (int o = tid * 16; o < Cfg::P_BYTES; o += Cfg::THREADS * 16)
                sts_f4(ring + s * Cfg::STAGE_BYTES + Cfg::A_BYTES + Cfg::B_BYTES + o, z);
        fence_proxy_async();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = static_cast<uint32_t>(lds_volatile_s32(tmem_word));
    grid_dependency_wait();                                // everything above overlapped the tail of the kernel ahead

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one()) {
            bool ok = true;
            uint32_t st = ring, full = bar_full, parity = 1;           // stage of step `it`, its barrier, the parity of its last use
            TF_DECL(p_empty = 0);
            TF_T(p_start);
            for (int it = 0, k = win0 * KW, w = win0 * WS; it < n_win; ++it, k += KW, w += WS) {
                if (it >= STAGES) {
                    TF_T(t0);
                    ok = mbar_wait_bounded(full + (bar_empty - bar_full), parity, abort_word);
                    TF_ADD(p_empty, t0);
                    if (!ok) break;
                }
                mbar_arrive_expect_tx(full, Cfg::A_BYTES + Cfg::B_BYTES);
                if constexpr (Cfg::SRC == kTf32Rows32) {
                    for (int kb = 0; kb < KW / 32; ++kb) tma_load_2d(st + kb * 16384, &map_a, k + kb * 32, bi, full);
                } else if constexpr (Cfg::SRC == kTf32Rows16) {
                    tma_load_2d(st, &map_a, k, bi, full);
                } else if (a_form) {
                    tma_load_3d(st, &map_a, 0, k, bi >> 5, full);
                } else {                                   // rows not a multiple of 32: four boxes of 32 rows, the ragged one zero-filled
                    for (int mb = 0; mb < 4; ++mb) tma_load_2d(st + mb * (KW * 128), &map_a, bi + mb * 32, k, full);
                }
                tma_load_3d(st + Cfg::A_BYTES, &map_b, 0, w, bj >> 5, full);
                st += Cfg::STAGE_BYTES;
                full += 8;
                if (full == bar_full + STAGES * 8) { st = ring; full = bar_full; parity ^= 1; }
            }
#ifdef NMSPMM_TF32_PROFILE
            TF_OUT(0, p_empty); TF_OUT(1, clock64() - p_start);
#endif
            if (!ok) atomicMax(g.status, kDevTimeoutEmpty);
        }
        __syncwarp();
    } else if (warp < FIRST_PRODUCT) {
        // ------------------------------------------------------------------ gather issuers: they take turns with the steps
        constexpr bool COLS = (Cfg::SRC == kTf32Cols);
        const uint32_t idesc_gather = Cfg::SRC == kTf32Rows16 ? umma_idesc_16(128, DIRECT ? 32 : Cfg::N1, a_form == kDtypeBF16)
                                                              : umma_idesc_tf32(128, DIRECT ? 32 : Cfg::N1, COLS);
        const uint32_t idesc_direct = umma_idesc_tf32(128, live_vecs * 32, COLS);
        // Low words of the operands' descriptors, 16-byte units: the next 32 bytes of K and the next stage are additions.
        const uint64_t a0 = COLS ? umma_desc_mn_tf32(ring, KW * 128, 512)
                                 : (Cfg::SRC == kTf32Rows32 ? umma_desc_k_major<128>(ring) : umma_desc_k_major<(KW * Cfg::EB < 128 ? 64 : 128)>(ring));
        const uint64_t p0 = Cfg::SRC == kTf32Rows16 ? umma_desc_k_major<(KW * Cfg::EB < 128 ? 64 : 128)>(ring + Cfg::A_BYTES + Cfg::B_BYTES)
                                                    : umma_desc_mn_tf32(ring + Cfg::A_BYTES + Cfg::B_BYTES, KW * 128, 512);
        const uint64_t b0 = umma_desc_mn_tf32(ring + Cfg::A_BYTES, WSP * 128, 512);      // (unpruned only)
        constexpr uint32_t P_STEP = (Cfg::SRC == kTf32Rows16) ? 2 : 64;
        auto a_step = [](int ks) { return Cfg::SRC == kTf32Cols ? ks * 64 : (Cfg::SRC == kTf32Rows32 ? (ks >> 2) * 1024 + (ks & 3) * 2 : ks * 2); };
        if (elect_one()) {
            bool ok = true;
            // (the stages of this thread's next step and of the step NBUF before it)
            uint32_t full = bar_full + (warp - 1) * 8, at = (warp - 1) * (Cfg::STAGE_BYTES / 16), parity = 0;
            uint32_t empty = bar_empty + (GW == 1 ? 0 : (warp - 1 + NBUF) % GW) * 8, empty_parity = 0;
            int buf = (warp - 1) % NBUF;
            if constexpr (Cfg::PAIRS) {
                constexpr int NP = Cfg::NP;
                int st = 2 * (warp - 1), free_st = -1, pb = (warp - 1) % NP;       // stages of the pair's first step and of the second of the pair whose buffers it takes
                uint32_t full_parity = 0, free_parity = 0;
                auto gather = [&](int stage, int b) {
                    const uint32_t off = stage * (Cfg::STAGE_BYTES / 16), gbuf = tmem_addr(tmem, 0, Cfg::ACOL0 + b * Cfg::N1);
#pragma unroll
                    for (int ks = 0; ks < Cfg::NKS; ++ks) {
                        if constexpr (Cfg::SRC == kTf32Rows16)
                            umma_f16_ss(gbuf, umma_desc_plus(a0, off + a_step(ks)), umma_desc_plus(p0, off + ks * P_STEP), idesc_gather, ks != 0);
                        else
                            umma_tf32_ss(gbuf, umma_desc_plus(a0, off + a_step(ks)), umma_desc_plus(p0, off + ks * P_STEP), idesc_gather, ks != 0);
                    }
                };
                for (int t = 2 * (warp - 1), pair = warp - 1; t < n_win; t += 2 * GW, pair += GW) {
                    const int st1 = (st + 1 == STAGES) ? 0 : st + 1;
                    const uint32_t parity1 = (st + 1 == STAGES) ? full_parity ^ 1 : full_parity;
                    if (pair >= NP) {
                        if (free_st < 0) free_st = (2 * (pair - NP) + 1) % STAGES;
                        ok = mbar_spin_bounded(bar_empty + free_st * 8, free_parity, abort_word);
                        free_st += 2 * GW;
                        if (free_st >= STAGES) { free_st -= STAGES; free_parity ^= 1; }
                    }
                    ok = ok && mbar_spin_bounded(bar_full + st * 8, full_parity, abort_word);
                    if (!ok) break;
                    tc_fence_after_sync();
                    gather(st, 2 * pb);
                    if (t + 1 < n_win) {
                        ok = mbar_spin_bounded(bar_full + st1 * 8, parity1, abort_word);
                        if (!ok) break;
                        tc_fence_after_sync();
                        gather(st1, 2 * pb + 1);
                    }
                    tc_commit(bar_gdone + pb * 8);
                    pb = (pb + GW) % NP;
                    st += 2 * GW;
                    if (st >= STAGES) { st -= STAGES; full_parity ^= 1; }
                }
            } else {
                TF_DECL(m_full = 0, m_free = 0, m_issue = 0);
                TF_T(m_start);
                for (int t = warp - 1; t < n_win; t += GW) {
                    TF_T(t1);
                    // the result buffer is free once the products of step t - NBUF are done, which is when that
                    // step's stage is (the stage's next phase ends with step t - NBUF + STAGES, not before this one).
                    // This wait has to come before the one on the stage: with two gathering threads and an odd number
                    // of stages, the step before in this stage was the other thread's and may still wait to be filled,
                    // where a wait by parity would take the phase before that one for the awaited one. Products are in
                    // order, so past this wait every step up to t - NBUF, t - STAGES among them, has been used up.
                    static_assert(DIRECT || NBUF <= STAGES, "a stage's last step is done once the result buffer is free");
                    if (!DIRECT && t >= NBUF) {
                        ok = mbar_spin_bounded(empty, empty_parity, abort_word);
                        empty += GW * 8;
                        if (GW == 1) {
                            if (empty == bar_empty + STAGES * 8) { empty = bar_empty; empty_parity ^= 1; }
                        } else if (empty >= bar_empty + STAGES * 8) { empty -= STAGES * 8; empty_parity ^= 1; }
                    }
                    TF_ADD(m_free, t1);
                    TF_T(t0);
                    ok = ok && mbar_spin_bounded(full, parity, abort_word);
                    TF_ADD(m_full, t0);
                    if (!ok) break;
                    TF_T(t2);
                    tc_fence_after_sync();
                    if (DIRECT) {
#pragma unroll
                        for (int ks = 0; ks < Cfg::NKS; ++ks)
                            umma_tf32_ss(tmem_addr(tmem, 0, 0), umma_desc_plus(a0, at + a_step(ks)), umma_desc_plus(b0, at + ks * 64), idesc_direct,
                                         (t | ks) != 0);
                        tc_commit(full + (bar_empty - bar_full));
                    } else {
                        const uint32_t gbuf = tmem_addr(tmem, 0, Cfg::ACOL0 + buf * Cfg::N1);
#pragma unroll
                        for (int ks = 0; ks < Cfg::NKS; ++ks) {
                            if constexpr (Cfg::SRC == kTf32Rows16)
                                umma_f16_ss(gbuf, umma_desc_plus(a0, at + a_step(ks)), umma_desc_plus(p0, at + ks * P_STEP), idesc_gather, ks != 0);
                            else
                                umma_tf32_ss(gbuf, umma_desc_plus(a0, at + a_step(ks)), umma_desc_plus(p0, at + ks * P_STEP), idesc_gather, ks != 0);
                        }
                        tc_commit(bar_gdone + buf * 8);
                        if (GW == 1) { if (++buf == NBUF) buf = 0; }
                        else buf = (buf + GW) % NBUF;
                    }
                    at += GW * (Cfg::STAGE_BYTES / 16);
                    full += GW * 8;
                    if (GW == 1) {
                        if (full == bar_full + STAGES * 8) { full = bar_full; at = 0; parity ^= 1; }
                    } else if (full >= bar_full + STAGES * 8) { full -= STAGES * 8; at -= STAGES * (Cfg::STAGE_BYTES / 16); parity ^= 1; }
                    TF_ADD(m_issue, t2);
            }
#ifdef NMSPMM_TF32_PROFILE
            TF_OUT(2, m_full); TF_OUT(3, m_free); TF_OUT(4, m_issue); TF_OUT(5, clock64() - m_start); if (warp == 1) { TF_OUT(8, 1); TF_OUT(9, n_win); }
#endif
            }
            if (!ok) atomicMax(g.status, kDevTimeoutMma);
            if (DIRECT) tc_commit(bar_acc);                // every MMA has completed: accumulators are final
        }
        __syncwarp();
    } else if (warp < FIRST_BUILDER) {
        // ------------------------------------------------------------------ product issuers
        if (!DIRECT && elect_one()) {
            constexpr uint32_t idesc_product = umma_idesc_tf32(128, VL, false);
            constexpr int VPI = QV / Cfg::PRODUCT_WARPS;   // vectors per issuer
            const int v_begin = (warp - FIRST_PRODUCT) * VPI, v_live = min(VPI, live_vecs / BPV - v_begin);
            const uint64_t b0 = umma_desc_mn_tf32(ring + Cfg::A_BYTES + v_begin * (BPV * WSP * 128), WSP * 128, 512);
            bool ok = true;
            uint32_t at = 0, empty = bar_empty;            // stage of step u, as a descriptor offset; its barrier
            uint32_t done_parity = 0;
            int buf = 0;
            if constexpr (Cfg::PAIRS) {
                auto products = [&](int u, int b) {
                    if (v_live > 0) {
                        const uint32_t gbuf = tmem_addr(tmem, 0, Cfg::ACOL0 + b * Cfg::N1 + v_begin * WSP), acc = tmem_addr(tmem, 0, v_begin * VL);
#pragma unroll
                        for (int v = 0; v < VPI; ++v) {
                            if (v < v_live) {
#pragma unroll
                                for (int gi = 0; gi < Cfg::G; ++gi)
                                    umma_tf32_ts(acc + v * VL, gbuf + v * WSP + gi * 8, umma_desc_plus(b0, at + v * (BPV * WSP * 8) + gi * 64),
                                                 idesc_product, (u | gi) != 0);
                            }
                        }
                        tc_commit(empty);
                    } else {
                        mbar_arrive(empty);
                    }
                    at += Cfg::STAGE_BYTES / 16;
                    empty += 8;
                    if (empty == bar_empty + STAGES * 8) { empty = bar_empty; at = 0; }
                };
                for (int u = 0; u < n_win; u += 2) {
                    ok = mbar_spin_bounded(bar_gdone + buf * 8, done_parity, abort_word);
                    if (!ok) break;
                    tc_fence_after_sync();
                    products(u, 2 * buf);
                    if (u + 1 < n_win) products(u + 1, 2 * buf + 1);
                    if (++buf == Cfg::NP) { buf = 0; done_parity ^= 1; }
                }
            } else {
                TF_DECL(c_gdone = 0, c_issue = 0);
                TF_T(c_start);
                for (int u = 0; u < n_win; ++u) {
                    TF_T(t0);
                    // (the step's B rows have landed: the gather was issued after their barrier had completed)
                    ok = mbar_spin_bounded(bar_gdone + buf * 8, done_parity, abort_word);
                    TF_ADD(c_gdone, t0);
                    if (!ok) break;
                    TF_T(t1);
                    tc_fence_after_sync();
                    if (v_live > 0) {
                        const uint32_t gbuf = tmem_addr(tmem, 0, Cfg::ACOL0 + buf * Cfg::N1 + v_begin * WSP), acc = tmem_addr(tmem, 0, v_begin * VL);
#pragma unroll
                        for (int v = 0; v < VPI; ++v) {
                            if (v < v_live) {
#pragma unroll
                                for (int gi = 0; gi < Cfg::G; ++gi)
                                    umma_tf32_ts(acc + v * VL, gbuf + v * WSP + gi * 8, umma_desc_plus(b0, at + v * (BPV * WSP * 8) + gi * 64),
                                                 idesc_product, (u | gi) != 0);
                            }
                        }
                        tc_commit(empty);                      // this half of the step's products has read the stage and the gather result
                    } else {
                        mbar_arrive(empty);                    // no vector of this half exists; the gather itself has completed
                    }
                    if (++buf == NBUF) { buf = 0; done_parity ^= 1; }
                    at += Cfg::STAGE_BYTES / 16;
                    empty += 8;
                    if (empty == bar_empty + STAGES * 8) { empty = bar_empty; at = 0; }
                    TF_ADD(c_issue, t1);
            }
#ifdef NMSPMM_TF32_PROFILE
            if (warp == FIRST_PRODUCT) { TF_OUT(6, c_gdone); TF_OUT(7, c_issue); TF_OUT(15, clock64() - c_start); }
#endif
            }
            if (!ok) atomicMax(g.status, kDevTimeoutMma);
            if (v_live > 0) tc_commit(bar_acc); else mbar_arrive(bar_acc);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ one-hot builders
        const int b = tid - FIRST_BUILDER * 32;
        const int quad = warp & 3;                         // TMEM lane quadrant this warp may touch
        bool alive = true;
        if (!DIRECT) {
            constexpr int GROUPS = Cfg::GROUPS;
            const int group = b / Cfg::NT, e = b % Cfg::NT;          // this thread keeps gathered column e of steps group, group + GROUPS, ...
            const int v = e / WSP, j = e % WSP;
            const bool has = e < Cfg::N1 && j < WS && v * BPV < live_vecs;
            const int q = (bj >> 5) + v * BPV, qs_shift = g.qs_shift;       // the (first) 32-column index list of vector v
            const int* dptr = g.D + ((static_cast<size_t>(q >> qs_shift) * g.W) << qs_shift) + (q & ((1 << qs_shift) - 1)) +
                              (static_cast<size_t>(j) << qs_shift);
            const int n_merged = (KW == 64) ? g.sched.n_win : (g.sched.n_win >> 1);
            const int* ciptr = (MODE == kModeHigh) ? g.cinfo + static_cast<size_t>(q >> qs_shift) * n_merged * 64 : nullptr;
            const uint32_t my_prev = prev_k + e;
            TF_DECL(b_empty = 0);
            // Index loads run ahead in registers: idx[] two to four turns (through column_info on the 64-k
            // format: k[] two turns behind them), each turn's value in a register of its own so that
            // nothing waits for a load before its turn.
            auto load_index = [&](int i) { return (has && i < n_win) ? __ldg(dptr + ((static_cast<size_t>(win0 + i) * WS) << qs_shift)) : 0; };
            auto load_k = [&](int i, int rank) {
                if constexpr (MODE != kModeHigh) return rank;
                const int m = (KW == 64) ? (win0 + i) : ((win0 + i) >> 1);
                return (has && i < n_win) ? __ldg(ciptr + static_cast<size_t>(m) * 64 + rank) : 0;
            };
            int idx[PD], kq[PD];
#pragma unroll
            for (int d = 0; d < PD; ++d) kq[d] = load_index(group + d * GROUPS);
#pragma unroll
            for (int d = 0; d < PD; ++d) idx[d] = load_index(group + (PD + d) * GROUPS);
#pragma unroll
            for (int d = 0; d < PD; ++d) kq[d] = load_k(group + d * GROUPS, kq[d]);
            for (int i0 = group; group < GROUPS && alive && i0 < n_win; i0 += PD * GROUPS) {
#pragma unroll
                for (int d = 0; d < PD; ++d) {
                    const int i = i0 + d * GROUPS;
                    if (i >= n_win || !alive) break;
                    int k = kq[d];
                    kq[d] = load_k(i + PD * GROUPS, idx[d]);
                    idx[d] = load_index(i + 2 * PD * GROUPS);
                    if (MODE == kModeHigh && KW == 32) k -= ((win0 + i) & 1) * 32;
                    const int s = i % STAGES;
                    if (i >= STAGES) {
                        TF_T(t1);
                        const bool ok = mbar_wait_bounded(bar_empty + s * 8, ((i / STAGES) - 1) & 1, abort_word);
                        TF_ADD(b_empty, t1);
                        if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
                    }
                    if (has) {
                        const uint32_t ps = ring + s * Cfg::STAGE_BYTES + Cfg::A_BYTES + Cfg::B_BYTES;
                        const int old = lds_s8(my_prev + s * 128);
                        if constexpr (Cfg::SRC == kTf32Rows16) {
                            if (old >= 0) sts_u16(ps + p16_offset<KW>(e, old), 0u);
                            sts_u16(ps + p16_offset<KW>(e, k), a_form == kDtypeBF16 ? 0x3F80u : 0x3C00u);      // 1.0
                        } else {
                            if (old >= 0) sts_f32(ps + p_offset<KW>(e, old), 0.f);
                            sts_f32(ps + p_offset<KW>(e, k), 1.f);
                        }
                        sts_s8(my_prev + s * 128, k);
                    }
                    fence_proxy_async();                   // the tensor core reads P through the asynchronous proxy
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_full + s * 8);
                }
            }
#ifdef NMSPMM_TF32_PROFILE
            (void)b_empty;
#endif
        }
        // ------------------------------------------------------------------ epilogue
        TF_T(e_start);
        bool ok = alive && mbar_wait_bounded(bar_acc, 0, abort_word);
        ok = __all_sync(0xffffffffu, ok);
        grid_launch_dependents();                          // only stores are left
        TF_T(e_go);
        if (ok) {
            tc_fence_after_sync();
            // every MMA has completed, so every TMA copy has landed and been read: the
            // stage ring is free and serves as the transposition patches
            constexpr int SHARES = Cfg::BUILDERS / 128, VPW = QT / SHARES;     // the warps of a quadrant share the vectors
            const int v0 = (warp - FIRST_BUILDER) / 4 * VPW;
            tf32_store_vectors<NS, C16>(tmem, quad, lane, v0, min(v0 + VPW, live_vecs), ring + (warp - FIRST_BUILDER) * kTf32PatchBytes, g,
                                        outs, bi, bj, sliced, slot);
        } else if (lane == 0) {
            atomicMax(g.status, kDevTimeoutMma);
        }
#ifdef NMSPMM_TF32_PROFILE
        if (b == 0) { TF_OUT(13, e_go - e_start); TF_OUT(14, clock64() - e_go); }
#endif
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, Cfg::TMEM_COLS);
    }
}

template <int NKEEP, int KW, int MODE, int QT, int VL, int SRC, bool C16>
static cudaError_t launch_tf32_from(const GemmArgs& a, const GemmOutputs& outs, int tiles, cudaStream_t st)
{
    using Cfg = Tf32Cfg<NKEEP, KW, MODE, QT, VL, SRC>;
    auto kernel = nm_gemm_tf32_kernel<NKEEP, KW, MODE, QT, VL, SRC, C16>;
    static bool configured[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && !configured[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    CUtensorMap map_a, map_b;
    const int K = a.sched.n_win * KW;
    const int lda = outs.lda ? outs.lda : a.M;             // a row-major caller's transposed copy is padded to 4 columns
    int a_form = (lda % 32 == 0) ? 1 : 0;
    if (SRC == kTf32Rows16) {
        a_form = outs.a_rows - 1;
        e = encode_tensor_map_rows16(&map_a, a.A, K, a.M, KW, 128);       // rows past M read as zeros
    } else if (SRC == kTf32Rows32) {
        e = encode_tensor_map_2d(&map_a, a.A, K, a.M, 32, 128, 2);
    } else {
        e = a_form ? encode_tensor_map_blocks32(&map_a, a.A, lda, K, KW, 4) : encode_tensor_map_2d(&map_a, a.A, lda, K, 32, KW, 1);
    }
    if (e != cudaSuccess) return e;
    e = encode_tensor_map_blocks32(&map_b, a.B, a.N, a.W, Cfg::WSP - (g_test_short_fill ? 1 : 0), QT);   // (test hook, see kernels.h)
    if (e != cudaSuccess) return e;
    return launch_overlapped(kernel, tiles, Cfg::THREADS, Cfg::SMEM_BYTES, st, a, map_a, map_b, outs, a_form);
}

template <int NKEEP, int KW, int MODE, int QT, int VL>
static cudaError_t launch_tf32(const GemmArgs& a, const GemmOutputs& outs, int tiles, cudaStream_t st)
{
    const bool c16 = outs.c_dtype != kDtypeF32;
    if (c16 && outs.n_out != 1) return cudaErrorInvalidValue;
    if (outs.a_rows == 0)                                  // 16-bit C: activations that had to be transposed ahead
        return c16 ? launch_tf32_from<NKEEP, KW, MODE, QT, VL, kTf32Cols, true>(a, outs, tiles, st)
                   : launch_tf32_from<NKEEP, KW, MODE, QT, VL, kTf32Cols, false>(a, outs, tiles, st);
    if (outs.a_rows == 1 + kDtypeF32)
        return c16 ? cudaErrorInvalidValue : launch_tf32_from<NKEEP, KW, MODE, QT, VL, kTf32Rows32, false>(a, outs, tiles, st);
    if constexpr (NKEEP != 32)
        return c16 ? launch_tf32_from<NKEEP, KW, MODE, QT, VL, kTf32Rows16, true>(a, outs, tiles, st) : cudaErrorInvalidValue;
    else
        return cudaErrorInvalidValue;
}

#define NMSPMM_TF32_VARIANT(NKEEP, KW, MODE, QT, VL)                                                                   \
    { NKEEP, Tf32Cfg<NKEEP, KW, MODE, QT, VL>::WS, KW, MODE, QT * 32, VL, Tf32Cfg<NKEEP, KW, MODE, QT, VL>::SMEM_BYTES,    \
      Tf32Cfg<NKEEP, KW, MODE, QT, VL>::STAGES, Tf32Cfg<NKEEP, KW, MODE, QT, VL>::THREADS, &launch_tf32<NKEEP, KW, MODE, QT, VL> }

extern const SlicedVariant kTf32GatherVariants[] = {
    NMSPMM_TF32_VARIANT(32, 32, kModeLow, 8, 32),  NMSPMM_TF32_VARIANT(32, 32, kModeLow, 4, 32),
    NMSPMM_TF32_VARIANT(16, 32, kModeLow, 8, 32),  NMSPMM_TF32_VARIANT(16, 32, kModeLow, 4, 32),
    NMSPMM_TF32_VARIANT(12, 32, kModeLow, 8, 32),  NMSPMM_TF32_VARIANT(12, 32, kModeLow, 4, 32),
    NMSPMM_TF32_VARIANT(8, 32, kModeLow, 8, 32),   NMSPMM_TF32_VARIANT(8, 32, kModeLow, 4, 32),
    NMSPMM_TF32_VARIANT(8, 32, kModeHigh, 8, 32),  NMSPMM_TF32_VARIANT(8, 32, kModeHigh, 4, 32),
    NMSPMM_TF32_VARIANT(4, 64, kModeHigh, 8, 32),  NMSPMM_TF32_VARIANT(4, 64, kModeHigh, 4, 32),
    NMSPMM_TF32_VARIANT(16, 32, kModeLow, 6, 32),  NMSPMM_TF32_VARIANT(12, 32, kModeLow, 6, 32),  NMSPMM_TF32_VARIANT(8, 32, kModeLow, 6, 32),
    NMSPMM_TF32_VARIANT(8, 32, kModeHigh, 6, 32),  NMSPMM_TF32_VARIANT(4, 64, kModeHigh, 6, 32),
    // vectors of 64 columns (two adjacent equal index lists): one gather and one N = 64 product per pair
    NMSPMM_TF32_VARIANT(16, 32, kModeLow, 8, 64),  NMSPMM_TF32_VARIANT(12, 32, kModeLow, 8, 64),
    NMSPMM_TF32_VARIANT(8, 32, kModeLow, 8, 64),   NMSPMM_TF32_VARIANT(8, 32, kModeHigh, 8, 64),
    NMSPMM_TF32_VARIANT(4, 64, kModeHigh, 8, 64),
};
extern const int kTf32GatherVariantCount = sizeof(kTf32GatherVariants) / sizeof(kTf32GatherVariants[0]);

#ifdef NMSPMM_TF32_PROFILE
// Diagnostic build only: reads and clears the phase counters.
extern "C" int nmspmm_debug_tf32_profile(unsigned long long* out16)
{
    if (cudaMemcpyFromSymbol(out16, g_tf32_profile, sizeof(unsigned long long) * 16) != cudaSuccess) return 1;
    unsigned long long zero[16] = {};
    return cudaMemcpyToSymbol(g_tf32_profile, zero, sizeof(zero)) == cudaSuccess ? 0 : 1;
}
#endif

}  // namespace nmspmm
