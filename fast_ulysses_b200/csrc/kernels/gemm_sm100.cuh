#pragma once
// Persistent, warp-specialised bf16 GEMM cores for sm_100a: D[M,N] = A[M,K] * B[N,K]^T with fp32
// accumulation in tensor memory. Either operand may instead be given with the contraction along
// its rows (A stored K x M, B stored K x N, "MN-major"): the weight gradient of a linear layer
// contracts over the tokens and reads dY and X as they lie in memory, without a transposed copy.
//
//   run_wide    one or two blocks of 256 rows and up to 256 columns per pair of CTAs: what is large enough to occupy the device
//   run_small   128 x 128 tiles on single CTAs: what is not, and what is short enough
//   run         128 x 256 tiles on single CTAs, A gathered from the peers by extra warps while the GEMM runs
//
// In each, warp 0 is the TMA producer (128B-swizzled operand tiles into a ring of shared-memory
// stages; of one operand where run_wide has a warp for each), warp 1 issues tcgen05.mma, and the other warps are the epilogue: they read the accumulator
// from tensor memory (each warp may touch one 32-lane quarter) and apply the epilogue functor. Tiles are
// visited in bands of M-tiles so that a wave of CTAs shares operand tiles through L2. No TMA load is
// multicast; every CTA fetches its own tiles. Kernels that write peers' memory from the epilogue run
// their handshake through `Epi::open` / `Epi::close`.
#include <cuda.h>
#include <cuda_bf16.h>

#include "handshake.cuh"
#include "ptx.cuh"

#include <type_traits>

namespace fu {
namespace gemm {

constexpr int BM       = 128;
constexpr int BN       = 256;
constexpr int BK       = 64;   // one 128-byte swizzle atom of bf16
constexpr int UMMA_K   = 16;
constexpr int STAGES   = 4;
constexpr int A_BYTES  = BM * BK * 2;
constexpr int B_BYTES  = BN * BK * 2;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int SMEM_BYTES  = STAGES * STAGE_BYTES + 1024;  // + slack to align the ring to 1024 B
constexpr int THREADS  = 192;
constexpr int BAND     = 16;   // M-tiles per rasterisation band
constexpr int TMEM_COLS = 512;

enum : uint32_t {
    ERR_NONE = 0,
    ERR_PRODUCER_WAIT = 1,
    ERR_MMA_WAIT_FULL = 2,
    ERR_MMA_WAIT_TMEM = 3,
    ERR_EPI_WAIT      = 4,
};

struct Core {
    CUtensorMap map_a;
    CUtensorMap map_b;
    int         M, N, K;
    int         tiles_m, tiles_n;
    uint32_t*   err;
};

__device__ __forceinline__ void tile_coords(const Core& c, int t, int& mt, int& nt)
{
    const int band_tiles = BAND * c.tiles_n;
    const int band       = t / band_tiles;
    const int r          = t - band * band_tiles;
    const int rows       = min(BAND, c.tiles_m - band * BAND);
    nt                   = r / rows;
    mt                   = band * BAND + (r - nt * rows);
}

__device__ __forceinline__ void flag_error(const Core& c, uint32_t code)
{
    if (c.err) {
        atomicCAS(c.err, 0u, code);
    }
}

// `Src::ready(mt, kb)` runs in the producer thread before the loads of K-block
// `kb` of M-tile `mt` are issued and may wait (bounded) for that part of A to exist; it returns
// false to give up. `Aux::run(aux_warp, lane)` is executed by `Aux::kWarps` extra warps (warps 6..)
// alongside the GEMM, e.g. to pull A from peers' memory into the buffer the GEMM reads.
// Epi requirements:
//   __device__ void open(int epi_warp)                       once, before the first tile
//   __device__ void tile(uint32_t tmem_acc, int mt, int nt, int quarter, int lane)
//   __device__ void close(int epi_tid)                       once, after the last tile (all 128 threads)
template <class Epi, class Src, class Aux>
__device__ __forceinline__ void run(const Core& core, Epi& epi, Src src, Aux aux)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t       full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2];
    __shared__ uint32_t       tmem_holder;

    const uint32_t base = (ptx::smem_addr(smem_raw) + 1023u) & ~1023u;
    uint8_t*       ring = smem_raw + (base - ptx::smem_addr(smem_raw));
    const int      warp = static_cast<int>(ptx::uniform(threadIdx.x >> 5));
    const int      lane = threadIdx.x & 31;
    const int      total_tiles = core.tiles_m * core.tiles_n;
    const int      kblocks     = (core.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            ptx::mbar_init(&tmem_full[a], 1);
            ptx::mbar_init(&tmem_empty[a], 4);
        }
        ptx::mbar_fence_init();
        ptx::tma_prefetch_desc(&core.map_a);
        ptx::tma_prefetch_desc(&core.map_b);
    }
    if (warp == 1) {
        ptx::tmem_alloc<TMEM_COLS>(&tmem_holder);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = ptx::uniform(tmem_holder);

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            bool     ok = true;
            for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
                int mt, nt;
                tile_coords(core, t, mt, nt);
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int      s      = it % STAGES;
                    const uint32_t parity = ((it / STAGES) & 1u) ^ 1u;
                    if (!ptx::mbar_wait(&empty[s], parity) || !src.ready(mt, kb)) {
                        flag_error(core, ERR_PRODUCER_WAIT);
                        ok = false;
                        break;
                    }
                    uint8_t* sa = ring + s * STAGE_BYTES;
                    uint8_t* sb = sa + A_BYTES;
                    ptx::mbar_expect_tx(&full[s], STAGE_BYTES);
                    ptx::tma_load_2d(sa, &core.map_a, kb * BK, mt * BM, &full[s]);
                    ptx::tma_load_2d(sb, &core.map_b, kb * BK, nt * BN, &full[s]);
                }
            }
        }
        __syncwarp();
    }
    else if (warp == 1) {
        const uint32_t  leader = ptx::elect_one();
        const uint32_t  idesc  = ptx::make_idesc(1, 1, BM, BN, 0, 0);
        const ptx::Desc a_desc(ptx::smem_desc_sw128(base, 16u, 1024)), b_desc(ptx::smem_desc_sw128(base + A_BYTES, 16u, 1024));
        const uint32_t  full_b = ptx::smem_addr(full), empty_b = ptx::smem_addr(empty);
        const uint32_t  tfull_b = ptx::smem_addr(tmem_full), tempty_b = ptx::smem_addr(tmem_empty);
        uint32_t        stage = 0, phase = 0, tcount = 0;
        uint32_t        gave_up = ERR_NONE;
        for (int t = blockIdx.x; t < total_tiles && !gave_up; t += gridDim.x, ++tcount) {
            const uint32_t acc = tcount & 1u;
            if (!ptx::mbar_wait_warp(tempty_b + acc * 8, ((tcount >> 1) & 1u) ^ 1u)) {
                gave_up = ERR_MMA_WAIT_TMEM;
                break;
            }
            ptx::tc_fence_after();
            for (int kb = 0; kb < kblocks; ++kb) {
                if (!ptx::mbar_wait_warp(full_b + stage * 8, phase)) {
                    gave_up = ERR_MMA_WAIT_FULL;
                    break;
                }
                ptx::tc_fence_after();
                const ptx::Desc a = a_desc.at(stage * STAGE_BYTES), b = b_desc.at(stage * STAGE_BYTES);
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k) {
                    ptx::mma_f16_ss_if<1>(tmem_base + acc * BN, a.at(32 * k), b.at(32 * k), idesc, static_cast<uint32_t>(kb | k), leader);
                }
                ptx::mma_commit_if<1>(empty_b + stage * 8, leader);
                if (++stage == STAGES) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            if (!gave_up) {
                ptx::mma_commit_if<1>(tfull_b + acc * 8, leader);
            }
        }
        if (gave_up) {
            flag_error(core, gave_up);
        }
        __syncwarp();
    }
    else if (warp >= 6) {
        aux.run(warp - 6, lane);
    }
    else {
        const int epi_warp = warp - 2;
        const int quarter  = warp & 3;  // the TMEM lane quarter this warp may access
        epi.open(epi_warp);
        uint32_t tcount = 0;
        bool     ok     = true;
        for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++tcount) {
            const uint32_t acc = tcount & 1u;
            if (!ptx::mbar_wait(&tmem_full[acc], (tcount >> 1) & 1u)) {
                flag_error(core, ERR_EPI_WAIT);
                ok = false;
                break;
            }
            ptx::tc_fence_after();
            int mt, nt;
            tile_coords(core, t, mt, nt);
            epi.tile(tmem_base + acc * BN + (static_cast<uint32_t>(quarter * 32) << 16), mt, nt, quarter, lane);
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                ptx::mbar_arrive(&tmem_empty[acc]);
            }
        }
        epi.close(threadIdx.x - 64);
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tmem_dealloc<TMEM_COLS>(tmem_base);
    }
}

// ---- work units of the cores below --------------------------------------------------------------------
// Both cores hand their epilogue 32 rows x 128 columns at a time ("a unit": one warp, one row per
// thread, the whole row of 128 fp32 in registers) and give the accumulator back to the MMA thread as
// soon as the registers are loaded, before any arithmetic or store. Epi requirements:
//   static constexpr bool kPeers          whether open() / close() run (kernels that touch peers)
//   void fetch(int col0, int lane)        before a unit's products are waited for: what can be read ahead
//   void open(int epi_tid), close(int epi_tid)          all epilogue threads, once before / after the tiles
//   void unit(uint32_t (&r)[128], int row0, int col0, int col_end, int lane, uint32_t stage)
//   void unit(uint32_t (&r)[64], ...)     the same of half as many columns, for run_small with 64 columns a warp
// Columns from `col_end` on are not the unit's. `stage` is the address of 4 KiB of shared memory of this warp's own (32 rows x 128 bytes).
constexpr int UNIT_STAGE_BYTES = 32 * 128;

template <int COLS>
__device__ __forceinline__ void load_unit(uint32_t taddr, uint32_t (&r)[COLS])
{
#pragma unroll
    for (int ch = 0; ch < COLS / 32; ++ch) {
        ptx::tmem_ld_32x32(taddr + ch * 32, *reinterpret_cast<uint32_t(*)[32]>(&r[ch * 32]));
    }
    ptx::tmem_ld_wait();
}

// ---- the GEMM on CTA pairs, two accumulator blocks per pair ---------------------------------------------
// A pair of CTAs (one cluster, tcgen05.mma.cta_group::2) owns MB x NB blocks of 256 x 256 outputs,
// MB * NB = 2: 512 x 256 or 256 x 512. Per 64-wide K-block a CTA loads its own 128 rows of A per block
// row and its own 128 rows of B per block column (48 KiB; four stages), and the even CTA's thread issues
// 2 x 4 MMAs of 256 x 256 x 16 over both CTAs' shared memory. All 512 tensor-memory columns hold
// accumulators.
//
// Why two blocks: shared memory moves 128 bytes a clock per SM. An MMA of 256 x 256 x 16 takes 128
// clocks and reads 4 KiB of A and 4 KiB of B from each SM (64 B/clk); with one block per pair TMA has to
// write 32 KiB per 512 clocks beside it (64 B/clk), all the bandwidth there is, with two blocks 48 KiB
// per 1024 (48 B/clk).
//
// Measured at 8192 cubed with operands of zeros (no power limit; SM clock 1965 MHz): 0.548 ms, 0.84 of the
// tensor pipe's rate (cuBLAS 0.523). The same kernel with its MMAs issued by one lane on its own took
// 0.753: see ptx.cuh, elect_one(). Random operands, back to back for seconds (1000 W power cap): 1330 -
// 1390 TFLOP/s on the feed-forward shapes, 9450 x 13824 x 5120 and its relatives (cuBLAS 1320 - 1430; the
// 128 x 256 single-CTA tiles before this kernel 1120 - 1200).
//
// A block may be narrower, `width` = 32 .. 256 columns in steps of 32, so that a problem of a few waves fills the last
// one, and a pair may own a single block (MB = NB = 1, whose accumulators alternate between the halves of tensor
// memory), for the same reason and because it hides the whole epilogue: with two blocks the second waits in
// tensor memory for the first one's arithmetic and stores, and the next tile behind it (6729 x 7632 x 2592 with a
// residual: 205 us with two, 184 with one). A narrow or single block makes less of each byte in
// shared memory, see block_clocks(); at the power limit that decides, see choose_shape().
//
// With two blocks there is no second accumulator buffer, so the blocks' order hides what it can of the epilogue, the reads
// of tensor memory: the first kStages K-blocks of a tile are multiplied into block 0 and then into block 1, and so are the
// last ones. Block 0 is finished (and read out) four stages before block 1, and the next tile can start in
// block 0 while block 1 is still being read out.
constexpr int WIDE_STAGES      = 4;  // of 48 KiB; six of 32 KiB with one block per pair
constexpr int WIDE_BLOCK_BYTES = 128 * BK * 2;  // 128 rows of one operand, one K-block
constexpr int WIDE_STAGE_BYTES = 3 * WIDE_BLOCK_BYTES;
constexpr int WIDE_EPI_WARPS   = 8;
constexpr int WIDE_FIRST_EPI   = 4;  // warp 3 is idle: it fills the first warpgroup, whose registers go to the others
constexpr int WIDE_B_WARP      = 2;  // the second operand's producer
constexpr int WIDE_THREADS     = 32 * (WIDE_FIRST_EPI + WIDE_EPI_WARPS);
constexpr int WIDE_REGS_LIGHT  = 88;   // 128 x 88 + 256 x 208 = the 384 x 168 of the launch
constexpr int WIDE_REGS_EPI    = 208;  // a unit's 128 values, a row of loads in flight, addresses
constexpr int WIDE_SMEM_BYTES  = WIDE_STAGES * WIDE_STAGE_BYTES + WIDE_EPI_WARPS * UNIT_STAGE_BYTES + 1024;
constexpr int WIDE_BAND_ROWS   = 4096;  // rows per rasterisation band: a wave of 74 tiles is roughly square

// Tiles are visited in bands of `band` M-tiles so that a wave of CTAs shares operand tiles through L2.
__device__ __forceinline__ void pair_tile_coords(int tiles_m, int tiles_n, int band_rows, int t, int& mt, int& nt)
{
    const int band_tiles = band_rows * tiles_n;
    const int band       = t / band_tiles;
    const int r          = t - band * band_tiles;
    const int rows       = min(band_rows, tiles_m - band * band_rows);
    nt                   = r / rows;
    mt                   = band * band_rows + (r - nt * rows);
}

// SPLIT: what whole waves leave over. A cluster of two or four pairs takes one block, each pair a part of its
// K-blocks; the CTAs with the same rows add up their sums as run_small's do, 256 / pairs columns each.
//
// The schedule: `full` whole tiles, then the remaining tiles block by block (two items each), which the
// host asks for when half as many items as pairs are left, so that the last wave is half as long.
struct WideCore {
    CUtensorMap map_a, map_b;
    int         M, N, K;
    int         tiles_m, tiles_n;  // of MB * 256 x NB * width
    int         width;             // columns of a block
    int         full, items;
    int         first;             // split kernel: the item of cluster 0
    int         a_mn, b_mn;
    int         overlap;           // the next kernel may come up beside this one, see host_util.h: launch_behind
    uint32_t*   err;
};

__device__ __forceinline__ void flag_error(uint32_t* err, uint32_t code)
{
    if (err) {
        atomicCAS(err, 0u, code);
    }
}

// `n`: how many items this pair has had before.
template <int MB, int NB>
struct WideItem {
    int m0, n0, u0, u1, width;
    __device__ __forceinline__ WideItem(const WideCore& c, int item, uint32_t n) : width(c.width)
    {
        const bool whole = MB * NB == 1 || item < c.full;
        const int  rest  = item - c.full;
        int        mt, nt;
        pair_tile_coords(c.tiles_m, c.tiles_n, WIDE_BAND_ROWS / (MB * 256), whole ? item : c.full + (rest >> 1), mt, nt);
        m0 = mt * MB * 256;
        n0 = nt * NB * width;
        if (MB * NB == 1) {
            u0 = n & 1u;
            u1 = u0 + 1;
            return;
        }
        u0 = whole ? 0 : (rest & 1);
        u1 = whole ? 2 : u0 + 1;
        // a block that lies outside the result altogether is not computed
        if (u1 == 2 && (MB == 2 ? m0 + 256 >= c.M : n0 + width >= c.N)) {
            u1 = 1;
        }
        if (u0 == 1 && (MB == 2 ? m0 + 256 >= c.M : n0 + width >= c.N)) {
            u1 = u0;  // empty
        }
    }
    __device__ __forceinline__ int row(int u) const { return m0 + (MB == 2 ? u * 256 : 0); }
    __device__ __forceinline__ int col(int u) const { return n0 + (NB == 2 ? u * width : 0); }
};

template <int MB, int NB, bool SPLIT, class Epi>
__device__ __forceinline__ void run_wide(const WideCore& core, Epi& epi)
{
    static_assert(MB * NB <= 2, "tensor memory holds two blocks of 256 x 256");
    constexpr int STAGES      = MB * NB == 2 ? WIDE_STAGES : WIDE_STAGES * 3 / 2;
    constexpr int STAGE_BYTES = (MB + NB) * WIDE_BLOCK_BYTES;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t       full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2];
    __shared__ uint32_t       tmem_holder;

    const uint32_t base = (ptx::smem_addr(smem_raw) + 1023u) & ~1023u;
    uint8_t*       ring = smem_raw + (base - ptx::smem_addr(smem_raw));
    const int      warp = static_cast<int>(ptx::uniform(threadIdx.x >> 5));
    const int      lane = threadIdx.x & 31;
    const int      crank = static_cast<int>(ptx::uniform(ptx::cluster_ctarank()));
    const int      csize = SPLIT ? static_cast<int>(ptx::uniform(ptx::cluster_nctarank())) : 2;
    const int      half  = crank & 1;  // 0: issues the MMAs; 1: the other rows
    const int      part = crank >> 1, parts = csize >> 1;
    const uint32_t even = static_cast<uint32_t>(crank & ~1);  // the pair's issuing CTA
    const int      all_kb = (core.K + BK - 1) / BK, share = SPLIT ? (all_kb + parts - 1) / parts : all_kb;
    const int      kb_0 = part * share, kblocks = SPLIT ? min(share, all_kb - kb_0) : all_kb;  // this pair's K-blocks
    const int      w_0 = SPLIT ? core.first + static_cast<int>(blockIdx.x) / csize : static_cast<int>(blockIdx.x >> 1);
    const int      w_end = SPLIT ? w_0 + 1 : core.items, w_inc = SPLIT ? 1 : static_cast<int>(gridDim.x >> 1);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], 1);
        }
        for (int u = 0; u < 2; ++u) {
            ptx::mbar_init(&tmem_full[u], 1);
            ptx::mbar_init(&tmem_empty[u], 2 * WIDE_EPI_WARPS);  // the epilogue warps of both CTAs
        }
        ptx::mbar_fence_init();
        ptx::tma_prefetch_desc(&core.map_a);
        ptx::tma_prefetch_desc(&core.map_b);
    }
    ptx::cluster_sync();  // both CTAs' barriers exist before either signals the other's
    if (warp == 1) {
        ptx::tmem_alloc_pair<TMEM_COLS>(&tmem_holder);
        ptx::tmem_relinquish_pair();
    }
    ptx::tc_fence_before();
    ptx::grid_wait();
    __syncthreads();
    if (core.overlap) {
        ptx::grid_trigger();  // with this CTA's tensor memory in hand
    }
    ptx::tc_fence_after();
    const uint32_t tmem_base = ptx::uniform(tmem_holder);

    if (warp < WIDE_FIRST_EPI) {
    ptx::setmaxnreg_dec<WIDE_REGS_LIGHT>();
    const uint32_t leader = ptx::elect_one();
    const uint32_t full_b = ptx::smem_addr(full), empty_b = ptx::smem_addr(empty);
    // With one block, whose K-block's products may take no more than 192 clocks, each operand has a producer of its own, and both look
    // at the next stage while they load this one: blocks of 128 and 96 columns 8 % faster on average, up to 30. Two blocks have
    // 1024 clocks a K-block and lose 1 % so.
    constexpr bool OPERAND_WARPS = MB * NB == 1;
    if (warp == 0 || (OPERAND_WARPS && warp == WIDE_B_WARP)) {
        const bool a_op = !OPERAND_WARPS || warp == 0, b_op = !OPERAND_WARPS || warp != 0;
        uint32_t   stage = 0, phase = 1;
        bool       ok = true, ready = false;
        // of an operand's 128 rows (or, stored the other way, two 64 x 64 blocks) B may need only a part
        const int      b_rows  = core.width / 2;
        const uint32_t b_bytes = core.b_mn ? (b_rows + 63) / 64 * 8192u : b_rows * 128u;
        for (int w = w_0; w < w_end && ok; w += w_inc) {
            const WideItem<MB, NB> item(core, w, 0);
            if (item.u0 == item.u1) {
                continue;
            }
            const uint32_t bytes = (MB == 2 ? item.u1 - item.u0 : 1) * WIDE_BLOCK_BYTES + (NB == 2 ? item.u1 - item.u0 : 1) * b_bytes;
            for (int kb = 0; kb < kblocks; ++kb) {
                if (!ready && !ptx::mbar_wait_warp(empty_b + stage * 8, phase)) {
                    ok = false;
                    break;
                }
                const uint32_t next = stage + 1 == STAGES ? 0 : stage + 1, next_phase = next == 0 ? phase ^ 1u : phase;
                const uint32_t ahead = OPERAND_WARPS ? ptx::mbar_test(empty_b + next * 8, next_phase) : 0u;
                const uint32_t sa = base + stage * STAGE_BYTES, sb = sa + MB * WIDE_BLOCK_BYTES, bar = full_b + stage * 8;
                if (a_op) {
                    if (half == 0) {
                        ptx::mbar_expect_tx_if(bar, 2 * bytes, leader);  // both operands' bytes of both CTAs
                    }
#pragma unroll
                    for (int u = 0; u < MB; ++u) {
                        if (MB == 2 && (u < item.u0 || u >= item.u1)) {
                            continue;
                        }
                        const int      m  = item.m0 + u * 256 + half * 128;
                        const uint32_t to = sa + u * WIDE_BLOCK_BYTES;
                        if (!core.a_mn) {
                            ptx::tma_load_2d_pair_if(to, &core.map_a, (kb_0 + kb) * BK, m, bar, leader);
                        }
                        else {  // 64 (k) x 64 (m) blocks of 8 KiB
                            ptx::tma_load_2d_pair_if(to, &core.map_a, m, (kb_0 + kb) * BK, bar, leader);
                            ptx::tma_load_2d_pair_if(to + 8192, &core.map_a, m + 64, (kb_0 + kb) * BK, bar, leader);
                        }
                    }
                }
                if (b_op) {
#pragma unroll
                    for (int u = 0; u < NB; ++u) {
                        if (NB == 2 && (u < item.u0 || u >= item.u1)) {
                            continue;
                        }
                        const int      n  = item.col(u) + half * b_rows;
                        const uint32_t to = sb + u * WIDE_BLOCK_BYTES;
                        if (!core.b_mn) {
                            ptx::tma_load_2d_pair_if(to, &core.map_b, (kb_0 + kb) * BK, n, bar, leader);
                        }
                        else {
                            ptx::tma_load_2d_pair_if(to, &core.map_b, n, (kb_0 + kb) * BK, bar, leader);
                            if (b_rows > 64) {
                                ptx::tma_load_2d_pair_if(to + 8192, &core.map_b, n + 64, (kb_0 + kb) * BK, bar, leader);
                            }
                        }
                    }
                }
                stage = next;
                phase = next_phase;
                ready = ptx::all_ready(ahead);
            }
        }
        if (!ok) {
            flag_error(core.err, ERR_PRODUCER_WAIT);
        }
        __syncwarp();
    }
    else if (warp == 1) {
        if (half == 0) {
            const uint32_t  idesc = ptx::make_idesc(1, 1, 256, core.width, core.a_mn ? 1 : 0, core.b_mn ? 1 : 0);
            // K-major: 16 bf16 along K are 32 bytes inside the swizzle atom. MN-major: 16 rows of K are
            // 2048 bytes, 64-column blocks 8 KiB apart.
            const uint32_t  a_step = core.a_mn ? 2048u : 32u, b_step = core.b_mn ? 2048u : 32u;
            const ptx::Desc a_desc(ptx::smem_desc_sw128(base, core.a_mn ? 8192u : 16u, 1024));
            const ptx::Desc b_desc(ptx::smem_desc_sw128(base + MB * WIDE_BLOCK_BYTES, core.b_mn ? 8192u : 16u, 1024));
            const uint32_t  tfull_b = ptx::smem_addr(tmem_full), tempty_b = ptx::smem_addr(tmem_empty);
            uint32_t        stage = 0, phase = 0, uses0 = 0, uses1 = 0;
            uint32_t        gave_up = ERR_NONE;
            const uint32_t  both = 3u << even;
            auto issue = [&](int u, uint32_t s, uint32_t accumulate) {  // one K-block into block u
                const ptx::Desc a = a_desc.at(s * STAGE_BYTES + (MB == 2 ? u * WIDE_BLOCK_BYTES : 0));
                const ptx::Desc b = b_desc.at(s * STAGE_BYTES + (NB == 2 ? u * WIDE_BLOCK_BYTES : 0));
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k) {
                    ptx::mma_f16_ss_if<2>(tmem_base + u * 256, a.at(a_step * k), b.at(b_step * k), idesc, accumulate | k, leader);
                }
            };
            auto advance = [](uint32_t& s, uint32_t& ph) {
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            };
            for (int w = w_0; w < w_end && !gave_up; w += w_inc) {
                const WideItem<MB, NB> item(core, w, uses0 + uses1);
                if (item.u0 == item.u1) {
                    continue;
                }
                for (int kb = 0; kb < kblocks && !gave_up;) {
                    const int left = kblocks - kb;
                    if (kb > 0 && left > STAGES && item.u1 - item.u0 == 2) {
                        // the middle of a whole tile: both blocks, one K-block after another
                        const int n = left - STAGES;
                        for (int i = 0; i < n; ++i) {
                            if (!ptx::mbar_wait_warp(full_b + stage * 8, phase)) {
                                gave_up = ERR_MMA_WAIT_FULL;
                                break;
                            }
                            ptx::tc_fence_after();
                            issue(0, stage, 1u);
                            issue(1, stage, 1u);
                            ptx::mma_commit_if<2>(empty_b + stage * 8, leader, both);
                            advance(stage, phase);
                        }
                        kb += n;
                        continue;
                    }
                    // the first K-blocks of a tile, its last ones, or any of a single block
                    const int run = min(left, STAGES);
                    uint32_t  s = stage, ph = phase;
                    for (int u = item.u0; u < item.u1 && !gave_up; ++u) {
                        if (kb == 0) {
                            uint32_t& uses = u == 0 ? uses0 : uses1;
                            if (!ptx::mbar_wait_warp_cluster(tempty_b + u * 8, (uses & 1u) ^ 1u)) {
                                gave_up = ERR_MMA_WAIT_TMEM;
                                break;
                            }
                            ++uses;
                            ptx::tc_fence_after();
                        }
                        s  = stage;
                        ph = phase;
                        for (int i = 0; i < run; ++i) {
                            if (u == item.u0) {
                                if (!ptx::mbar_wait_warp(full_b + s * 8, ph)) {
                                    gave_up = ERR_MMA_WAIT_FULL;
                                    break;
                                }
                                ptx::tc_fence_after();
                            }
                            issue(u, s, static_cast<uint32_t>(kb | i));
                            if (u + 1 == item.u1) {
                                ptx::mma_commit_if<2>(empty_b + s * 8, leader, both);
                            }
                            advance(s, ph);
                        }
                        if (!gave_up && run == left) {
                            ptx::mma_commit_if<2>(tfull_b + u * 8, leader, both);
                        }
                    }
                    stage = s;
                    phase = ph;
                    kb += run;
                }
            }
            if (gave_up) {
                flag_error(core.err, gave_up);
            }
        }
        __syncwarp();
    }
    if (SPLIT) {  // the epilogue warps' exchange
        ptx::cluster_sync();
        ptx::cluster_sync();
    }
    }
    else {
        ptx::setmaxnreg_inc<WIDE_REGS_EPI>();
        const int epi_warp = warp - WIDE_FIRST_EPI;
        const int quarter  = warp & 3;        // the TMEM lane quarter this warp may access
        const int cg       = epi_warp >> 2;   // which 128 of a block's 256 columns
        const uint32_t stage = base + STAGES * STAGE_BYTES + epi_warp * UNIT_STAGE_BYTES;
        if (Epi::kPeers) {
            epi.open(threadIdx.x - 32 * WIDE_FIRST_EPI);
        }
        if constexpr (SPLIT) {
            const WideItem<MB, NB> item(core, w_0, 0);
            const int              width = 256 / parts;
            bool                   ok    = item.u0 != item.u1;  // an empty item only takes part in the barriers
            if (ok) {
                epi.fetch(item.col(item.u0) + part * width + cg * (width / 2), lane);
            }
            if (ok && !ptx::mbar_wait(&tmem_full[item.u0], 0u)) {
                flag_error(core.err, ERR_EPI_WAIT);
                ok = false;
            }
            ptx::tc_fence_after();
            const uint32_t taddr = tmem_base + item.u0 * 256 + (static_cast<uint32_t>(quarter * 32) << 16);
            const uint32_t slot  = base + quarter * 32768 + lane * 16;  // this warp's rows: [columns / 4][lane] of 16 bytes per pair
            ptx::cluster_sync();  // every pair's products are complete: its stages may be overwritten
#pragma unroll 1
            for (int ch = 0; ok && ch < 8; ++ch) {
                const int      col = cg * 128 + ((ch + 2 * part) & 7) * 16, owner = col / width;
                const uint32_t dst = ptx::cluster_addr(slot + (part * width + col - owner * width) * 128, owner * 2 + half);
                uint32_t       r[16];
                ptx::tmem_ld_32x16(taddr + col, r);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    ptx::st_cluster_v4(dst + g * 512, r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
                }
            }
            ptx::cluster_sync();
            auto finish = [&](auto w) {
                constexpr int W = decltype(w)::value;
                float         v[W];
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    v[k] = 0.0f;
                }
#pragma unroll 1
                for (int from = 0; from < parts; ++from) {
#pragma unroll
                    for (int g = 0; g < W / 4; ++g) {
                        const uint4 q = ptx::ld_shared_v4(slot + (from * 2 * W + cg * W + g * 4) * 128);
                        v[4 * g] += __uint_as_float(q.x);
                        v[4 * g + 1] += __uint_as_float(q.y);
                        v[4 * g + 2] += __uint_as_float(q.z);
                        v[4 * g + 3] += __uint_as_float(q.w);
                    }
                }
                epi.template piece<W>(v, item.row(item.u0) + half * 128 + quarter * 32, item.col(item.u0) + (2 * part + cg) * W, core.N, lane, stage);
            };
            if (ok) {
                if (parts == 2) {
                    finish(std::integral_constant<int, 64>{});
                }
                else {
                    finish(std::integral_constant<int, 32>{});
                }
            }
        }
        else {
        uint32_t uses[2] = {0, 0};
        bool     ok      = true;
        for (int w = w_0; w < w_end && ok; w += w_inc) {
            const WideItem<MB, NB> item(core, w, uses[0] + uses[1]);
            const int              cols = core.width / 2, col0 = cg * cols;  // a warp's share of a block
            for (int u = item.u0; u < item.u1; ++u) {
                epi.fetch(item.col(u) + col0, lane);
                if (!ptx::mbar_wait(&tmem_full[u], uses[u] & 1u)) {
                    flag_error(core.err, ERR_EPI_WAIT);
                    ok = false;
                    break;
                }
                ++uses[u];
                ptx::tc_fence_after();
                uint32_t r[128];
                load_unit(tmem_base + u * 256 + col0 + (static_cast<uint32_t>(quarter * 32) << 16), r);
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    ptx::mbar_arrive_cluster(ptx::cluster_addr(&tmem_empty[u], even));
                }
                epi.unit(r, item.row(u) + half * 128 + quarter * 32, item.col(u) + col0, item.col(u) + col0 + cols, lane, stage);
            }
        }
        }
        if (Epi::kPeers) {
            epi.close(threadIdx.x - 32 * WIDE_FIRST_EPI);
        }
    }

    // Neither CTA may free its tensor memory, or leave, while the other can still signal it or
    // read its shared memory.
    ptx::tc_fence_before();
    ptx::cluster_sync();
    if (warp == 1) {
        ptx::tmem_dealloc_pair<TMEM_COLS>(tmem_base);
    }
}

// ---- the GEMM on single CTAs, 128 x 128 tiles -------------------------------------------------------------
// For problems with too few 256 x 256 blocks to occupy the device: four times as many tiles, a short
// epilogue, and nothing shared between SMs. Bound by shared memory (its MMAs read 128 B/clk by
// themselves) at about half the tensor pipe's rate, which a problem of this size does not reach anyway.
// The two halves of the tensor memory in use alternate between tiles.
//
// SPLIT: the CTAs of a cluster (2, 4 or 8) take a part of the K-blocks of one tile each, for problems whose
// tiles leave SMs idle. They add up their fp32 sums through distributed shared memory, every CTA 128 / size
// columns of the tile in the order of the CTAs, and each finishes and writes its columns.
constexpr int SMALL_STAGES      = 6;
constexpr int SMALL_STAGE_BYTES = 2 * WIDE_BLOCK_BYTES;
// A warp of the epilogue takes 32 rows and `cols` columns of a tile. 64 where nothing speaks against it: a launch of one tile a CTA waits
// for the whole epilogue. 78 products on single tiles 6 % faster than with 128, 68 x 13304 x 128 with the GELU's derivative 8.1 -> 6.2 us,
// 2985 x 5360 x 480 with GELU 28.2 -> 22.6. 128 where a head is needed at once, and in clusters, whose CTAs have 64 columns or fewer
// to finish and lose 0.2 us by the larger block.
constexpr int small_epi_warps(int cols) { return 4 * 128 / cols; }
constexpr int small_threads(int cols) { return 32 * (2 + small_epi_warps(cols)); }
constexpr int small_smem_bytes(int cols) { return SMALL_STAGES * SMALL_STAGE_BYTES + small_epi_warps(cols) * UNIT_STAGE_BYTES + 1024; }

template <bool SPLIT, int COLS, class Epi>
__device__ __forceinline__ void run_small(const WideCore& core, Epi& epi)
{
    static_assert(!SPLIT || COLS == 128, "a warp finishes all of a CTA's columns of a shared tile");
    constexpr int EPI_WARPS = small_epi_warps(COLS);
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t       full[SMALL_STAGES], empty[SMALL_STAGES], tmem_full[2], tmem_empty[2];
    __shared__ uint32_t       tmem_holder;

    const uint32_t base = (ptx::smem_addr(smem_raw) + 1023u) & ~1023u;
    uint8_t*       ring = smem_raw + (base - ptx::smem_addr(smem_raw));
    const int      warp = static_cast<int>(ptx::uniform(threadIdx.x >> 5));
    const int      lane = threadIdx.x & 31;
    const int      tiles   = core.tiles_m * core.tiles_n;  // of 128 x 128 here
    const int      kblocks = (core.K + BK - 1) / BK;
    const int      csize   = SPLIT ? static_cast<int>(ptx::uniform(ptx::cluster_nctarank())) : 1;
    const int      crank   = SPLIT ? static_cast<int>(ptx::uniform(ptx::cluster_ctarank())) : 0;
    const int      share   = SPLIT ? (kblocks + csize - 1) / csize : kblocks;
    const int      kb_0 = crank * share, kb_n = SPLIT ? min(kblocks, kb_0 + share) : kblocks;  // this CTA's K-blocks
    const int      t_0 = SPLIT ? blockIdx.x / csize : blockIdx.x, t_inc = SPLIT ? gridDim.x / csize : gridDim.x;

    if (warp == 0 && lane == 0) {
        ptx::tma_prefetch_desc(&core.map_a);
        ptx::tma_prefetch_desc(&core.map_b);
        for (int s = 0; s < SMALL_STAGES; ++s) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            ptx::mbar_init(&tmem_full[a], 1);
            ptx::mbar_init(&tmem_empty[a], EPI_WARPS);
        }
        ptx::mbar_fence_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc<256>(&tmem_holder);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    ptx::grid_wait();
    __syncthreads();
    if (core.overlap) {
        ptx::grid_trigger();  // with this CTA's tensor memory in hand
    }
    ptx::tc_fence_after();
    const uint32_t tmem_base = ptx::uniform(tmem_holder);
    const uint32_t leader = ptx::elect_one();
    const uint32_t full_b = ptx::smem_addr(full), empty_b = ptx::smem_addr(empty);

    if (warp == 0) {
        // The next stage is looked at while this one's loads are issued: looked at only on coming to it, a K-block took the producer
        // 390 clocks instead of 310, and the products take 256 (256 x 256 x 4096 15.5 -> 13.6 us, 120 x 5120 x 5120 14.8 -> 13.1). With a
        // producer for each operand it is 270, but the seventh warp costs a launch 0.1 - 0.3 us: over 210 sizes nothing gained.
        uint32_t stage = 0, phase = 1;
        bool     ok = true, ready = false;
        for (int t = t_0; t < tiles && ok; t += t_inc) {
            int mt, nt;
            pair_tile_coords(core.tiles_m, core.tiles_n, 16, t, mt, nt);
            for (int kb = kb_0; kb < kb_n; ++kb) {
                if (!ready && !ptx::mbar_wait_warp(empty_b + stage * 8, phase)) {
                    ok = false;
                    break;
                }
                const uint32_t next = stage + 1 == SMALL_STAGES ? 0 : stage + 1, next_phase = next == 0 ? phase ^ 1u : phase;
                const uint32_t ahead = ptx::mbar_test(empty_b + next * 8, next_phase);
                const uint32_t sa = base + stage * SMALL_STAGE_BYTES, sb = sa + WIDE_BLOCK_BYTES, bar = full_b + stage * 8;
                ptx::mbar_expect_tx_if(bar, SMALL_STAGE_BYTES, leader);
                if (!core.a_mn) {
                    ptx::tma_load_2d_if(sa, &core.map_a, kb * BK, mt * 128, bar, leader);
                }
                else {
                    ptx::tma_load_2d_if(sa, &core.map_a, mt * 128, kb * BK, bar, leader);
                    ptx::tma_load_2d_if(sa + 8192, &core.map_a, mt * 128 + 64, kb * BK, bar, leader);
                }
                if (!core.b_mn) {
                    ptx::tma_load_2d_if(sb, &core.map_b, kb * BK, nt * 128, bar, leader);
                }
                else {
                    ptx::tma_load_2d_if(sb, &core.map_b, nt * 128, kb * BK, bar, leader);
                    ptx::tma_load_2d_if(sb + 8192, &core.map_b, nt * 128 + 64, kb * BK, bar, leader);
                }
                stage = next;
                phase = next_phase;
                ready = ptx::all_ready(ahead);
            }
        }
        if (!ok) {
            flag_error(core.err, ERR_PRODUCER_WAIT);
        }
        __syncwarp();
    }
    else if (warp == 1) {
        const uint32_t  idesc  = ptx::make_idesc(1, 1, 128, 128, core.a_mn ? 1 : 0, core.b_mn ? 1 : 0);
        const uint32_t  a_step = core.a_mn ? 2048u : 32u, b_step = core.b_mn ? 2048u : 32u;
        const ptx::Desc a_desc(ptx::smem_desc_sw128(base, core.a_mn ? 8192u : 16u, 1024));
        const ptx::Desc b_desc(ptx::smem_desc_sw128(base + WIDE_BLOCK_BYTES, core.b_mn ? 8192u : 16u, 1024));
        const uint32_t  tfull_b = ptx::smem_addr(tmem_full), tempty_b = ptx::smem_addr(tmem_empty);
        uint32_t        stage = 0, phase = 0, tcount = 0;
        uint32_t        gave_up = ERR_NONE;
        for (int t = t_0; t < tiles && !gave_up; t += t_inc, ++tcount) {
            const uint32_t acc = tcount & 1u;
            if (!ptx::mbar_wait_warp(tempty_b + acc * 8, ((tcount >> 1) & 1u) ^ 1u)) {
                gave_up = ERR_MMA_WAIT_TMEM;
                break;
            }
            ptx::tc_fence_after();
            for (int kb = kb_0; kb < kb_n; ++kb) {
                if (!ptx::mbar_wait_warp(full_b + stage * 8, phase)) {
                    gave_up = ERR_MMA_WAIT_FULL;
                    break;
                }
                ptx::tc_fence_after();
                const ptx::Desc a = a_desc.at(stage * SMALL_STAGE_BYTES), b = b_desc.at(stage * SMALL_STAGE_BYTES);
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k) {
                    ptx::mma_f16_ss_if<1>(tmem_base + acc * 128, a.at(a_step * k), b.at(b_step * k), idesc,
                                          static_cast<uint32_t>((kb - kb_0) | k), leader);
                }
                ptx::mma_commit_if<1>(empty_b + stage * 8, leader);
                if (++stage == SMALL_STAGES) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            if (!gave_up) {
                ptx::mma_commit_if<1>(tfull_b + acc * 8, leader);
            }
        }
        if (gave_up) {
            flag_error(core.err, gave_up);
        }
        __syncwarp();
    }
    else {
        const int epi_warp = warp - 2;
        const int quarter  = warp & 3;
        const int cg       = epi_warp >> 2;  // which COLS of the tile's columns
        const uint32_t stage = base + SMALL_STAGES * SMALL_STAGE_BYTES + epi_warp * UNIT_STAGE_BYTES;
        if (Epi::kPeers) {
            epi.open(threadIdx.x - 64);
        }
        uint32_t tcount = 0;
        for (int t = t_0; t < tiles; t += t_inc, ++tcount) {
            const uint32_t acc = tcount & 1u;
            int            mt, nt;
            pair_tile_coords(core.tiles_m, core.tiles_n, 16, t, mt, nt);
            epi.fetch(nt * 128 + (SPLIT ? crank * (128 / csize) : cg * COLS), lane);
            const bool ok = ptx::mbar_wait(&tmem_full[acc], (tcount >> 1) & 1u);
            if (!ok) {
                flag_error(core.err, ERR_EPI_WAIT);
            }
            if constexpr (SPLIT) {  // one tile per cluster; also after a timeout: the other CTAs wait in its barriers
                ptx::tc_fence_after();
                const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
                const int      row0 = mt * 128 + quarter * 32, width = 128 / csize;
                const uint32_t slot = base + quarter * 16384 + lane * 16;  // this warp's rows: [columns / 4][lane] of 16 bytes per CTA
                ptx::cluster_sync();  // every CTA's products are complete: its stages may be overwritten
#pragma unroll 1
                for (int ch = 0; ch < 8; ++ch) {  // the next CTA's columns first, so that not all write to one
                    const int      col = (ch * 16 + (crank + 1) * width) & 127, owner = col / width;
                    const uint32_t dst = ptx::cluster_addr(slot + (crank * width + col - owner * width) * 128, owner);
                    uint32_t       r[16];
                    ptx::tmem_ld_32x16(taddr + col, r);
                    ptx::tmem_ld_wait();
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        ptx::st_cluster_v4(dst + g * 512, r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
                    }
                }
                ptx::cluster_sync();
                auto finish = [&](auto w) {
                    constexpr int W = decltype(w)::value;
                    float         v[W];
#pragma unroll
                    for (int k = 0; k < W; ++k) {
                        v[k] = 0.0f;
                    }
#pragma unroll 1
                    for (int from = 0; from < csize; ++from) {
#pragma unroll
                        for (int g = 0; g < W / 4; ++g) {
                            const uint4 q = ptx::ld_shared_v4(slot + (from * W + g * 4) * 128);
                            v[4 * g] += __uint_as_float(q.x);
                            v[4 * g + 1] += __uint_as_float(q.y);
                            v[4 * g + 2] += __uint_as_float(q.z);
                            v[4 * g + 3] += __uint_as_float(q.w);
                        }
                    }
                    epi.template piece<W>(v, row0, nt * 128 + crank * W, core.N, lane, stage);
                };
                if (ok) {
                    if (csize == 2) {
                        finish(std::integral_constant<int, 64>{});
                    }
                    else if (csize == 4) {
                        finish(std::integral_constant<int, 32>{});
                    }
                    else {
                        finish(std::integral_constant<int, 16>{});
                    }
                }
                break;
            }
            if (!ok) {
                break;
            }
            ptx::tc_fence_after();
            uint32_t r[COLS];
            load_unit(tmem_base + acc * 128 + cg * COLS + (static_cast<uint32_t>(quarter * 32) << 16), r);
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                ptx::mbar_arrive(&tmem_empty[acc]);
            }
            epi.unit(r, mt * 128 + quarter * 32, nt * 128 + cg * COLS, nt * 128 + (cg + 1) * COLS, lane, stage);
        }
        if (Epi::kPeers) {
            epi.close(threadIdx.x - 64);
        }
    }

    if (SPLIT && warp < 2) {  // the epilogue warps' exchange
        ptx::cluster_sync();
        ptx::cluster_sync();
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tmem_dealloc<256>(tmem_base);
    }
}

// ---- W columns of a unit through the staging buffer -----------------------------------------------------------
// A thread holds a row, so its global accesses would be 32 scattered pieces per instruction. They go
// through the warp's staging buffer instead: W / 8 lanes move the W columns of one row (eight lanes and 128
// bytes for half a unit). 16-byte units are XOR-swizzled by the row: neither side has bank conflicts. All
// accesses of a lane are in flight together: with each store waiting for its load, writing a unit out took
// 3700 clocks, most of a small GEMM's time.
__device__ __forceinline__ uint32_t stage_unit(uint32_t stage, int row, int unit)
{
    return stage + row * 128 + ((unit ^ (row & 7)) << 4);
}

// 32 rows x W columns of a bf16 matrix into the staging buffer; what lies outside reads as zero.
template <int W>
__device__ __forceinline__ void stage_in(uint32_t stage, const __nv_bfloat16* src, int64_t ld, int row0, int col0, int M, int N,
                                         int lane)
{
    constexpr int U = W / 8, ROWS = 32 / U;  // lanes a row, rows an access
    const int     unit = lane % U, col = col0 + unit * 8, first = lane / U;
    uint4         v[U];
    if (row0 + 32 <= M && col0 + W <= N) {  // warp-uniform
        const __nv_bfloat16* p = src + static_cast<int64_t>(row0 + first) * ld + col;
#pragma unroll
        for (int i = 0; i < U; ++i) {
            v[i] = *reinterpret_cast<const uint4*>(p + i * ROWS * ld);
        }
    }
    else if ((N - col0) % 8 == 0) {  // uniform: whole units or none
        const __nv_bfloat16* p = src + static_cast<int64_t>(row0 + first) * ld + col;
#pragma unroll
        for (int i = 0; i < U; ++i) {
            v[i] = make_uint4(0u, 0u, 0u, 0u);
            if (row0 + i * ROWS + first < M && col < N) {
                v[i] = *reinterpret_cast<const uint4*>(p + i * ROWS * ld);
            }
        }
    }
    else {
#pragma unroll
        for (int i = 0; i < U; ++i) {
            const int row = row0 + i * ROWS + first;
            v[i]          = make_uint4(0u, 0u, 0u, 0u);
            if (row < M) {
                const __nv_bfloat16* p = src + static_cast<int64_t>(row) * ld + col;
                if (col + 8 <= N) {
                    v[i] = *reinterpret_cast<const uint4*>(p);
                }
                else if (col < N) {
                    __nv_bfloat16 e[8] = {};
                    for (int j = 0; j < N - col; ++j) {
                        e[j] = p[j];
                    }
                    v[i] = *reinterpret_cast<const uint4*>(e);
                }
            }
        }
    }
    __syncwarp();  // the buffer's previous contents have been read
#pragma unroll
    for (int i = 0; i < U; ++i) {
        ptx::st_shared_v4(stage_unit(stage, i * ROWS + first, unit), v[i]);
    }
    __syncwarp();
}

// The rows of the staging buffer to a bf16 matrix. The caller's threads have each written their row.
template <int W>
__device__ __forceinline__ void stage_out(uint32_t stage, __nv_bfloat16* dst, int64_t ld, int row0, int col0, int M, int N,
                                          int lane)
{
    constexpr int U = W / 8, ROWS = 32 / U;
    const int     unit = lane % U, col = col0 + unit * 8, first = lane / U;
    uint4         v[U];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < U; ++i) {
        v[i] = ptx::ld_shared_v4(stage_unit(stage, i * ROWS + first, unit));
    }
    __syncwarp();  // the buffer may be refilled
    if (row0 + 32 <= M && col0 + W <= N) {  // warp-uniform
        __nv_bfloat16* p = dst + static_cast<int64_t>(row0 + first) * ld + col;
#pragma unroll
        for (int i = 0; i < U; ++i) {
            ptx::st_v4(p + i * ROWS * ld, v[i]);
        }
        return;
    }
    if ((N - col0) % 8 == 0) {  // uniform: whole units or none
        __nv_bfloat16* p = dst + static_cast<int64_t>(row0 + first) * ld + col;
#pragma unroll
        for (int i = 0; i < U; ++i) {
            if (row0 + i * ROWS + first < M && col < N) {
                ptx::st_v4(p + i * ROWS * ld, v[i]);
            }
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
        const int row = row0 + i * ROWS + first;
        if (row < M) {
            __nv_bfloat16* p = dst + static_cast<int64_t>(row) * ld + col;
            if (col + 8 <= N) {
                ptx::st_v4(p, v[i]);
            }
            else if (col < N) {
                const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (j < N - col) {
                        p[j] = __ushort_as_bfloat16(static_cast<unsigned short>(w[j >> 1] >> (16 * (j & 1))));
                    }
                }
            }
        }
    }
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// All `threads` epilogue threads of a CTA.
__device__ __forceinline__ void epi_barrier(int threads)
{
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

}  // namespace gemm
}  // namespace fu
