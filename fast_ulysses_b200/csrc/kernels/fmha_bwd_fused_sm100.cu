// Non-causal flash attention backward for head_dim 128: one software-pipelined pass on tcgen05.
//
// One persistent CTA per SM owns a 128-row K/V block of one (batch, head) at a time and sweeps all
// 128-row query blocks i. Five products per block pair, everything transposed so that the kv row
// sits on the TMEM lane axis and the probabilities can be fed back as the A operand:
//   S^T(i)  = K Q_i^T            (SS)      C1: P^T = exp2(S^T c - lse)               -> TMEM (bf16)
//   dP^T(i) = V dO_i^T           (SS)      C2: dS^T = P^T o (dP^T - delta)           -> TMEM + smem
//   dV     += P^T dO_i           (A from TMEM)
//   dK     += dS^T Q_i           (A from TMEM)
//   dQ_i^T  = K^T dS^T           (SS, both operands MN-major); drained by eight extra warps with
//                                coalesced fp32 reductions into a global accumulator
// Tensor memory: S^T/P^T | dP^T/dS^T/dQ^T | dV | dK, 128 fp32 columns each (all 512).
//
// Issue order per block: dP(i), dV(i), S(i+1), dK(i), dQ(i). C1(i+1) runs under dK(i) and dQ(i),
// C2(i) under dV(i) and S(i+1). dP(i+1) is the first product that needs the columns of dQ_i^T back:
// the drain warps copy them to registers, release the columns at once and only then issue their
// reductions, which overlap the next block. The softmax scale is applied to dK in the epilogue and
// to dQ when the accumulator is rounded, not to every element of dS.
//
// Measured limits (S = 32768, 5 heads, SM clock counter): a 128x128x16 MMA takes 64 clocks when its
// descriptors are ready (8 per product: 512), a tensor-memory load-and-wait about 200, and the fp32
// reductions of all SMs together move 6.1 TB/s into L2 whatever their width (64 KiB per block: 3130
// clocks). The dependent chain dP -> C2 -> dK, dQ -> drain -> dP sets the period, about 3700 clocks against
// the 2560 of the products. With random operands the power limit lowers the clock below that. 37888 tokens x 4 heads: 4.83 ms with
// zeros, with random numbers 5.91 in a launch by itself and 6.78 in launches repeated for seconds. With one thing as it was before (ms with
// zeros; all of them 5.12, 6.09, 6.99 and a chain of 4050): statistics read one value at a time 5.14, dS stored eight registers at a time
// 5.11, P in one piece 4.93, arithmetic that is not packed 4.85, the check for kv rows that do not exist in the inner loop 4.85.
// Tried and no faster: dK begun on the first
// half of dS, the products issued by three warps, paced issue, a share of the exponentials on the FMA pipe.
// Warps: 0 = TMA producer, 1 = MMA issuer, 2..9 = two threads per kv row, 10..17 = dQ drain.
#include "cluster_plan.h"
#include "fu_kernels.h"
#include "host_util.h"
#include "ptx.cuh"
#include "tma_host.h"

#include <cuda_bf16.h>

#include <algorithm>

namespace {

using namespace fu;

constexpr int D           = 128;
constexpr int BLK         = 128;
constexpr int TILE_BYTES  = BLK * D * 2;  // 32 KiB
constexpr int HALF_BYTES  = TILE_BYTES / 2;
constexpr int STAGES      = 2;
constexpr int OFF_K       = 0;
constexpr int OFF_V       = OFF_K + TILE_BYTES;
constexpr int OFF_Q       = OFF_V + TILE_BYTES;            // STAGES tiles
constexpr int OFF_DO      = OFF_Q + STAGES * TILE_BYTES;   // STAGES tiles
constexpr int OFF_DS      = OFF_DO + STAGES * TILE_BYTES;  // dS^T, [kv x q], 128B-swizzled halves
constexpr int OFF_STATS   = OFF_DS + TILE_BYTES;           // per stage: lse2[128] | delta[128]
constexpr int OFF_BARS    = OFF_STATS + STAGES * 1024;
constexpr int SMEM_BYTES  = OFF_BARS + 256;
constexpr int THREADS     = 576;

static_assert(SMEM_BYTES <= 232448, "shared memory budget");

enum : uint32_t { ERR_ALIGN = 30, ERR_LOAD = 31, ERR_MMA = 32, ERR_COMPUTE = 33, ERR_DRAIN = 34 };

struct Params {
    CUtensorMap    map_q, map_k, map_v, map_do;
    const float*   lse2;    // (B, H, Sq_pad) log-sum-exp in base 2, +inf in the padding
    const float*   delta;   // (B, H, Sq_pad)
    float*         dq_acc;  // (B, Sq, H, 128) fp32, zeroed by the launcher
    __nv_bfloat16* dk;
    __nv_bfloat16* dv;
    int64_t        dk_row, dk_head, dk_batch, dv_row, dv_head, dv_batch;
    int            B, H, Sq, Skv, Sq_pad;
    int            n_q, kv_blocks, total_work;
    int            first;  // split kernel: the item of cluster 0
    int            overlap;  // the next kernel may come up beside this one
    float          scale, scale_log2;
    uint32_t*      err;
    uint64_t*      trace;
};

struct Bars {
    uint64_t kv_full, kv_empty;
    uint64_t q_full[STAGES], do_full[STAGES], empty[STAGES];
    uint64_t s_full, dp_full, p_ready, ds_ready, dq_full, dq_free, acc_full, acc_free;
    uint32_t tmem_holder;
};
static_assert(sizeof(Bars) <= 256, "barrier block");

__device__ __forceinline__ void flag(const Params& p, uint32_t code)
{
    if (p.err) {
        atomicCAS(p.err, 0u, code);
    }
}

__device__ __forceinline__ void stamp(const Params& p, uint32_t it, int ev)
{
    if (p.trace && blockIdx.x == 0 && (threadIdx.x & 31u) == 0u && it >= 64u && it < 72u) {
        p.trace[(it - 64u) * 16 + ev] = clock64();
    }
}

// CTAs that run at the same time own neighbouring K/V blocks of one head. Each starts its sweep
// over the query blocks at a different block, so that their dQ reductions do not all land on the
// same addresses at the same moment.
__device__ __forceinline__ int first_block(const Params& p, int jb, int n_q)
{
    return static_cast<int>(static_cast<int64_t>(jb) * n_q / p.kv_blocks);
}

__device__ __forceinline__ void red_add(float* addr, float v)
{
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(v) : "memory");
}

// 16 query columns of S^T -> 8 packed probability pairs. All threads of a warp want the same statistics, and a shared-memory
// load takes a turn of the memory that the products read their operands from whatever its width: four values each.
template <int C>
__device__ __forceinline__ void c1_chunk(const uint32_t (&r)[16], uint32_t (&pk)[32], const float* lse2, float c)
{
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 l = *reinterpret_cast<const float4*>(lse2 + C * 16 + 4 * k);
        float        t0, t1, t2, t3;  // the exponents, negated
        ptx::fma2(t0, t1, __uint_as_float(r[4 * k]), __uint_as_float(r[4 * k + 1]), -c, -c, l.x, l.y);
        ptx::fma2(t2, t3, __uint_as_float(r[4 * k + 2]), __uint_as_float(r[4 * k + 3]), -c, -c, l.z, l.w);
        pk[C * 8 + 2 * k]     = ptx::pack_bf16x2(ptx::ex2(-t0), ptx::ex2(-t1));
        pk[C * 8 + 2 * k + 1] = ptx::pack_bf16x2(ptx::ex2(-t2), ptx::ex2(-t3));
    }
}

// Stores half H of a row's probabilities over the scores, which have been read; kv rows that do not exist have none.
template <int H>
__device__ __forceinline__ void store_p(uint32_t t_s, uint32_t (&pk)[32], bool tail, bool kv_ok)
{
    if (tail && !kv_ok) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            pk[H * 16 + k] = 0u;
        }
    }
    ptx::tmem_st_32x16(t_s + H * 16, reinterpret_cast<const uint32_t(&)[16]>(pk[H * 16]));
}

// 16 query columns of dP^T -> 8 packed dS pairs (without the softmax scale), into the swizzled shared-memory row and over the
// first columns that this thread has already read, four at a time: with both stores behind all eight the registers that wait
// for them cost 4 %.
template <int C>
__device__ __forceinline__ void c2_chunk(const uint32_t (&r)[16], const uint32_t (&pk)[32], const float* delta,
                                         uint32_t t_dp, uint8_t* ds_row, int row_in)
{
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        uint32_t dd[4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            // the difference in fp32 (it cancels), the product with the bf16 probabilities as a packed pair
            const float4 l = *reinterpret_cast<const float4*>(delta + C * 16 + 8 * k + 4 * j);
            float        d0, d1, d2, d3;
            ptx::fma2(d0, d1, l.x, l.y, -1.0f, -1.0f, __uint_as_float(r[8 * k + 4 * j]), __uint_as_float(r[8 * k + 4 * j + 1]));
            ptx::fma2(d2, d3, l.z, l.w, -1.0f, -1.0f, __uint_as_float(r[8 * k + 4 * j + 2]), __uint_as_float(r[8 * k + 4 * j + 3]));
            dd[2 * j]     = ptx::mul_bf16x2(pk[C * 8 + 4 * k + 2 * j], ptx::pack_bf16x2(d0, d1));
            dd[2 * j + 1] = ptx::mul_bf16x2(pk[C * 8 + 4 * k + 2 * j + 1], ptx::pack_bf16x2(d2, d3));
        }
        *reinterpret_cast<uint4*>(ds_row + (((2 * C + k) ^ (row_in & 7)) << 4)) = make_uint4(dd[0], dd[1], dd[2], dd[3]);
        ptx::tmem_st_32x4(t_dp + C * 8 + k * 4, dd);
    }
}

// 32 columns of one accumulator row, rounded
__device__ __forceinline__ void store_row32(__nv_bfloat16* dst, const float (&v)[32], float scale)
{
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        uint4 a;
        a.x = ptx::pack_bf16x2(v[8 * k] * scale, v[8 * k + 1] * scale);
        a.y = ptx::pack_bf16x2(v[8 * k + 2] * scale, v[8 * k + 3] * scale);
        a.z = ptx::pack_bf16x2(v[8 * k + 4] * scale, v[8 * k + 5] * scale);
        a.w = ptx::pack_bf16x2(v[8 * k + 6] * scale, v[8 * k + 7] * scale);
        *reinterpret_cast<uint4*>(dst + 8 * k) = a;
    }
}

// The end of an item whose query blocks were shared by the CTAs of a cluster: each holds its part of the
// sums dV and dK. They are cut into 32 units of 32 rows x 32 columns, four to each element-wise warp, and
// dealt to the CTAs in turn; every CTA sends the others' units of its own sums through distributed
// shared memory, so that all send, receive and write at once, and adds the parts up in the order of the
// CTAs. The Q and dO tiles are done with by then: units received lie at their place, each as eight
// rows of 32 x 16 bytes, so that a warp's store covers 512 contiguous bytes. Executed by the
// element-wise warps; the others take part in the two cluster barriers.
constexpr int UNITS      = 32;
constexpr int UNIT_BYTES = 32 * 32 * 4;
static_assert(30 * UNIT_BYTES <= 2 * STAGES * TILE_BYTES, "exchange area: (CTAs - 1) x units of a CTA, at most 30 for up to 8 CTAs");

__device__ __forceinline__ void join_shares(const Params& p, uint32_t base, uint32_t t_dv, uint32_t t_dk, int warp_in, int lane, int crank,
                                            int csize, __nv_bfloat16* dv, __nv_bfloat16* dk, bool kv_ok)
{
    ptx::tc_fence_after();
    const int      per  = (UNITS + csize - 1) / csize;
    const uint32_t area = base + OFF_Q + lane * 16;
    const int      c2   = warp_in >> 2;
    ptx::cluster_sync();  // every CTA's products are complete: its Q and dO tiles may be overwritten
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const int u = warp_in * 4 + i, owner = u % csize;
        if (owner == crank) {
            continue;
        }
        const int      slot = (crank - (crank > owner ? 1 : 0)) * per + u / csize;
        const uint32_t dst  = ptx::cluster_addr(area + slot * UNIT_BYTES, owner);
        uint32_t       r[32];
        ptx::tmem_ld_32x32((i < 2 ? t_dv : t_dk) + (2 * c2 + (i & 1)) * 32, r);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            ptx::st_cluster_v4(dst + g * 512, r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
        }
    }
    ptx::cluster_sync();
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const int u = warp_in * 4 + i, ch = 2 * c2 + (i & 1);
        if (u % csize != crank) {
            continue;
        }
        float acc[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            acc[k] = 0.0f;
        }
#pragma unroll 1
        for (int r = 0; r < csize; ++r) {
            if (r == crank) {
                uint32_t own[32];
                ptx::tmem_ld_32x32((i < 2 ? t_dv : t_dk) + ch * 32, own);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < 32; ++k) {
                    acc[k] += __uint_as_float(own[k]);
                }
            }
            else {
                const uint32_t src = area + ((r - (r > crank ? 1 : 0)) * per + u / csize) * UNIT_BYTES;
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    const uint4 v = ptx::ld_shared_v4(src + g * 512);
                    acc[4 * g] += __uint_as_float(v.x);
                    acc[4 * g + 1] += __uint_as_float(v.y);
                    acc[4 * g + 2] += __uint_as_float(v.z);
                    acc[4 * g + 3] += __uint_as_float(v.w);
                }
            }
        }
        if (kv_ok) {
            store_row32((i < 2 ? dv : dk) + ch * 32, acc, i < 2 ? 1.0f : p.scale);
        }
    }
}

// SPLIT: one item per cluster, each CTA its share of the query blocks.
template <bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1) fmha_bwd_fused_kernel(const __grid_constant__ Params p)
{
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t base = ptx::smem_addr(sm);
    Bars&          bar  = *reinterpret_cast<Bars*>(sm + OFF_BARS);
    const int      warp = static_cast<int>(ptx::uniform(threadIdx.x >> 5));
    const int      lane = threadIdx.x & 31;
    if (base & 1023u) {
        if (threadIdx.x == 0) {
            flag(p, ERR_ALIGN);
        }
        return;
    }

    if (threadIdx.x == 0) {
        ptx::mbar_init(&bar.kv_full, 1);
        ptx::mbar_init(&bar.kv_empty, 1);
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(&bar.q_full[s], 1);
            ptx::mbar_init(&bar.do_full[s], 1);
            ptx::mbar_init(&bar.empty[s], 1);
        }
        ptx::mbar_init(&bar.s_full, 1);
        ptx::mbar_init(&bar.dp_full, 1);
        ptx::mbar_init(&bar.p_ready, 8);  // one arrival per warp
        ptx::mbar_init(&bar.ds_ready, 8);  // one arrival per warp
        ptx::mbar_init(&bar.dq_full, 1);
        ptx::mbar_init(&bar.dq_free, 8);  // one arrival per warp
        ptx::mbar_init(&bar.acc_full, 1);
        ptx::mbar_init(&bar.acc_free, 8);  // one arrival per warp
        ptx::mbar_fence_init();
        ptx::tma_prefetch_desc(&p.map_q);
        ptx::tma_prefetch_desc(&p.map_k);
        ptx::tma_prefetch_desc(&p.map_v);
        ptx::tma_prefetch_desc(&p.map_do);
    }
    if (warp == 1) {
        ptx::tmem_alloc<512>(&bar.tmem_holder);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    ptx::grid_wait();
    __syncthreads();
    if (p.overlap) {
        ptx::grid_trigger();  // with this CTA's tensor memory in hand
    }
    ptx::tc_fence_after();
    const uint32_t tmem = ptx::uniform(bar.tmem_holder);
    const int      crank = SPLIT ? static_cast<int>(ptx::uniform(ptx::cluster_ctarank())) : 0;
    const int      csize = SPLIT ? static_cast<int>(ptx::uniform(ptx::cluster_nctarank())) : 1;
    const int      w_0   = SPLIT ? p.first + static_cast<int>(blockIdx.x) / csize : static_cast<int>(blockIdx.x);
    const int      w_end = SPLIT ? w_0 + 1 : p.total_work;
    const int      w_inc = SPLIT ? 1 : static_cast<int>(gridDim.x);
    const int      share = (p.n_q + csize - 1) / csize;
    const int      i_lo  = crank * share;  // this CTA's query blocks: i_lo .. i_lo + n_q
    const int      n_q   = min(share, p.n_q - i_lo);

    // The first two roles are run by the whole warp, see ptx.cuh: elect_one().
    const uint32_t leader = ptx::elect_one();
    auto           b_of   = [](uint64_t& x) { return ptx::smem_addr(&x); };
    if (warp == 0) {
        // ---------------------------------------------------------------- producer
        uint32_t s = 0, ph = 1, wc = 0;
        bool     ok = true;
        for (int w = w_0; w < w_end && ok; w += w_inc, ++wc) {
            const int jb = w % p.kv_blocks;
            const int h  = (w / p.kv_blocks) % p.H;
            const int b  = w / (p.kv_blocks * p.H);
            if (!ptx::mbar_wait_warp(b_of(bar.kv_empty), (wc & 1u) ^ 1u)) {
                ok = false;
                break;
            }
            ptx::mbar_expect_tx_if(b_of(bar.kv_full), 2 * TILE_BYTES, leader);
            for (int half = 0; half < 2; ++half) {
                ptx::tma_load_4d_if(base + OFF_K + half * HALF_BYTES, &p.map_k, half * 64, jb * BLK, h, b, b_of(bar.kv_full), leader);
                ptx::tma_load_4d_if(base + OFF_V + half * HALF_BYTES, &p.map_v, half * 64, jb * BLK, h, b, b_of(bar.kv_full), leader);
            }
            const float* lse2  = p.lse2 + (static_cast<int64_t>(b) * p.H + h) * p.Sq_pad;
            const float* delta = p.delta + (static_cast<int64_t>(b) * p.H + h) * p.Sq_pad;
            int          i     = first_block(p, jb, n_q);
            for (int i0 = 0; i0 < n_q; ++i0) {
                const uint32_t ss = base + OFF_STATS + s * 1024, qf = b_of(bar.q_full[0]) + s * 8, df = b_of(bar.do_full[0]) + s * 8;
                // one release per stage (after dK of the block that used it): the statistics of
                // a stage are read by the element-wise warps until then
                if (!ptx::mbar_wait_warp(b_of(bar.empty[0]) + s * 8, ph)) {
                    ok = false;
                    break;
                }
                ptx::mbar_expect_tx_if(qf, TILE_BYTES + 512, leader);
                for (int half = 0; half < 2; ++half) {
                    ptx::tma_load_4d_if(base + OFF_Q + s * TILE_BYTES + half * HALF_BYTES, &p.map_q, half * 64, (i_lo + i) * BLK, h, b, qf,
                                        leader);
                }
                ptx::bulk_g2s_if(ss, lse2 + (i_lo + i) * BLK, 512, qf, leader);
                ptx::mbar_expect_tx_if(df, TILE_BYTES + 512, leader);
                for (int half = 0; half < 2; ++half) {
                    ptx::tma_load_4d_if(base + OFF_DO + s * TILE_BYTES + half * HALF_BYTES, &p.map_do, half * 64, (i_lo + i) * BLK, h, b, df,
                                        leader);
                }
                ptx::bulk_g2s_if(ss + 512, delta + (i_lo + i) * BLK, 512, df, leader);
                i = i + 1 < n_q ? i + 1 : 0;
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
        if (!ok) {
            flag(p, ERR_LOAD);
        }
        __syncwarp();
    }
    else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        constexpr uint32_t idesc_kk = ptx::make_idesc(1, 1, BLK, BLK, 0, 0);  // A, B K-major
        constexpr uint32_t idesc_tn = ptx::make_idesc(1, 1, BLK, D, 0, 1);    // A from TMEM, B MN-major
        constexpr uint32_t idesc_nn = ptx::make_idesc(1, 1, D, BLK, 1, 1);    // A, B MN-major
        // one descriptor per operand and role, built once; every MMA below only steps it
        const ptx::Desc k_kmaj(ptx::smem_desc_sw128(base + OFF_K, 16, 1024));
        const ptx::Desc v_kmaj(ptx::smem_desc_sw128(base + OFF_V, 16, 1024));
        const ptx::Desc q_kmaj(ptx::smem_desc_sw128(base + OFF_Q, 16, 1024));
        const ptx::Desc do_kmaj(ptx::smem_desc_sw128(base + OFF_DO, 16, 1024));
        const ptx::Desc k_mn(ptx::smem_desc_sw128(base + OFF_K, HALF_BYTES, 1024));
        const ptx::Desc q_mn(ptx::smem_desc_sw128(base + OFF_Q, HALF_BYTES, 1024));
        const ptx::Desc do_mn(ptx::smem_desc_sw128(base + OFF_DO, HALF_BYTES, 1024));
        const ptx::Desc ds_mn(ptx::smem_desc_sw128(base + OFF_DS, HALF_BYTES, 1024));
        uint32_t        it = 0, wc = 0, s = 0, ph = 0;
        bool            ok = true;
        auto issue_s = [&](uint32_t stage) {  // S^T = K Q^T
            const ptx::Desc qd = q_kmaj.at(stage * TILE_BYTES);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
                const uint32_t off = (kk >> 2) * HALF_BYTES + (kk & 3) * 32;
                ptx::mma_f16_ss_if<1>(tmem, k_kmaj.at(off), qd.at(off), idesc_kk, kk, leader);
            }
            ptx::mma_commit_if<1>(b_of(bar.s_full), leader);
        };
        for (int w = w_0; w < w_end && ok; w += w_inc, ++wc) {
            if (!ptx::mbar_wait_warp(b_of(bar.kv_full), wc & 1u) || !ptx::mbar_wait_warp(b_of(bar.q_full[0]) + s * 8, ph)) {
                ok = false;
                break;
            }
            ptx::tc_fence_after();
            issue_s(s);
            for (int i = 0; i < n_q; ++i, ++it) {
                const ptx::Desc o_k = do_kmaj.at(s * TILE_BYTES), o_m = do_mn.at(s * TILE_BYTES), q_m = q_mn.at(s * TILE_BYTES);
                const uint32_t  next = s + 1 == STAGES ? 0 : s + 1, next_ph = next == 0 ? ph ^ 1u : ph;
                // the previous block's dQ^T must have left the columns dP^T is written to
                if (!ptx::mbar_wait_warp(b_of(bar.do_full[0]) + s * 8, ph) || !ptx::mbar_wait_warp(b_of(bar.dq_free), (it & 1u) ^ 1u)) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                stamp(p, it, 1);
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {  // dP^T = V dO^T
                    const uint32_t off = (kk >> 2) * HALF_BYTES + (kk & 3) * 32;
                    ptx::mma_f16_ss_if<1>(tmem + 128, v_kmaj.at(off), o_k.at(off), idesc_kk, kk, leader);
                }
                ptx::mma_commit_if<1>(b_of(bar.dp_full), leader);
                if (!ptx::mbar_wait_warp(b_of(bar.p_ready), it & 1u)
                    || (i == 0 && !ptx::mbar_wait_warp(b_of(bar.acc_free), (wc & 1u) ^ 1u))) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                stamp(p, it, 0);
#pragma unroll
                for (int kk = 0; kk < BLK / 16; ++kk) {  // dV += P^T dO   (contraction over q)
                    ptx::mma_f16_ts_if(tmem + 256, tmem + (kk >> 2) * 64 + (kk & 3) * 8, o_m.at(kk * 2048), idesc_tn,
                                       static_cast<uint32_t>(i | kk), leader);
                }
                if (i + 1 < n_q) {
                    if (!ptx::mbar_wait_warp(b_of(bar.q_full[0]) + next * 8, next_ph)) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    issue_s(next);
                }
                stamp(p, it, 2);
                if (!ptx::mbar_wait_warp(b_of(bar.ds_ready), it & 1u)) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                stamp(p, it, 3);
#pragma unroll
                for (int kk = 0; kk < BLK / 16; ++kk) {  // dK += dS^T Q
                    ptx::mma_f16_ts_if(tmem + 384, tmem + 128 + (kk >> 2) * 64 + (kk & 3) * 8, q_m.at(kk * 2048), idesc_tn,
                                       static_cast<uint32_t>(i | kk), leader);
                }
                ptx::mma_commit_if<1>(b_of(bar.empty[0]) + s * 8, leader);
#pragma unroll
                for (int kk = 0; kk < BLK / 16; ++kk) {  // dQ^T = K^T dS^T   (contraction over kv)
                    ptx::mma_f16_ss_if<1>(tmem + 128, k_mn.at(kk * 2048), ds_mn.at(kk * 2048), idesc_nn, kk, leader);
                }
                ptx::mma_commit_if<1>(b_of(bar.dq_full), leader);
                stamp(p, it, 4);
                s  = next;
                ph = next_ph;
            }
            if (ok) {
                ptx::mma_commit_if<1>(b_of(bar.acc_full), leader);
                ptx::mma_commit_if<1>(b_of(bar.kv_empty), leader);
            }
        }
        if (!ok) {
            flag(p, ERR_MMA);
        }
        __syncwarp();
    }
    else if (warp < 10) {
        // ---------------------------------------------------------------- element-wise warps
        // two threads per kv row: warps 2..5 take query columns 0..63 of a block, warps 6..9 columns
        // 64..127; each writes its packed bf16 results over the start of the columns it read itself
        const int      quarter  = warp & 3;
        const int      c2       = (warp - 2) >> 2;
        const int      row_in   = quarter * 32 + lane;
        const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t t_s = tmem + lane_off + c2 * 64, t_dp = tmem + 128 + lane_off + c2 * 64;
        const uint32_t t_dv = tmem + 256 + lane_off, t_dk = tmem + 384 + lane_off;
        uint8_t*       ds_row = sm + OFF_DS + c2 * HALF_BYTES + row_in * 128;
        const float    c = p.scale_log2;
        uint32_t       it = 0, wc = 0;
        bool           ok = true;
        for (int w = w_0; w < w_end && ok; w += w_inc, ++wc) {
            const int  jb    = w % p.kv_blocks;
            const int  h     = (w / p.kv_blocks) % p.H;
            const int  b     = w / (p.kv_blocks * p.H);
            const int  kvr   = jb * BLK + row_in;
            const bool kv_ok = kvr < p.Skv;
            const bool tail  = jb * BLK + quarter * 32 + 32 > p.Skv;  // some of this warp's rows do not exist
            for (int i = 0; i < n_q; ++i, ++it) {
                const int    s     = it % STAGES;
                const float* lse2  = reinterpret_cast<const float*>(sm + OFF_STATS + s * 1024) + c2 * 64;
                const float* delta = lse2 + 128;
                uint32_t     pk[32];  // this thread's 64 probabilities, bf16 pairs
                if (!ptx::mbar_wait(&bar.s_full, it & 1u)) {
                    flag(p, ERR_COMPUTE);
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                if (threadIdx.x == 64) {
                    stamp(p, it, 5);
                }
                {
                    // loads run one 16-column chunk ahead of the arithmetic
                    uint32_t ra[16], rb[16];
                    ptx::tmem_ld_32x16(t_s, ra);
                    ptx::tmem_ld_wait();
                    ptx::tmem_ld_32x16(t_s + 16, rb);
                    c1_chunk<0>(ra, pk, lse2, c);
                    ptx::tmem_ld_wait();
                    ptx::tmem_ld_32x16(t_s + 32, ra);
                    c1_chunk<1>(rb, pk, lse2, c);
                    ptx::tmem_ld_wait();
                    ptx::tmem_ld_32x16(t_s + 48, rb);
                    store_p<0>(t_s, pk, tail, kv_ok);
                    c1_chunk<2>(ra, pk, lse2, c);
                    ptx::tmem_ld_wait();
                    c1_chunk<3>(rb, pk, lse2, c);
                    store_p<1>(t_s, pk, tail, kv_ok);
                }
                ptx::tmem_st_wait();
                ptx::tc_fence_before();
                ptx::mbar_arrive_warp(&bar.p_ready);
                if (threadIdx.x == 64) {
                    stamp(p, it, 6);
                }

                if (!ptx::mbar_wait(&bar.dp_full, it & 1u)) {
                    flag(p, ERR_COMPUTE);
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                if (threadIdx.x == 64) {
                    stamp(p, it, 7);
                }
                {
                    uint32_t ra[16], rb[16];
                    ptx::tmem_ld_32x16(t_dp, ra);
                    ptx::tmem_ld_wait();
                    ptx::tmem_ld_32x16(t_dp + 16, rb);
                    c2_chunk<0>(ra, pk, delta, t_dp, ds_row, row_in);
                    ptx::tmem_ld_wait();
                    ptx::tmem_ld_32x16(t_dp + 32, ra);
                    c2_chunk<1>(rb, pk, delta, t_dp, ds_row, row_in);
                    ptx::tmem_ld_wait();
                    ptx::tmem_ld_32x16(t_dp + 48, rb);
                    c2_chunk<2>(ra, pk, delta, t_dp, ds_row, row_in);
                    ptx::tmem_ld_wait();
                    c2_chunk<3>(rb, pk, delta, t_dp, ds_row, row_in);
                }
                ptx::tmem_st_wait();
                ptx::fence_proxy_async_smem();
                ptx::tc_fence_before();
                ptx::mbar_arrive_warp(&bar.ds_ready);
                if (threadIdx.x == 64) {
                    stamp(p, it, 8);
                }
            }
            // dK, dV of this block
            if (ok && !ptx::mbar_wait(&bar.acc_full, wc & 1u)) {
                flag(p, ERR_COMPUTE);
                ok = false;
            }
            __nv_bfloat16* dv = p.dv + b * p.dv_batch + static_cast<int64_t>(kvr) * p.dv_row + h * p.dv_head;
            __nv_bfloat16* dk = p.dk + b * p.dk_batch + static_cast<int64_t>(kvr) * p.dk_row + h * p.dk_head;
            if (SPLIT) {  // also after a timeout: the other CTAs wait in its barriers
                join_shares(p, base, t_dv, t_dk, c2 * 4 + quarter, lane, crank, csize, dv, dk, kv_ok && ok);
                break;
            }
            if (!ok) {
                break;
            }
            ptx::tc_fence_after();
#pragma unroll 1
            for (int ch = 2 * c2; ch < 2 * c2 + 2; ++ch) {
                float rv[32], rk[32];
                ptx::tmem_ld_32x32(t_dv + ch * 32, reinterpret_cast<uint32_t(&)[32]>(rv));
                ptx::tmem_ld_32x32(t_dk + ch * 32, reinterpret_cast<uint32_t(&)[32]>(rk));
                ptx::tmem_ld_wait();
                if (kv_ok) {
                    store_row32(dv + ch * 32, rv, 1.0f);
                    store_row32(dk + ch * 32, rk, p.scale);
                }
            }
            ptx::tc_fence_before();
            ptx::mbar_arrive_warp(&bar.acc_free);
        }
    }
    else {
        // ---------------------------------------------------------------- dQ drain
        // dQ_i^T sits in tensor memory with the head dimension on the lanes: lane d of a warp adds
        // its query columns into dq_acc[q][d], so that every warp-wide reduction covers 128
        // contiguous bytes of one query row. Warps 10..13 take query columns 0..63, warps 14..17
        // columns 64..127. The columns are released as soon as they are in registers. What waits in the memory queue
        // behind a burst of reductions is every other warp's loads, stores and products: the address arithmetic between them
        // is what keeps them apart (37888 x 4 with zeros, beside 4.92 ms of the kernel of that time: rows at constant offsets 6.35, four
        // floats a reduction 6.81, paced by the clock 5.0 - 5.3 in groups of two or four and 6.4 one by one, by nanosleep 5.56).
        const int      quarter  = warp & 3;
        const int      qh       = (warp - 10) >> 2;
        const int      dcol     = quarter * 32 + lane;
        const uint32_t t_dq     = tmem + 128 + qh * 64 + (static_cast<uint32_t>(quarter * 32) << 16);
        const int64_t  q_stride = static_cast<int64_t>(p.H) * D;
        uint32_t       it       = 0;
        bool           ok       = true;
        for (int w = w_0; w < w_end && ok; w += w_inc) {
            const int h  = (w / p.kv_blocks) % p.H;
            const int b  = w / (p.kv_blocks * p.H);
            float*    dq = p.dq_acc + (static_cast<int64_t>(b) * p.Sq * p.H + h) * D + dcol;
            const int first = first_block(p, w % p.kv_blocks, n_q);
            for (int i0 = 0; i0 < n_q; ++i0, ++it) {
                const int i = i_lo + (i0 + first < n_q ? i0 + first : i0 + first - n_q);
                if (!ptx::mbar_wait(&bar.dq_full, it & 1u)) {
                    flag(p, ERR_DRAIN);
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                if (threadIdx.x == 320) {
                    stamp(p, it, 9);
                }
                uint32_t r0[32], r1[32];
                ptx::tmem_ld_32x32(t_dq, r0);
                ptx::tmem_ld_32x32(t_dq + 32, r1);
                ptx::tmem_ld_wait();
                ptx::tc_fence_before();
                ptx::mbar_arrive_warp(&bar.dq_free);
                if (threadIdx.x == 320) {
                    stamp(p, it, 10);
                }
                const int q0    = i * BLK + qh * 64;
                const int valid = p.Sq - q0;  // query rows of this half that exist
                float*    row   = dq + static_cast<int64_t>(q0) * q_stride;
#pragma unroll
                for (int k = 0; k < 32; ++k) {
                    if (k < valid) {
                        red_add(row + k * q_stride, __uint_as_float(r0[k]));
                    }
                }
#pragma unroll
                for (int k = 0; k < 32; ++k) {
                    if (32 + k < valid) {
                        red_add(row + (32 + k) * q_stride, __uint_as_float(r1[k]));
                    }
                }
            }
        }
    }

    if (SPLIT && (warp < 2 || warp >= 10)) {  // the element-wise warps' exchange
        ptx::cluster_sync();
        ptx::cluster_sync();
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tmem_dealloc<512>(tmem);
    }
}

// Items beyond whole waves of one per SM are shared out, see cluster_plan.h. Times in query blocks (2.1 us).
// 8191 tokens x 10 heads (640 items on 148 SMs): 844 -> 777 us, 4000 x 5 (160 items): 166 -> 113, 1000 x 5
// (40 items): 31.7 -> 22.5.
fu::ClusterPlan plan_split(int items, int n_q, int sms, int dev)
{
    static fu::ClusterCapacity capacity;
    return fu::plan_clusters(items, n_q, sms, {2.0, 1.0, 1.0},
                             [&](int csize) { return capacity.of(fmha_bwd_fused_kernel<true>, csize, dev, THREADS, SMEM_BYTES); });
}

}  // namespace

// Launched by fu_fmha_bwd (fmha_bwd_sm100.cu) after its pre-pass has filled lse2 / delta and the
// fp32 dQ accumulator has been zeroed; the caller rounds the accumulator to bf16 afterwards.
int fu_fmha_bwd_fused_launch(const FuFmhaArgs* a, const float* lse2, const float* delta, int sq_pad, void* stream)
{
    Params p{};
    int    rc = make_map_bshd(&p.map_q, a->q, a->batch, a->seq_q, a->heads, a->q_row, a->q_head, a->q_batch, BLK);
    if (rc == FU_OK) {
        rc = make_map_bshd(&p.map_do, a->d_o, a->batch, a->seq_q, a->heads, a->o_row, a->o_head, a->o_batch, BLK);
    }
    if (rc == FU_OK) {
        rc = make_map_bshd(&p.map_k, a->k, a->batch, a->seq_kv, a->heads, a->k_row, a->k_head, a->k_batch, BLK);
    }
    if (rc == FU_OK) {
        rc = make_map_bshd(&p.map_v, a->v, a->batch, a->seq_kv, a->heads, a->v_row, a->v_head, a->v_batch, BLK);
    }
    if (rc != FU_OK) {
        return rc;
    }
    p.lse2       = lse2;
    p.delta      = delta;
    p.dq_acc     = a->dq_acc;
    p.dk         = static_cast<__nv_bfloat16*>(a->dk);
    p.dv         = static_cast<__nv_bfloat16*>(a->dv);
    p.dk_row     = a->k_row;
    p.dk_head    = a->k_head;
    p.dk_batch   = a->k_batch;
    p.dv_row     = a->v_row;
    p.dv_head    = a->v_head;
    p.dv_batch   = a->v_batch;
    p.B          = a->batch;
    p.H          = a->heads;
    p.Sq         = a->seq_q;
    p.Skv        = a->seq_kv;
    p.Sq_pad     = sq_pad;
    p.n_q        = sq_pad / BLK;
    p.kv_blocks  = (a->seq_kv + BLK - 1) / BLK;
    p.total_work = p.kv_blocks * p.H * p.B;
    p.scale      = a->scale;
    p.scale_log2 = a->scale * 1.4426950408889634f;
    p.err        = a->err;
    p.overlap    = a->ctas <= 0;
    p.trace      = a->trace;
    int dev = 0, sms = 0;
    FU_CUDA_OK(cudaGetDevice(&dev));
    FU_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    rc = fu::raise_smem_limit(fmha_bwd_fused_kernel<false>, SMEM_BYTES);
    if (rc != FU_OK) {
        return rc;
    }
    const int             items = p.total_work;
    const fu::ClusterPlan plan  = a->ctas > 0 || a->trace ? fu::ClusterPlan{items, 1, 0.0} : plan_split(items, p.n_q, sms, dev);
    p.total_work                = plan.whole;
    p.first                     = plan.whole;
    if (plan.whole > 0) {
        int grid = a->ctas > 0 ? std::min(a->ctas, sms) : sms;
        grid     = std::max(1, std::min(grid, p.total_work));
        // in the ordinary way: taken up by the SMs in the order in which the pre-pass left them it is 5 % slower (8191 x 10
        // 655 -> 687 us, 3039 x 24 253 -> 270)
        fmha_bwd_fused_kernel<false><<<grid, THREADS, SMEM_BYTES, static_cast<cudaStream_t>(stream)>>>(p);
        FU_CUDA_OK(cudaGetLastError());
    }
    if (plan.csize > 1) {
        cudaLaunchConfig_t  cfg  = {};
        cudaLaunchAttribute attr = fu::cluster_attr(plan.csize);
        cfg.gridDim              = dim3(static_cast<unsigned>((items - plan.whole) * plan.csize), 1, 1);
        cfg.blockDim             = dim3(THREADS, 1, 1);
        cfg.dynamicSmemBytes     = SMEM_BYTES;
        cfg.stream               = static_cast<cudaStream_t>(stream);
        cfg.attrs                = &attr;
        cfg.numAttrs             = 1;
        FU_CUDA_OK(cudaLaunchKernelEx(&cfg, fmha_bwd_fused_kernel<true>, p));
    }
    return FU_OK;
}
