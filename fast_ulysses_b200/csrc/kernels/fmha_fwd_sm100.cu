// Non-causal flash attention forward for head_dim 128 on the tcgen05 tensor cores.
//
// One persistent CTA per SM works on (batch, head, 256 query rows) items: two 128-row query tiles
// that share every K/V tile. Warp roles:
//   warp 0       TMA producer: Q (once per item), then K and V tiles through two-stage rings
//   warp 1       MMA issuer: S_t = Q_t K^T (operands in shared memory), O_t += P_t V (P read
//                from tensor memory, V as an MN-major shared-memory operand)
//   warps 2, 3   idle (they fill warpgroup 0 so that register counts can be set per warpgroup:
//                warpgroup 0 gives registers away, the softmax warpgroups take them)
//   warps 4..7   softmax for query tile 0, warps 8..11 for query tile 1: one thread per row;
//                exponentials against a loose reference, P written back over S in tensor memory as
//                packed bf16, O rescaled in tensor memory only when a row leaves the reference's range;
//                final normalisation, bf16 store and log-sum-exp
// Tensor memory (512 columns): S0 | S1 | O0 | O1, 128 fp32 columns each; P_t aliases S_t.
// The two query tiles are staggered (QK of tile 0 for step j+1 is issued between the two PV of
// step j), so each softmax has two MMA slots of cover.
//
// What bounds it: a tile's scores, softmax, P V and next scores form one chain through the columns S_t and
// P_t share, and two tiles are all that fit. The chain is about 2850 clocks per 128 kv rows (SM clock,
// zeros, no power limit): 100 to load the first scores, 96 exponentials per thread, their hand-over, the
// last 32 under most of P V, then 2 + 8 MMAs (640) and two barrier wake-ups (300). The exponentials take
// 9 - 12 clocks each on the special-function unit, whose floor for both tiles is 2050 per step; a quarter
// of them on the FMA pipe is the best split (16384 tokens x 10 heads: 1.187 ms with random operands at the
// power limit and 0.948 with zeros, 1.201 and 0.992 with none, 1.277 and 1.056 with three eighths). No
// maximum is taken in an ordinary step (1.253 and 1.010 with one, and with O written row by row). Tried and slower: half steps of 64 kv rows with two score
// buffers per tile (1.17 ms), two threads per row (1.03), an issuing warp per tile (1.40: the tiles then
// run in step and contend).
//
// q, k, v, o use the (batch, seq, heads, 128) layout of the all-to-all windows, so attention reads
// what the fused QKV kernel scattered and writes what the output projection pulls, with no copy.
// The reference has no attention kernel (examples/dit_attention.py:57 calls torch SDPA).
#include "cluster_plan.h"
#include "fu_kernels.h"
#include "host_util.h"
#include "ptx.cuh"
#include "tma_host.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

namespace {

using namespace fu;

constexpr int D         = 128;
constexpr int BM        = 128;  // rows per query tile
constexpr int QT        = 2;    // query tiles per CTA
constexpr int BN        = 128;  // kv rows per step
constexpr int KV_STAGES = 2;
constexpr int TILE_BYTES = 128 * D * 2;       // 32 KiB: a 128 x 128 bf16 tile as two 64-column halves
constexpr int HALF_BYTES = TILE_BYTES / 2;
constexpr int OUT_BYTES  = 32 * 128;          // per softmax warp: 32 rows x 64 columns of the result
constexpr int SMEM_BYTES = (QT + 2 * KV_STAGES) * TILE_BYTES + 8 * OUT_BYTES + 1024;
constexpr int THREADS    = 32 * 12;            // three warpgroups: {producer, MMA, 2 idle}, softmax 0, softmax 1
constexpr int REGS_SMALL = 104;                 // warpgroup 0 after it has given registers away
constexpr int REGS_SOFTMAX = 200;              // per scheduler: 32 x (104 + 2 x 200) = 16128 of 16384 registers
constexpr float RANGE = 8.0f;                 // in log2 units
constexpr float RANGE_SUM = 256.0f;            // 2^RANGE
constexpr int   kPolyPairs = 4;               // of every 16 exponential pairs, on the FMA pipe by default

enum : uint32_t { ERR_LOAD = 11, ERR_MMA = 12, ERR_SOFTMAX = 13 };

struct Params {
    CUtensorMap    map_q, map_k, map_v;
    __nv_bfloat16* o;
    float*         lse;         // (B, H, Sq)
    int64_t        o_row, o_head, o_batch;  // element strides of o
    int            B, H, Sq, Skv;
    int            q_blocks, total_work, n_kv;
    int            first;       // split kernel: the item of cluster 0
    int            overlap;     // the next kernel may come up beside this one
    float          scale, scale_log2;
    uint32_t*      err;
    uint64_t*      trace;
};

__device__ __forceinline__ void flag(const Params& p, uint32_t code)
{
    if (p.err) {
        atomicCAS(p.err, 0u, code);
    }
}

struct Barriers {
    uint64_t q_full, q_empty;
    uint64_t k_full[KV_STAGES], k_empty[KV_STAGES], v_full[KV_STAGES], v_empty[KV_STAGES];
    uint64_t s_full[QT], p_lo[QT], p_hi[QT], o_final[QT], o_free[QT], merge;
};

// exp2 of a pair on the FMA pipe instead of the special-function unit: floor by a round-down add of
// 1.5 * 2^23 (the integer part lands in the low mantissa bits), the minimax quintic for 2^fraction on
// [0, 1) (Remez exchange; relative error 1.5e-7 evaluated in fp32, as good as the special-function
// unit's), and the integer part added to the exponent field. That field would wrap below -127: such arguments
// become the next number above it, whose result is 2^-143 and thus a bf16 zero, as the special-function
// unit's is (a weight of 2^-126 is not nothing beside a value of 2^127).
__device__ __forceinline__ void ex2_poly2(float& e0, float& e1, float x0, float x1)
{
    constexpr float MAGIC = 12582912.0f;
    constexpr float C0 = 0.9999999403953552f, C1 = 0.6931530833244324f, C2 = 0.24015361070632935f, C3 = 0.05582631751894951f,
                    C4 = 0.00898933969438076f, C5 = 0.0018775766948238015f;
    x0 = fmaxf(x0, -0x1.fbfffep6f);
    x1 = fmaxf(x1, -0x1.fbfffep6f);
    float t0, t1, i0, i1, f0, f1, p0, p1;
    ptx::add2_rm(t0, t1, x0, x1, MAGIC, MAGIC);
    ptx::add2(i0, i1, t0, t1, -MAGIC, -MAGIC);
    ptx::fma2(f0, f1, i0, i1, -1.0f, -1.0f, x0, x1);
    ptx::fma2(p0, p1, f0, f1, C5, C5, C4, C4);
    ptx::fma2(p0, p1, p0, p1, f0, f1, C3, C3);
    ptx::fma2(p0, p1, p0, p1, f0, f1, C2, C2);
    ptx::fma2(p0, p1, p0, p1, f0, f1, C1, C1);
    ptx::fma2(p0, p1, p0, p1, f0, f1, C0, C0);
    e0 = __uint_as_float(__float_as_uint(p0) + (__float_as_uint(t0) << 23));
    e1 = __uint_as_float(__float_as_uint(p1) + (__float_as_uint(t1) << 23));
}

// Whether pair `i` of 16 takes the FMA-pipe path: NP of them, spread evenly so both pipes stay fed.
template <int NP>
__device__ constexpr bool on_fma_pipe(int i)
{
    return NP > 0 && (i * NP) % 16 < NP;
}

// 32 columns of one row: P = exp2(S * c - m * c) as packed bf16, row sum into l4. NP of every 16
// pairs take the FMA-pipe path, the rest the special-function unit. RAGGED: columns from `valid` on do not
// exist and weigh nothing, whatever the scale makes of their -inf.
template <int NP, bool RAGGED = false>
__device__ __forceinline__ void exp_chunk(const uint32_t* r, float c, float nmc, float (&l4)[4], uint32_t* pk, int valid = 32)
{
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float x0, x1, e0, e1;
        ptx::fma2(x0, x1, __uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]), c, c, nmc, nmc);
        if (on_fma_pipe<NP>(i)) {
            ex2_poly2(e0, e1, x0, x1);
        }
        else {
            e0 = ptx::ex2(x0);
            e1 = ptx::ex2(x1);
        }
        if (RAGGED) {
            e0 = 2 * i < valid ? e0 : 0.0f;
            e1 = 2 * i + 1 < valid ? e1 : 0.0f;
        }
        ptx::add2(l4[(2 * i) & 3], l4[(2 * i + 1) & 3], l4[(2 * i) & 3], l4[(2 * i + 1) & 3], e0, e1);
        pk[i] = ptx::pack_bf16x2(e0, e1);
    }
}

// Optional timeline (TRACE builds only): CTA 0 stores the SM clock of pipeline events of kv steps
// 64..71 of its first work item, 32 slots per step: 0..9 softmax tile 0, 10..19 softmax tile 1,
// 20..31 the MMA issuer.
template <bool TRACE>
__device__ __forceinline__ void stamp(const Params& p, uint32_t step, int ev)
{
    if (TRACE && blockIdx.x == 0 && (threadIdx.x & 31) == 0 && step >= 64u && step < 72u) {
        p.trace[(step - 64u) * 32 + ev] = clock64();
    }
}

// The end of an item whose kv tiles were shared by the CTAs of a cluster: every CTA holds an unnormalised
// O (256 x 128 in tensor memory), and for each row its reference and sum. The result is cut into eight
// units of one query tile x 32 columns, dealt to the CTAs in order; each sends the others' units of its O
// through distributed shared memory, so all of them send, receive and write at once, and the sum over
// the shares runs in their order. The operand tiles are done with by then: units received lie at
// their place, 16 KiB each, the (reference, sum) pairs behind them. Executed by the softmax warps; the
// other warps take part in the two cluster barriers.
constexpr int UNITS       = 8;
constexpr int UNIT_BYTES  = BM * 128;         // 128 rows x 32 fp32
constexpr int PAIRS_OFF   = 160 * 1024;       // (cluster size - 1) x units of a CTA <= 10 for 2..6 and 8 CTAs
static_assert(PAIRS_OFF + 8 * QT * BM * 8 <= (QT + 2 * KV_STAGES) * TILE_BYTES, "exchange area");

__device__ __forceinline__ void join_shares(const Params& p, int b, int h, int row, int t, int quarter, int lane, uint32_t to,
                                            float m_log2, float l, int crank, int csize, uint32_t base, uint32_t stage)
{
    ptx::tc_fence_after();
    const int row_in = quarter * 32 + lane;
    auto first_unit = [&](int r) { return (r * UNITS + csize - 1) / csize; };  // units [first_unit(r), first_unit(r + 1)) are CTA r's
    ptx::cluster_sync();  // every CTA's products are complete: its operand tiles may be overwritten
    for (int r = 0; r < csize; ++r) {
        ptx::st_cluster_v2f(ptx::cluster_addr(base + PAIRS_OFF + ((crank * QT + t) * BM + row_in) * 8, r), m_log2, l);
    }
#pragma unroll 1
    for (int ch = 0; ch < 4; ++ch) {
        const int u     = t * 4 + ch;
        const int owner = u * csize / UNITS;
        if (owner == crank) {
            continue;
        }
        const int      slot = (crank - (crank > owner ? 1 : 0)) * (first_unit(owner + 1) - first_unit(owner)) + u - first_unit(owner);
        // through the warp's staging buffer, so that a store instruction writes 512 contiguous bytes of the
        // other CTA's memory (a row per lane, 32 separate pieces, took three times as long)
        const uint32_t dst = ptx::cluster_addr(base + slot * UNIT_BYTES + quarter * OUT_BYTES + lane * 16, owner);
        uint32_t       r[32];
        ptx::tmem_ld_32x32(to + ch * 32, r);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            ptx::st_shared_v4(stage + lane * 128 + ((g ^ (lane & 7)) << 4), make_uint4(r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]));
        }
        __syncwarp();
        uint4 v[8];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            v[g] = ptx::ld_shared_v4(stage + g * 512 + lane * 16);
        }
        __syncwarp();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            ptx::st_cluster_v4(dst + g * 512, v[g].x, v[g].y, v[g].z, v[g].w);
        }
    }
    ptx::cluster_sync();
    const int first = first_unit(crank), mine = first_unit(crank + 1) - first;
    if (first + mine <= t * 4 || first >= t * 4 + 4) {
        return;  // none of this query tile
    }
    const uint32_t pairs = base + PAIRS_OFF + (t * BM + row_in) * 8;
    float          top = -INFINITY, sum = 0.0f;
    for (int r = 0; r < csize; ++r) {
        top = fmaxf(top, ptx::ld_shared_v2f(pairs + r * QT * BM * 8).x);
    }
    for (int r = 0; r < csize; ++r) {
        const float2 ml = ptx::ld_shared_v2f(pairs + r * QT * BM * 8);
        sum += ptx::ex2(ml.x - top) * ml.y;
    }
    const float inv   = 1.0f / sum;
    const int   row_w = row - lane;
#pragma unroll 1
    for (int ch = max(0, first - t * 4); ch < min(4, first + mine - t * 4); ++ch) {
        float acc[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            acc[i] = 0.0f;
        }
#pragma unroll 1
        for (int r = 0; r < csize; ++r) {
            const float w = ptx::ex2(ptx::ld_shared_v2f(pairs + r * QT * BM * 8).x - top) * inv;
            if (r == crank) {
                uint32_t o[32];
                ptx::tmem_ld_32x32(to + ch * 32, o);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    acc[i] += __uint_as_float(o[i]) * w;
                }
            }
            else {
                const uint32_t src = base + ((r - (r > crank ? 1 : 0)) * mine + t * 4 + ch - first) * UNIT_BYTES + row_in * 128;
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    const uint4 v = ptx::ld_shared_v4(src + ((g ^ (lane & 7)) << 4));
                    acc[4 * g] += __uint_as_float(v.x) * w;
                    acc[4 * g + 1] += __uint_as_float(v.y) * w;
                    acc[4 * g + 2] += __uint_as_float(v.z) * w;
                    acc[4 * g + 3] += __uint_as_float(v.w) * w;
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            ptx::st_shared_v4(stage + lane * 128 + ((g ^ (lane & 7)) << 4),
                              make_uint4(ptx::pack_bf16x2(acc[8 * g], acc[8 * g + 1]), ptx::pack_bf16x2(acc[8 * g + 2], acc[8 * g + 3]),
                                         ptx::pack_bf16x2(acc[8 * g + 4], acc[8 * g + 5]), ptx::pack_bf16x2(acc[8 * g + 6], acc[8 * g + 7])));
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // four lanes per row
            const int   r = i * 8 + (lane >> 2);
            const uint4 v = ptx::ld_shared_v4(stage + r * 128 + (((lane & 3) ^ (r & 7)) << 4));
            if (row_w + r < p.Sq) {
                ptx::st_v4(p.o + b * p.o_batch + static_cast<int64_t>(row_w + r) * p.o_row + h * p.o_head + ch * 32 + (lane & 3) * 8, v);
            }
        }
        if (ch == 0 && row < p.Sq && p.lse) {
            p.lse[(static_cast<int64_t>(b) * p.H + h) * p.Sq + row] = (top + ptx::lg2(sum)) * 0.6931471805599453f;
        }
    }
}

// What a CTA takes for an item. kTwoTiles: two query tiles, all kv tiles. kShared: the same two query tiles,
// but the CTAs of a cluster take a part of the kv tiles each. kOneTile: one query tile, whose even kv
// tiles go through the first half of the kernel (scores, P, O) and the odd ones through the second; the two
// results meet in the epilogue, which reads both from tensor memory. Half as many steps per
// item and twice as many items, for problems that leave SMs idle; every K and V tile then serves 128
// rows instead of 256, so it reads them twice as often.
enum class Form { kTwoTiles, kShared, kOneTile };

template <int NP, bool TRACE, Form FORM>
__global__ void __launch_bounds__(THREADS, 1) fmha_fwd_kernel(const __grid_constant__ Params p)
{
    constexpr bool SPLIT    = FORM == Form::kShared;
    constexpr bool ONE      = FORM == Form::kOneTile;
    constexpr int  ROWS     = ONE ? BM : QT * BM;  // query rows of an item
    extern __shared__ uint8_t smem_raw[];
    __shared__ Barriers       bar;
    __shared__ uint32_t       tmem_holder;

    const uint32_t base = (ptx::smem_addr(smem_raw) + 1023u) & ~1023u;
    // layout: Q0 | Q1 | K[0] | K[1] | V[0] | V[1]
    const uint32_t sq_addr = base;
    const uint32_t sk_addr = base + QT * TILE_BYTES;
    const uint32_t sv_addr = sk_addr + KV_STAGES * TILE_BYTES;

    const int warp = static_cast<int>(ptx::uniform(threadIdx.x >> 5));
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        ptx::mbar_init(&bar.q_full, 1);
        ptx::mbar_init(&bar.q_empty, 1);
        for (int s = 0; s < KV_STAGES; ++s) {
            ptx::mbar_init(&bar.k_full[s], 1);
            ptx::mbar_init(&bar.k_empty[s], 1);
            ptx::mbar_init(&bar.v_full[s], 1);
            ptx::mbar_init(&bar.v_empty[s], 1);
        }
        for (int t = 0; t < QT; ++t) {
            ptx::mbar_init(&bar.s_full[t], 1);
            ptx::mbar_init(&bar.p_lo[t], 4);  // one arrival per warp
            ptx::mbar_init(&bar.p_hi[t], 4);
            ptx::mbar_init(&bar.o_final[t], 1);
            ptx::mbar_init(&bar.o_free[t], ONE ? 8 : 4);  // every warp that reads it
        }
        ptx::mbar_init(&bar.merge, 8);
        ptx::mbar_fence_init();
        ptx::tma_prefetch_desc(&p.map_q);
        ptx::tma_prefetch_desc(&p.map_k);
        ptx::tma_prefetch_desc(&p.map_v);
    }
    if (warp == 1) {
        ptx::tmem_alloc<512>(&tmem_holder);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    ptx::grid_wait();
    __syncthreads();
    if (p.overlap) {
        ptx::grid_trigger();  // with this CTA's tensor memory in hand
    }
    ptx::tc_fence_after();
    const uint32_t tmem = ptx::uniform(tmem_holder);
    // The items of this CTA and the kv tiles of each: every gridDim.x-th item and all of its tiles; or
    // (SPLIT) one item per cluster, each CTA its share of the tiles.
    const int crank = SPLIT ? static_cast<int>(ptx::uniform(ptx::cluster_ctarank())) : 0;
    const int csize = SPLIT ? static_cast<int>(ptx::uniform(ptx::cluster_nctarank())) : 1;
    const int w_0   = SPLIT ? p.first + static_cast<int>(blockIdx.x) / csize : static_cast<int>(blockIdx.x);
    const int w_end = SPLIT ? w_0 + 1 : p.total_work;
    const int w_inc = SPLIT ? 1 : static_cast<int>(gridDim.x);
    const int share = SPLIT ? (p.n_kv + csize - 1) / csize : p.n_kv;
    const int j_0   = crank * share;
    const int n_kv  = SPLIT ? min(share, p.n_kv - j_0) : p.n_kv;

    if (warp < 4) {
    ptx::setmaxnreg_dec<REGS_SMALL>();
    // Both roles are run by the whole warp, see ptx.cuh: elect_one().
    const uint32_t leader = ptx::elect_one();
    auto           b_of   = [](uint64_t& x) { return ptx::smem_addr(&x); };
    if (warp == 0) {
        // ---------------------------------------------------------------- producer
        uint32_t stage = 0, phase = 1, wc = 0;
        bool     ok = true;
        for (int w = w_0; w < w_end && ok; w += w_inc, ++wc) {
            const int qb = w % p.q_blocks;
            const int h  = (w / p.q_blocks) % p.H;
            const int b  = w / (p.q_blocks * p.H);
            if (!ptx::mbar_wait_warp(b_of(bar.q_empty), (wc & 1u) ^ 1u)) {
                ok = false;
                break;
            }
            ptx::mbar_expect_tx_if(b_of(bar.q_full), ROWS / BM * TILE_BYTES, leader);
            for (int t = 0; t < ROWS / BM; ++t) {
                for (int half = 0; half < 2; ++half) {
                    ptx::tma_load_4d_if(sq_addr + t * TILE_BYTES + half * HALF_BYTES, &p.map_q, half * 64,
                                        qb * ROWS + t * BM, h, b, b_of(bar.q_full), leader);
                }
            }
            for (int j = 0; j < n_kv; ++j) {
                const uint32_t kf = b_of(bar.k_full[0]) + stage * 8, vf = b_of(bar.v_full[0]) + stage * 8;
                if (!ptx::mbar_wait_warp(b_of(bar.k_empty[0]) + stage * 8, phase)) {
                    ok = false;
                    break;
                }
                ptx::mbar_expect_tx_if(kf, TILE_BYTES, leader);
                for (int half = 0; half < 2; ++half) {
                    ptx::tma_load_4d_if(sk_addr + stage * TILE_BYTES + half * HALF_BYTES, &p.map_k, half * 64, (j_0 + j) * BN, h, b, kf,
                                        leader);
                }
                if (!ptx::mbar_wait_warp(b_of(bar.v_empty[0]) + stage * 8, phase)) {
                    ok = false;
                    break;
                }
                ptx::mbar_expect_tx_if(vf, TILE_BYTES, leader);
                for (int half = 0; half < 2; ++half) {
                    ptx::tma_load_4d_if(sv_addr + stage * TILE_BYTES + half * HALF_BYTES, &p.map_v, half * 64, (j_0 + j) * BN, h, b, vf,
                                        leader);
                }
                if (++stage == KV_STAGES) {
                    stage = 0;
                    phase ^= 1u;
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
        constexpr uint32_t idesc_qk = ptx::make_idesc(1, 1, BM, BN, 0, 0);  // both K-major
        constexpr uint32_t idesc_pv = ptx::make_idesc(1, 1, BM, D, 0, 1);   // V is MN-major
        // one descriptor per operand, built once; every MMA below only steps it
        const ptx::Desc desc_q(ptx::smem_desc_sw128(sq_addr, 16, 1024));
        const ptx::Desc desc_k(ptx::smem_desc_sw128(sk_addr, 16, 1024));
        const ptx::Desc desc_v(ptx::smem_desc_sw128(sv_addr, HALF_BYTES, 1024));
        uint32_t        stage = 0, phase = 0, it = 0, wc = 0;
        bool            ok = true;

        auto issue_qk = [&](int t, uint32_t st) {
            const ptx::Desc qa = desc_q.at(ONE ? 0 : t * TILE_BYTES), ka = desc_k.at(st * TILE_BYTES);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
                const uint32_t off = (kk >> 2) * HALF_BYTES + (kk & 3) * 32;
                ptx::mma_f16_ss_if<1>(tmem + t * 128, qa.at(off), ka.at(off), idesc_qk, kk, leader);
            }
            ptx::mma_commit_if<1>(b_of(bar.s_full[0]) + t * 8, leader);
        };
        // The softmax hands P over in two parts, 96 kv rows and 32, so that most of P_t V runs under the
        // last exponentials: what is left behind them is on the way to the next step's scores.
        auto issue_pv = [&](int t, uint32_t st, auto part, uint32_t accumulate) {
            // 16 kv rows = 2048 bytes further down; the two 64-wide halves of d are HALF_BYTES
            // apart (leading byte offset), 8-row groups 1024 bytes apart
            const ptx::Desc va = desc_v.at(st * TILE_BYTES);
#pragma unroll
            for (int kk = decltype(part)::value ? 6 : 0; kk < (decltype(part)::value ? 8 : 6); ++kk) {
                ptx::mma_f16_ts_if(tmem + 256 + t * 128, tmem + t * 128 + kk * 8, va.at(kk * 2048), idesc_pv,
                                   accumulate | static_cast<uint32_t>(kk), leader);
            }
        };

        if constexpr (ONE) {
            // kv tile n of the CTA's sequence of tiles is in stage n % 2 and that stage's n / 2-th fill
            static_assert(KV_STAGES == 2, "stages by parity");
            uint32_t steps[QT] = {0, 0}, n_0 = 0;
            auto     qk = [&](int t, uint32_t n) {
                if (!ptx::mbar_wait_warp(b_of(bar.k_full[0]) + (n & 1u) * 8, (n >> 1) & 1u)) {
                    return false;
                }
                ptx::tc_fence_after();
                issue_qk(t, n & 1u);
                ptx::mma_commit_if<1>(b_of(bar.k_empty[0]) + (n & 1u) * 8, leader);
                return true;
            };
            for (int w = w_0; w < w_end && ok; w += w_inc, ++wc, n_0 += n_kv) {
                ok = ptx::mbar_wait_warp(b_of(bar.q_full), wc & 1u) && qk(0, n_0) && (n_kv < 2 || qk(1, n_0 + 1));
                for (int j = 0; j < n_kv && ok; j += 2) {
#pragma unroll
                    for (int t = 0; t < QT; ++t) {
                        if (j + t >= n_kv) {
                            break;
                        }
                        const uint32_t n = n_0 + j + t;
                        ok = ptx::mbar_wait_warp(b_of(bar.v_full[0]) + (n & 1u) * 8, (n >> 1) & 1u)
                             && ptx::mbar_wait_warp(b_of(bar.p_lo[t]), steps[t] & 1u)
                             && (j != 0 || ptx::mbar_wait_warp(b_of(bar.o_free[t]), (wc & 1u) ^ 1u));
                        if (!ok) {
                            break;
                        }
                        ptx::tc_fence_after();
                        issue_pv(t, n & 1u, std::integral_constant<int, 0>{}, static_cast<uint32_t>(j));
                        ok = ptx::mbar_wait_warp(b_of(bar.p_hi[t]), steps[t] & 1u);
                        if (!ok) {
                            break;
                        }
                        ptx::tc_fence_after();
                        issue_pv(t, n & 1u, std::integral_constant<int, 1>{}, 1u);
                        ptx::mma_commit_if<1>(b_of(bar.v_empty[0]) + (n & 1u) * 8, leader);
                        if (j + t + 2 >= n_kv) {
                            ptx::mma_commit_if<1>(b_of(bar.o_final[t]), leader);
                        }
                        else if (!qk(t, n + 2)) {
                            ok = false;
                            break;
                        }
                        ++steps[t];
                    }
                }
                ptx::mma_commit_if<1>(b_of(bar.q_empty), leader);
            }
        }
        else {
        for (int w = w_0; w < w_end && ok; w += w_inc, ++wc) {
            // prologue: S for both query tiles of kv step 0
            if (!ptx::mbar_wait_warp(b_of(bar.q_full), wc & 1u)
                || !ptx::mbar_wait_warp(b_of(bar.k_full[0]) + stage * 8, phase)) {
                ok = false;
                break;
            }
            ptx::tc_fence_after();
            issue_qk(0, stage);
            issue_qk(1, stage);
            ptx::mma_commit_if<1>(b_of(bar.k_empty[0]) + stage * 8, leader);
            for (int j = 0; j < n_kv && ok; ++j, ++it) {
                const uint32_t next = stage + 1 == KV_STAGES ? 0 : stage + 1, next_phase = next == 0 ? phase ^ 1u : phase;
                const bool     more = j + 1 < n_kv;
                if (!ptx::mbar_wait_warp(b_of(bar.v_full[0]) + stage * 8, phase)
                    || (more && !ptx::mbar_wait_warp(b_of(bar.k_full[0]) + next * 8, next_phase))) {
                    ok = false;
                    break;
                }
#pragma unroll
                for (int t = 0; t < QT; ++t) {
                    stamp<TRACE>(p, it, 20 + t * 6 + 0);
                    if (!ptx::mbar_wait_warp(b_of(bar.p_lo[t]), it & 1u)
                        || (j == 0 && !ptx::mbar_wait_warp(b_of(bar.o_free[t]), (wc & 1u) ^ 1u))) {
                        ok = false;
                        break;
                    }
                    stamp<TRACE>(p, it, 20 + t * 6 + 1);
                    ptx::tc_fence_after();
                    issue_pv(t, stage, std::integral_constant<int, 0>{}, static_cast<uint32_t>(j));
                    stamp<TRACE>(p, it, 20 + t * 6 + 2);
                    if (!ptx::mbar_wait_warp(b_of(bar.p_hi[t]), it & 1u)) {
                        ok = false;
                        break;
                    }
                    stamp<TRACE>(p, it, 20 + t * 6 + 3);
                    ptx::tc_fence_after();
                    issue_pv(t, stage, std::integral_constant<int, 1>{}, 1u);
                    if (!more) {
                        ptx::mma_commit_if<1>(b_of(bar.o_final[t]), leader);
                    }
                    else {
                        issue_qk(t, next);  // S_t is free again: PV_t above is ordered before it
                    }
                    stamp<TRACE>(p, it, 20 + t * 6 + 4);
                }
                if (!ok) {
                    break;
                }
                ptx::mma_commit_if<1>(b_of(bar.v_empty[0]) + stage * 8, leader);
                if (more) {
                    ptx::mma_commit_if<1>(b_of(bar.k_empty[0]) + next * 8, leader);
                }
                stage = next;
                phase = next_phase;
            }
            ptx::mma_commit_if<1>(b_of(bar.q_empty), leader);
        }
        }
        if (!ok) {
            flag(p, ERR_MMA);
        }
        __syncwarp();
    }
    if (SPLIT) {  // the softmax warps' exchange
        ptx::cluster_sync();
        ptx::cluster_sync();
    }
    }
    else {
        ptx::setmaxnreg_inc<REGS_SOFTMAX>();
        // ---------------------------------------------------------------- softmax + epilogue
        const int      t       = (warp - 4) >> 2;          // query tile
        const int      quarter = warp & 3;                 // TMEM lane quarter of this warp
        const int      row_in  = quarter * 32 + lane;      // row inside the query tile
        const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t ts      = tmem + t * 128 + lane_off;        // S_t / P_t
        const uint32_t to      = tmem + 256 + t * 128 + lane_off;  // O_t
        const float    c       = p.scale_log2;
        uint32_t       scount = 0, wc = 0;
        bool           ok = true;

        for (int w = w_0; w < w_end && ok; w += w_inc, ++wc) {
            const int qb  = w % p.q_blocks;
            const int h   = (w / p.q_blocks) % p.H;
            const int b   = w / (p.q_blocks * p.H);
            const int row = qb * ROWS + (ONE ? 0 : t * BM) + row_in;
            // Exponentials are taken against a reference that is only roughly the row's maximum: that of the row's
            // first step, until a step's exponentials leave a range of 2^RANGE above it; then it moves to that
            // step's maximum. The weight of the key it was taken from is exactly 1, and weights are rounded to
            // bf16, so a reference near the largest weight is also the more precise one (one key: the result is its
            // value). Whether a step stays inside is read off the sum of its exponentials, so an ordinary
            // step takes no maximum of the row; only the last quarter, which is handed over later, and the columns
            // on the FMA pipe, whose exponent field wraps where the special-function unit returns infinity, are
            // judged by their scores. A row whose scores have all been -inf so far has no reference yet and takes
            // the one of the first step that has others.
            float m_ref = 0.0f;
            bool  begun = false;
            float l4[4] = {0.f, 0.f, 0.f, 0.f};

            const int j_first = ONE ? t : 0;
            for (int j = j_first; j < n_kv; j += ONE ? 2 : 1, ++scount) {
                if (!ptx::mbar_wait(&bar.s_full[t], scount & 1u)) {
                    flag(p, ERR_SOFTMAX);
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                stamp<TRACE>(p, scount, t * 10 + 0);
                const int valid = min(BN, p.Skv - (j_0 + j) * BN);  // columns of this step that exist
                // The whole row of S in registers; the first quarter is waited for by itself.
                uint32_t r[BN];
                ptx::tmem_ld_32x32(ts, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
                ptx::tmem_ld_wait();
#pragma unroll
                for (int ch = 1; ch < 4; ++ch) {
                    ptx::tmem_ld_32x32(ts + ch * 32, *reinterpret_cast<uint32_t(*)[32]>(&r[ch * 32]));
                }
                stamp<TRACE>(p, scount, t * 10 + 1);
                // The last block of a ragged sequence holds columns that do not exist: they become -inf, which
                // no maximum sees, and exp_chunk gives them no weight.
                auto mask = [&](int from) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        if (from + i >= valid) {
                            r[from + i] = 0xff800000u;
                        }
                    }
                };
                if (j == j_first) {
                    ptx::tmem_ld_wait();
                    if (valid < BN) {
                        mask(0);
                        mask(32);
                        mask(64);
                        mask(96);
                    }
                    float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                    for (int i = 0; i < BN; i += 8) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            mx4[u] = ptx::max3_nan(mx4[u], __uint_as_float(r[i + 2 * u]), __uint_as_float(r[i + 2 * u + 1]));
                        }
                    }
                    const float mx = ptx::max3_nan(ptx::max3_nan(mx4[0], mx4[1], mx4[2]), mx4[3], mx4[3]);
                    begun          = mx != -INFINITY;
                    m_ref          = begun ? mx : 0.0f;
                }
                uint32_t pk[48];
                float    s4[4] = {0.f, 0.f, 0.f, 0.f};
                float    nmc = -m_ref * c;
                // P = exp2(S * c - m_ref * c) as packed bf16, three quarters of the row
                if (valid == BN) {
                    exp_chunk<NP>(&r[0], c, nmc, s4, &pk[0]);
                    ptx::tmem_ld_wait();
                    exp_chunk<NP>(&r[32], c, nmc, s4, &pk[16]);
                    exp_chunk<NP>(&r[64], c, nmc, s4, &pk[32]);
                }
                else {
                    mask(0);
                    exp_chunk<0, true>(&r[0], c, nmc, s4, &pk[0], valid);
                    ptx::tmem_ld_wait();
                    mask(32);
                    mask(64);
                    mask(96);
                    exp_chunk<0, true>(&r[32], c, nmc, s4, &pk[16], valid - 32);
                    exp_chunk<0, true>(&r[64], c, nmc, s4, &pk[32], valid - 64);
                }
                float mx2[2] = {-INFINITY, -INFINITY};
#pragma unroll
                for (int i = 96; i < BN; i += 4) {
                    mx2[0] = ptx::max3_nan(mx2[0], __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
                    mx2[1] = ptx::max3_nan(mx2[1], __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
                }
#pragma unroll
                for (int i = 0; i < 48; ++i) {
                    if (on_fma_pipe<NP>(i % 16)) {
                        mx2[i & 1] = ptx::max3_nan(mx2[i & 1], __uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
                    }
                }
                const float tail = ptx::max3_nan(mx2[0], mx2[1], mx2[1]);
                const float part = (s4[0] + s4[1]) + (s4[2] + s4[3]);
                const float last = fmaf(tail, c, nmc);
                // A NaN among the scores reaches `part` or `last` and fails their test: the slow path and the last
                // quarter behind it then run on the special-function unit, which keeps it (the FMA-pipe form's clamp
                // would turn it into a number).
                const bool fine = part < RANGE_SUM && last < RANGE && begun;
                const bool slow = __any_sync(0xffffffffu, !fine);
                if (slow) {
                    // The maximum of the whole row; the first three quarters are still in tensor memory.
                    float mx = tail;
#pragma unroll 1
                    for (int ch = 0; ch < 6; ++ch) {
                        uint32_t rs[16];
                        ptx::tmem_ld_32x16(ts + ch * 16, rs);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            mx = ch * 16 + i < valid ? fmaxf(mx, __uint_as_float(rs[i])) : mx;
                        }
                    }
                    const float m_new = fine || mx == -INFINITY ? m_ref : mx;
                    if (j != j_first) {  // the commit behind S_t also covers the product before it: O is complete
                        const float alpha = begun ? ptx::ex2((m_ref - m_new) * c) : 1.0f;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            l4[u] *= alpha;
                        }
#pragma unroll 1
                        for (int ch = 0; ch < 8; ++ch) {
                            uint32_t ro[16];
                            ptx::tmem_ld_32x16(to + ch * 16, ro);
                            ptx::tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                ro[i] = __float_as_uint(__uint_as_float(ro[i]) * alpha);
                            }
                            ptx::tmem_st_32x16(to + ch * 16, ro);
                        }
                        ptx::tmem_st_wait();
                    }
                    m_ref = m_new;
                    begun = begun || mx != -INFINITY;
                    nmc   = -m_ref * c;
                    s4[0] = s4[1] = s4[2] = s4[3] = 0.f;
#pragma unroll
                    for (int ch = 0; ch < 3; ++ch) {
                        ptx::tmem_ld_32x32(ts + ch * 32, *reinterpret_cast<uint32_t(*)[32]>(&r[ch * 32]));
                        ptx::tmem_ld_wait();
                        if (valid < BN) {
                            mask(ch * 32);
                        }
                        exp_chunk<0, true>(&r[ch * 32], c, nmc, s4, &pk[ch * 16], valid - ch * 32);
                    }
                }
                stamp<TRACE>(p, scount, t * 10 + 2);
                // written over S, of which only the last quarter is still needed and in registers
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) {
                    ptx::tmem_st_32x16(ts + ch * 16, *reinterpret_cast<uint32_t(*)[16]>(&pk[ch * 16]));
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    l4[u] += s4[u];
                }
                stamp<TRACE>(p, scount, t * 10 + 3);
                ptx::tmem_st_wait();
                ptx::tc_fence_before();
                ptx::mbar_arrive_warp(&bar.p_lo[t]);
                stamp<TRACE>(p, scount, t * 10 + 4);
                if (valid == BN && !slow) {
                    exp_chunk<NP>(&r[96], c, nmc, l4, pk);
                }
                else {
                    exp_chunk<0, true>(&r[96], c, nmc, l4, pk, valid - 96);
                }
                ptx::tmem_st_32x16(ts + 48, *reinterpret_cast<uint32_t(*)[16]>(&pk[0]));
                stamp<TRACE>(p, scount, t * 10 + 5);
                ptx::tmem_st_wait();
                ptx::tc_fence_before();
                ptx::mbar_arrive_warp(&bar.p_hi[t]);
                stamp<TRACE>(p, scount, t * 10 + 6);
            }
            if (SPLIT) {
                ok = ok && ptx::mbar_wait(&bar.o_final[t], wc & 1u);
                if (!ok) {
                    flag(p, ERR_SOFTMAX);
                }
                join_shares(p, b, h, row, t, quarter, lane, to, begun ? m_ref * c : -INFINITY, (l4[0] + l4[1]) + (l4[2] + l4[3]), crank, csize, base,
                            sv_addr + KV_STAGES * TILE_BYTES + (warp - 4) * OUT_BYTES);
                break;
            }
            if (!ok) {
                break;
            }
            // epilogue: O / l -> bf16, log-sum-exp
            if (!ptx::mbar_wait(&bar.o_final[t], wc & 1u)) {
                flag(p, ERR_SOFTMAX);
                break;
            }
            float l = (l4[0] + l4[1]) + (l4[2] + l4[3]), m_log2 = begun ? m_ref * c : -INFINITY;
            float weight[QT] = {1.0f, 1.0f};  // of the two O of a row (kOneTile)
            if (ONE) {
                const uint32_t pair = sq_addr + TILE_BYTES + row_in * 8;  // where the second query tile would be
                ptx::st_shared_v2f(pair + t * BM * 8, m_log2, l);
                ptx::mbar_arrive_warp(&bar.merge);
                if (!ptx::mbar_wait(&bar.merge, wc & 1u) || !ptx::mbar_wait(&bar.o_final[t ^ 1], wc & 1u)) {
                    flag(p, ERR_SOFTMAX);
                    break;
                }
                const float2 a = ptx::ld_shared_v2f(pair), d = ptx::ld_shared_v2f(pair + BM * 8);
                m_log2    = fmaxf(a.x, d.x);
                weight[0] = ptx::ex2(a.x - m_log2);
                weight[1] = ptx::ex2(d.x - m_log2);
                l         = weight[0] * a.y + weight[1] * d.y;
            }
            ptx::tc_fence_after();
            const float    inv    = 1.0f / l;
            const bool     row_ok = row < p.Sq;
            // A thread has a row; written straight out, every store instruction would touch 32 lines (3700
            // clocks for the CTA's tile). Through shared memory eight lanes write 128 bytes of one row.
            const uint32_t stage = sv_addr + KV_STAGES * TILE_BYTES + (warp - 4) * OUT_BYTES;
            const int      row_w = row - lane;  // first row of this warp
            __nv_bfloat16* dst   = p.o + b * p.o_batch + static_cast<int64_t>(row_w + (lane >> 3)) * p.o_row + h * p.o_head
                                 + (lane & 7) * 8;
#pragma unroll 1
            for (int half = ONE ? t : 0; half < (ONE ? t + 1 : 2); ++half) {  // kOneTile: 64 columns for each half of the warps
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t r[32];
                    if (ONE) {
                        uint32_t r1[32];
                        ptx::tmem_ld_32x32(tmem + 256 + lane_off + half * 64 + ch * 32, r);
                        ptx::tmem_ld_32x32(tmem + 384 + lane_off + half * 64 + ch * 32, r1);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            r[i] = __float_as_uint(__uint_as_float(r[i]) * weight[0] + __uint_as_float(r1[i]) * weight[1]);
                        }
                    }
                    else {
                        ptx::tmem_ld_32x32(to + half * 64 + ch * 32, r);
                        ptx::tmem_ld_wait();
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        uint32_t pk[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            pk[i] = ptx::pack_bf16x2(__uint_as_float(r[8 * g + 2 * i]) * inv, __uint_as_float(r[8 * g + 2 * i + 1]) * inv);
                        }
                        ptx::st_shared_v4(stage + lane * 128 + (((ch * 4 + g) ^ (lane & 7)) << 4), make_uint4(pk[0], pk[1], pk[2], pk[3]));
                    }
                }
                if (ONE) {
                    ptx::tc_fence_before();
                    ptx::mbar_arrive_warp(&bar.o_free[0]);
                    ptx::mbar_arrive_warp(&bar.o_free[1]);
                }
                else if (half == 1) {  // O is in registers or on its way out: the next item's first product may overwrite it
                    ptx::tc_fence_before();
                    ptx::mbar_arrive_warp(&bar.o_free[t]);
                }
                __syncwarp();
                uint4 v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = i * 4 + (lane >> 3);
                    v[i]        = ptx::ld_shared_v4(stage + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (row_w + i * 4 + (lane >> 3) < p.Sq) {
                        ptx::st_v4(dst + half * 64 + i * 4 * p.o_row, v[i]);
                    }
                }
            }
            if (row_ok && p.lse && (!ONE || t == 0)) {
                p.lse[(static_cast<int64_t>(b) * p.H + h) * p.Sq + row] = (m_log2 + ptx::lg2(l)) * 0.6931471805599453f;
            }
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tmem_dealloc<512>(tmem);
    }
}

// Items beyond whole waves of one per SM are shared out, see cluster_plan.h. Times in kv tiles (1.45 us).
// 8191 tokens x 10 heads (320 items on 148 SMs): 304 -> 249 us; 4000 x 10 (160 items): 104 -> 75.
fu::ClusterPlan plan_split(int items, int n_kv, int sms, int dev)
{
    static fu::ClusterCapacity capacity;
    return fu::plan_clusters(items, n_kv, sms, {3.0, 4.5, 2.0}, [&](int csize) {
        return capacity.of(fmha_fwd_kernel<kPolyPairs, false, Form::kShared>, csize, dev, THREADS, SMEM_BYTES);
    });
}

}  // namespace

extern "C" int fu_fmha_fwd(const FuFmhaArgs* a, void* stream)
{
    if (!a || !a->q || !a->k || !a->v || !a->o) {
        return fu::fail(FU_E_ARG, "fu_fmha_fwd: null operand");
    }
    if (a->head_dim != D) {
        return fu::fail(FU_E_UNSUPPORTED, "fu_fmha_fwd: head_dim %d (only 128 is built)", a->head_dim);
    }
    if (a->batch < 1 || a->heads < 1 || a->seq_q < 1 || a->seq_kv < 1) {
        return fu::fail(FU_E_ARG, "fu_fmha_fwd: empty problem");
    }
    if ((reinterpret_cast<uintptr_t>(a->o) & 15u) || (a->o_row % 8) || (a->o_head % 8) || (a->o_batch % 8)) {
        return fu::fail(FU_E_ARG, "fu_fmha_fwd: o needs 16-byte aligned rows");
    }
    Params p{};
    int    rc = make_map_bshd(&p.map_q, a->q, a->batch, a->seq_q, a->heads, a->q_row, a->q_head, a->q_batch, BM);
    if (rc == FU_OK) {
        rc = make_map_bshd(&p.map_k, a->k, a->batch, a->seq_kv, a->heads, a->k_row, a->k_head, a->k_batch, BN);
    }
    if (rc == FU_OK) {
        rc = make_map_bshd(&p.map_v, a->v, a->batch, a->seq_kv, a->heads, a->v_row, a->v_head, a->v_batch, BN);
    }
    if (rc != FU_OK) {
        return rc;
    }
    p.o          = static_cast<__nv_bfloat16*>(a->o);
    p.lse        = a->lse;
    p.o_row      = a->o_row;
    p.o_head     = a->o_head;
    p.o_batch    = a->o_batch;
    p.B          = a->batch;
    p.H          = a->heads;
    p.Sq         = a->seq_q;
    p.Skv        = a->seq_kv;
    p.q_blocks   = (a->seq_q + QT * BM - 1) / (QT * BM);
    p.total_work = p.q_blocks * p.H * p.B;
    p.n_kv       = (a->seq_kv + BN - 1) / BN;
    p.scale      = a->scale;
    p.scale_log2 = a->scale * 1.4426950408889634f;
    p.err        = a->err;
    p.overlap    = a->ctas <= 0;

    int dev = 0, sms = 0;
    FU_CUDA_OK(cudaGetDevice(&dev));
    FU_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // how many of every 16 exponential pairs go to the FMA pipe: FU_FMHA_POLY(n) in flags, default kPolyPairs
    const int np = (a->flags & FU_FMHA_POLY_SET) ? ((a->flags >> 8) & 15) : kPolyPairs;
    if (np < 0 || np > 6 || (np & 1)) {
        return fu::fail(FU_E_ARG, "fu_fmha_fwd: %d of 16 exponential pairs on the FMA pipe is not built (0, 2, 4, 6)", np);
    }
    auto launch = [&](auto kernel) -> int {
        const int limit = fu::raise_smem_limit(kernel, SMEM_BYTES);
        if (limit != FU_OK) {
            return limit;
        }
        int grid = a->ctas > 0 ? std::min(a->ctas, sms) : sms;
        grid     = std::max(1, std::min(grid, p.total_work));
        if (p.overlap) {
            FU_CUDA_OK(fu::launch_behind(kernel, dim3(static_cast<unsigned>(grid)), dim3(THREADS), SMEM_BYTES, static_cast<cudaStream_t>(stream), p));
            return FU_OK;
        }
        kernel<<<grid, THREADS, SMEM_BYTES, static_cast<cudaStream_t>(stream)>>>(p);
        FU_CUDA_OK(cudaGetLastError());
        return FU_OK;
    };
    p.trace = a->trace;
    if (a->trace) {
        if (np != kPolyPairs) {
            return fu::fail(FU_E_ARG, "fu_fmha_fwd: the timeline build exists for the default exponential split only");
        }
        return launch(fmha_fwd_kernel<kPolyPairs, true, Form::kTwoTiles>);
    }
    if (np == kPolyPairs && a->ctas <= 0) {
        const fu::ClusterPlan plan = plan_split(p.total_work, p.n_kv, sms, dev);
        // One query tile per item where that takes fewer steps of the busiest SM; its steps are a tenth longer
        // (K and V are read twice as often). 2 x 1000 tokens x 5 heads (80 items instead of 40 in clusters of
        // three): 16.0 -> 11.8 us; 4000 x 4: 35.2 -> 30.7; 1000 x 20 would take two waves, 20.8 for 18.0.
        const int one_blocks = (a->seq_q + BM - 1) / BM, one_items = one_blocks * p.H * p.B;
        if (p.n_kv > 1 && ((one_items + sms - 1) / sms) * 1.1 * ((p.n_kv + 1) / 2 + 3.0) < plan.cost) {
            p.q_blocks   = one_blocks;
            p.total_work = one_items;
            return launch(fmha_fwd_kernel<kPolyPairs, false, Form::kOneTile>);
        }
        if (plan.csize > 1) {
            const int items = p.total_work;
            p.total_work    = plan.whole;
            if (plan.whole > 0) {
                rc = launch(fmha_fwd_kernel<kPolyPairs, false, Form::kTwoTiles>);
                if (rc != FU_OK) {
                    return rc;
                }
            }
            p.first                   = plan.whole;
            cudaLaunchConfig_t  cfg   = {};
            cudaLaunchAttribute attr  = fu::cluster_attr(plan.csize);
            cfg.gridDim               = dim3(static_cast<unsigned>((items - plan.whole) * plan.csize), 1, 1);
            cfg.blockDim              = dim3(THREADS, 1, 1);
            cfg.dynamicSmemBytes      = SMEM_BYTES;
            cfg.stream                = static_cast<cudaStream_t>(stream);
            cfg.attrs                 = &attr;
            cfg.numAttrs              = 1;
            FU_CUDA_OK(cudaLaunchKernelEx(&cfg, fmha_fwd_kernel<kPolyPairs, false, Form::kShared>, p));
            return FU_OK;
        }
    }
    switch (np) {
    case 0: return launch(fmha_fwd_kernel<0, false, Form::kTwoTiles>);
    case 2: return launch(fmha_fwd_kernel<2, false, Form::kTwoTiles>);
    case 4: return launch(fmha_fwd_kernel<4, false, Form::kTwoTiles>);
    case 6: return launch(fmha_fwd_kernel<6, false, Form::kTwoTiles>);
    default: return fu::fail(FU_E_ARG, "fu_fmha_fwd: %d of 16 exponential pairs on the FMA pipe is not built (0, 2, 4, 6)", np);
    }
}
