// tcgen05 GEMM kernels built on gemm_sm100.cuh:
//
//   fu_gemm_bf16          C = act(A * B^T + bias) + residual, bf16 in/out, fp32 accumulate.
//   fu_qkv_rope_scatter   the fused mode-0 path: QKV projection whose epilogue applies per-head
//                         RMSNorm and 3D RoPE to q and k in registers and stores every head-row
//                         straight into the owning rank's q/k/v window at its permuted
//                         (sequence-gathered, head-scattered) position over NVLink. The all-to-all
//                         is the address of the store; there is no separate exchange or permute.
//
// The reference has no GEMM: its example wraps nn.Linear + separate norm/RoPE around two
// all_to_all_4d calls (examples/dit_attention.py:45-63). These kernels replace that composition.
#include "cluster_plan.h"
#include "fu_kernels.h"
#include "gemm_sm100.cuh"
#include "host_util.h"
#include "tma_host.h"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <limits>

namespace {

using namespace fu;
using namespace fu::gemm;

// ---- plain epilogue --------------------------------------------------------------------------------
// GELU(x) = x * sigmoid(2u), u = sqrt(2/pi) (x + 0.044715 x^3), written with one exponential and one
// reciprocal: 1 + tanh(u) = 2 sigmoid(2u), without tanhf's branches and without the cancellation of
// 1 + tanh for negative x. The approximations' relative error (about 1e-6) is far below the bf16 result's.
__device__ __forceinline__ float sigmoid2(float u)
{
    return __fdividef(1.0f, 1.0f + __expf(-2.0f * u));
}
__device__ __forceinline__ float gelu_tanh(float x)
{
    return x * sigmoid2(0.7978845608028654f * x * (1.0f + 0.044715f * x * x));
}
__device__ __forceinline__ float gelu_erf(float x)
{
    return 0.5f * x * (1.0f + erff(x * 0.7071067811865476f));
}
__device__ __forceinline__ float gelu_tanh_grad(float x)
{
    const float x2 = x * x;
    const float s  = sigmoid2(0.7978845608028654f * x * (1.0f + 0.044715f * x2));
    return s + x * s * (1.0f - s) * 1.5957691216057308f * (1.0f + 0.134145f * x2);
}

// ACT: 0 none, 1 GELU (tanh form), 2 GELU (erf form), 3 the tanh form's derivative at aux.
template <int ACT>
struct PlainEpi {
    static constexpr bool kPeers = false;
    __nv_bfloat16*       c;
    const __nv_bfloat16* residual;
    const void*          bias;
    int64_t              ldc;
    int                  M, N, bias_bf16;
    const __nv_bfloat16* aux;    // act 3: where the tanh-form GELU's derivative is evaluated
    __nv_bfloat16*       c_pre;  // optional second output: the value before the activation
    float                ahead[4];

    __device__ void open(int) {}
    __device__ void close(int) {}

    template <int W>
    __device__ __forceinline__ static void pack_row(const float (&v)[W], uint32_t stage, int lane)
    {
#pragma unroll
        for (int g = 0; g < W / 8; ++g) {
            ptx::st_shared_v4(stage_unit(stage, lane, g), make_uint4(pack_bf16(v[8 * g], v[8 * g + 1]), pack_bf16(v[8 * g + 2], v[8 * g + 3]),
                                                                     pack_bf16(v[8 * g + 4], v[8 * g + 5]), pack_bf16(v[8 * g + 6], v[8 * g + 7])));
        }
    }

    // The bias of the 128 columns from col0 on, four a lane, while their products are still being computed: the loads' latency
    // behind the products cost a unit 0.7 us (256 x 512 x 256 with GELU 5.9 us so, 6.7 with read-only loads of all 64 columns by
    // every thread, 10 % more with ordinary ones). A warp with 64 columns fetches 128 too: told not to, launches take 0.3 % longer.
    __device__ __forceinline__ void fetch(int col0, int lane)
    {
        if (bias) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int col = col0 + lane * 4 + k;
                ahead[k]      = col >= N ? 0.0f : bias_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(bias)[col])
                                                            : static_cast<const float*>(bias)[col];
            }
        }
    }

    // W columns of 32 rows, a row per thread; none from column N on. Lane `first` has fetched the bias of the first four.
    // Each thread needs all of them: they go through the staging buffer.
    template <int W>
    __device__ __forceinline__ void piece(float (&v)[W], int row0, int col0, int N, int lane, uint32_t stage, int first = 0) const
    {
        if (row0 >= M || col0 >= N) {
            return;  // warp-uniform
        }
        if (bias) {
            if (lane >= first && lane < first + W / 4) {
                ptx::st_shared_v4(stage + (lane - first) * 16, make_uint4(__float_as_uint(ahead[0]), __float_as_uint(ahead[1]),
                                                                          __float_as_uint(ahead[2]), __float_as_uint(ahead[3])));
            }
            __syncwarp();
#pragma unroll
            for (int g = 0; g < W / 4; ++g) {
                const uint4 q = ptx::ld_shared_v4(stage + g * 16);
                v[4 * g] += __uint_as_float(q.x), v[4 * g + 1] += __uint_as_float(q.y);
                v[4 * g + 2] += __uint_as_float(q.z), v[4 * g + 3] += __uint_as_float(q.w);
            }
            __syncwarp();
        }
        if (c_pre) {
            pack_row(v, stage, lane);
            stage_out<W>(stage, c_pre, ldc, row0, col0, M, N, lane);
        }
        if (ACT == 1 || ACT == 2) {
#pragma unroll
            for (int j = 0; j < W; ++j) {
                v[j] = ACT == 1 ? gelu_tanh(v[j]) : gelu_erf(v[j]);
            }
        }
        if (ACT == 3) {
            stage_in<W>(stage, aux, ldc, row0, col0, M, N, lane);
#pragma unroll
            for (int g = 0; g < W / 8; ++g) {
                const uint4           q = ptx::ld_shared_v4(stage_unit(stage, lane, g));
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 f = __bfloat1622float2(h[k]);
                    v[8 * g + 2 * k] *= gelu_tanh_grad(f.x);
                    v[8 * g + 2 * k + 1] *= gelu_tanh_grad(f.y);
                }
            }
        }
        if (residual) {
            stage_in<W>(stage, residual, ldc, row0, col0, M, N, lane);
#pragma unroll
            for (int g = 0; g < W / 8; ++g) {
                const uint4           q = ptx::ld_shared_v4(stage_unit(stage, lane, g));
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 f = __bfloat1622float2(h[k]);
                    v[8 * g + 2 * k] += f.x;
                    v[8 * g + 2 * k + 1] += f.y;
                }
            }
        }
        pack_row(v, stage, lane);
        stage_out<W>(stage, c, ldc, row0, col0, M, N, lane);
    }

    // Half a unit: a warp's share of a small tile.
    __device__ __forceinline__ void unit(const uint32_t (&r)[64], int row0, int col0, int col_end, int lane, uint32_t stage) const
    {
        float v[64];
#pragma unroll
        for (int j = 0; j < 64; ++j) {
            v[j] = __uint_as_float(r[j]);
        }
        piece<64>(v, row0, col0, min(N, col_end), lane, stage);
    }

    __device__ __forceinline__ void unit(const uint32_t (&r)[128], int row0, int col0, int col_end, int lane, uint32_t stage) const
    {
        const int end = min(N, col_end);
        float     v[64];
#pragma unroll
        for (int j = 0; j < 64; ++j) {
            v[j] = __uint_as_float(r[j]);
        }
        // One copy of the code: with both halves unrolled, fetching it took the first unit of a launch that finds other
        // kernels' code in the caches 24000 clocks instead of 11000 (256 x 512 x 256 with GELU: 20.5 -> 14.4 us).
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            piece<64>(v, row0, col0 + h * 64, end, lane, stage, h * 16);
#pragma unroll
            for (int j = 0; j < 64; ++j) {
                v[j] = __uint_as_float(r[64 + j]);
            }
        }
    }
};

template <int ACT>
struct PlainArgs {
    WideCore      core;
    PlainEpi<ACT> epi;
};

template <int MB, int NB, int ACT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WIDE_THREADS, 1) gemm_wide_kernel(const __grid_constant__ PlainArgs<ACT> a)
{
    PlainEpi<ACT> epi = a.epi;
    run_wide<MB, NB, false>(a.core, epi);
}

template <int ACT>
__global__ void __launch_bounds__(WIDE_THREADS, 1) gemm_wide_split_kernel(const __grid_constant__ PlainArgs<ACT> a)
{
    PlainEpi<ACT> epi = a.epi;
    run_wide<1, 2, true>(a.core, epi);
}

template <int ACT>
__global__ void __launch_bounds__(small_threads(64), 1) gemm_small_kernel(const __grid_constant__ PlainArgs<ACT> a)
{
    PlainEpi<ACT> epi = a.epi;
    run_small<false, 64>(a.core, epi);
}

template <int ACT>
__global__ void __launch_bounds__(small_threads(128), 1) gemm_split_kernel(const __grid_constant__ PlainArgs<ACT> a)
{
    PlainEpi<ACT> epi = a.epi;
    run_small<true, 128>(a.core, epi);
}

// ---- fused QKV epilogue: RMSNorm + 3D RoPE + scatter ---------------------------------------------------
constexpr int HEAD_DIM = 128;
constexpr int MAX_HEADS = 128;

struct QkvParams {
    uint8_t*      win[3][FU_MAX_WORLD];  // q, k, v window base on every rank
    Peers         peers;
    const float2* rope;     // [s_local][64] (cos, sin) per rotated pair
    const float*  gamma_q;  // [128]
    const float*  gamma_k;
    float         eps;
    int           M, heads;          // rows = b * s_local; heads per projection
    int64_t       s_local, seq_off, s_total;
    uint8_t       owner[MAX_HEADS];  // head -> rank that owns it
    uint8_t       local[MAX_HEADS];  // head -> index inside its owner's shard
    uint8_t       heads_of[FU_MAX_WORLD];
    int           handshake;
    int           n_types, n_normed;
    int           tables_aligned;  // rope and both gammas to 16 bytes
    __nv_bfloat16* y_save;
    int64_t       ld_y;
};

// The functor keeps a reference to the parameters (they stay in the kernel's constant bank) and
// only its own mutable state in registers. A unit is one head of 32 tokens: a thread has the whole
// 128-value row in registers, so the sum of squares needs no second read of the accumulator.
template <int EPI_THREADS>
struct QkvEpi {
    static constexpr bool kPeers = true;
    const QkvParams& p;
    uint64_t         base_epoch;

    __device__ explicit QkvEpi(const QkvParams& params) : p(params), base_epoch(0) {}
    __device__ void fetch(int, int) {}

    __device__ void open(int epi_tid)
    {
        const Peers& peers     = p.peers;
        const int    handshake = p.handshake;
        base_epoch = *reinterpret_cast<volatile uint64_t*>(&peers.own->epoch);
        if (handshake && epi_tid < 32) {
            if (blockIdx.x == 0) {
                hs_announce(peers, base_epoch + 1);
            }
            hs_await(peers, base_epoch + 1, FU_ST_OPEN_TIMEOUT);
        }
        epi_barrier(EPI_THREADS);  // no epilogue thread stores to a peer before the owners said "go"
    }

    __device__ void close(int epi_tid)
    {
        __shared__ uint32_t ticket;
        const Peers& peers     = p.peers;
        const int    handshake = p.handshake;
        ptx::fence_sys();
        epi_barrier(EPI_THREADS);
        if (epi_tid == 0) {
            ticket = atomicAdd(&peers.own->arrive[0], 1u);
        }
        epi_barrier(EPI_THREADS);
        if (ticket == gridDim.x - 1 && epi_tid < 32) {
            if (handshake) {
                ptx::fence_sys();
                hs_announce(peers, base_epoch + 2);
                hs_await(peers, base_epoch + 2, FU_ST_CLOSE_TIMEOUT);
            }
            if (epi_tid == 0) {
                peers.own->arrive[0] = 0;
                __threadfence();
                *reinterpret_cast<volatile uint64_t*>(&peers.own->epoch) = base_epoch + 2;
            }
        }
    }

    // Four neighbours of a table that the caller need not have aligned to more than its elements.
    __device__ __forceinline__ float4 load4(const float* p) const
    {
        if (this->p.tables_aligned) {
            return *reinterpret_cast<const float4*>(p);
        }
        return make_float4(p[0], p[1], p[2], p[3]);
    }

    // 64 columns of a head: rotate (NORMED), round, and store each row's 128 bytes to its owner. The
    // staging buffer makes every store instruction write whole 128-byte lines: written straight from
    // the accumulator layout (a lane is a row) each would scatter 32 separate 16-byte pieces, which
    // NVLink carries at a fraction of its rate.
    template <int H, bool NORMED>
    __device__ __forceinline__ void half(const uint32_t (&r)[128], float scale, const float* gamma, const float2* cs,
                                         unsigned long long my_dst, int lane, uint32_t stage) const
    {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            uint32_t o[4];
            if (NORMED) {
                const float4 g0 = load4(gamma + H * 64 + g * 8);
                const float4 g1 = load4(gamma + H * 64 + g * 8 + 4);
                const float  gm[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
                const float4 t0 = load4(&cs[H * 32 + g * 4].x);
                const float4 t1 = load4(&cs[H * 32 + g * 4 + 2].x);
                const float  cc[4] = {t0.x, t0.z, t1.x, t1.z}, sn[4] = {t0.y, t0.w, t1.y, t1.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float x0 = __uint_as_float(r[H * 64 + g * 8 + 2 * k]) * scale * gm[2 * k];
                    const float x1 = __uint_as_float(r[H * 64 + g * 8 + 2 * k + 1]) * scale * gm[2 * k + 1];
                    o[k]           = pack_bf16(x0 * cc[k] - x1 * sn[k], x0 * sn[k] + x1 * cc[k]);
                }
            }
            else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    o[k] = pack_bf16(__uint_as_float(r[H * 64 + g * 8 + 2 * k]), __uint_as_float(r[H * 64 + g * 8 + 2 * k + 1]));
                }
            }
            ptx::st_shared_v4(stage_unit(stage, lane, g), make_uint4(o[0], o[1], o[2], o[3]));
        }
        __syncwarp();
        uint4              v[8];
        unsigned long long to[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int from = i * 4 + (lane >> 3);
            v[i]           = ptx::ld_shared_v4(stage_unit(stage, from, lane & 7));
            to[i]          = __shfl_sync(0xffffffffu, my_dst, from);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (to[i]) {
                ptx::st_v4(reinterpret_cast<uint4*>(to[i]) + H * 8 + (lane & 7), v[i]);
            }
        }
        __syncwarp();  // the buffer may be refilled
    }

    template <int H>
    __device__ __forceinline__ void save(const uint32_t (&r)[128], int row0, int col0, int lane, uint32_t stage) const
    {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            uint32_t o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                o[k] = pack_bf16(__uint_as_float(r[H * 64 + g * 8 + 2 * k]), __uint_as_float(r[H * 64 + g * 8 + 2 * k + 1]));
            }
            ptx::st_shared_v4(stage_unit(stage, lane, g), make_uint4(o[0], o[1], o[2], o[3]));
        }
        stage_out<64>(stage, p.y_save, p.ld_y, row0, col0 + H * 64, p.M, 0x7fffffff, lane);
    }

    __device__ __forceinline__ void unit(const uint32_t (&r)[128], int row0, int col0, int, int lane, uint32_t stage) const
    {
        const int head_global = col0 / HEAD_DIM;
        const int type        = head_global / p.heads;  // 0 q, 1 k, 2 v
        if (row0 >= p.M || type >= p.n_types) {
            return;  // warp-uniform
        }
        const int     row    = row0 + lane;
        const bool    row_ok = row < p.M;
        const int64_t batch  = row / p.s_local;
        const int64_t s      = row - batch * p.s_local;
        const int     head   = head_global - type * p.heads;
        const int     peer   = p.owner[head];
        const int64_t hp     = p.heads_of[peer];
        uint8_t*      dst    = p.win[type][peer] + (((batch * p.s_total + p.seq_off + s) * hp + p.local[head]) * HEAD_DIM) * 2;
        const unsigned long long my_dst = row_ok ? reinterpret_cast<unsigned long long>(dst) : 0ull;
        if (type < p.n_normed) {
            float ss4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < HEAD_DIM; ++j) {
                const float x = __uint_as_float(r[j]);
                ss4[j & 3] += x * x;
            }
            const float   scale = rsqrtf(((ss4[0] + ss4[1]) + (ss4[2] + ss4[3])) * (1.0f / HEAD_DIM) + p.eps);
            const float*  gamma = type == 0 ? p.gamma_q : p.gamma_k;
            const float2* cs    = p.rope + (row_ok ? s : 0) * (HEAD_DIM / 2);
            if (p.y_save) {
                save<0>(r, row0, col0, lane, stage);
                save<1>(r, row0, col0, lane, stage);
            }
            half<0, true>(r, scale, gamma, cs, my_dst, lane, stage);
            half<1, true>(r, scale, gamma, cs, my_dst, lane, stage);
        }
        else {
            half<0, false>(r, 1.0f, nullptr, nullptr, my_dst, lane, stage);
            half<1, false>(r, 1.0f, nullptr, nullptr, my_dst, lane, stage);
        }
    }
};

struct QkvArgs {
    WideCore  core;
    QkvParams epi;
};

template <int MB, int NB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WIDE_THREADS, 1) qkv_wide_kernel(const __grid_constant__ QkvArgs a)
{
    QkvEpi<32 * WIDE_EPI_WARPS> epi(a.epi);
    run_wide<MB, NB, false>(a.core, epi);
}

__global__ void __launch_bounds__(small_threads(128), 1) qkv_small_kernel(const __grid_constant__ QkvArgs a)
{
    QkvEpi<32 * small_epi_warps(128)> epi(a.epi);
    run_small<false, 128>(a.core, epi);
}

// ---- fused mode-1 path: pull attention output from peers, feed the output projection -----------------
// A[m, head*128 + x] = O_owner(head)[batch, seq_off + s, local head, x]. Four extra warps per CTA
// copy (M-tile, peer) blocks from the peers' O buffers into a local gather buffer with plain
// loads over NVLink and publish a flag per block; the TMA producer of whichever CTA needs that
// part of A waits for the flag (bounded) and then loads it from local memory, so every remote byte
// crosses NVLink once and the transfer overlaps the GEMM tile by tile. No multicast anywhere.
struct PullParams {
    const uint8_t* peer_o[FU_MAX_WORLD];
    Peers          peers;
    uint8_t*       gather;   // (M, heads_total * 128) bf16, local
    uint32_t*      ready;    // [tiles_m * world], zero before launch
    int            M, tiles_m, heads_total;
    int64_t        s_local, seq_off, s_total;
    uint8_t        heads_of[FU_MAX_WORLD];
    uint16_t       head_start[FU_MAX_WORLD];
    uint8_t        owner[MAX_HEADS];
    int            handshake;
    uint32_t*      err;
};

struct PullSrc {
    const PullParams& p;
    int               seen_mt, seen_peer;
    __device__ explicit PullSrc(const PullParams& params) : p(params), seen_mt(-1), seen_peer(-1) {}

    __device__ bool ready(int mt, int kb)
    {
        const int peer = p.owner[kb >> 1];  // BK = 64: two K-blocks per head
        if (mt == seen_mt && peer == seen_peer) {
            return true;
        }
        const uint32_t* f  = p.ready + mt * p.peers.world + peer;
        const uint64_t  t0 = ptx::globaltimer_ns();
        uint32_t        spins = 0;
        while (ptx::ld_acquire_gpu_u32(f) == 0u) {
            if ((++spins & 255u) == 0u && ptx::globaltimer_ns() - t0 > p.peers.timeout_ns) {
                return false;
            }
        }
        ptx::fence_proxy_async();  // generic-proxy writes by the pullers -> TMA reads below
        seen_mt   = mt;
        seen_peer = peer;
        return true;
    }
};

struct PullAux {
    static constexpr int kWarps = 4;
    const PullParams&    p;
    __device__ explicit PullAux(const PullParams& params) : p(params) {}

    __device__ static void aux_barrier() { asm volatile("bar.sync 2, 128;" ::: "memory"); }

    __device__ void run(int aux_warp, int lane) const
    {
        __shared__ uint32_t ticket;
        const Peers&   peers = p.peers;
        const int      tid   = aux_warp * 32 + lane;
        const uint64_t base  = *reinterpret_cast<volatile uint64_t*>(&peers.own->epoch);
        // Opening: every rank says "my attention output is complete" (stream order put this kernel
        // after its attention kernel) and nobody reads a peer before that.
        if (p.handshake && aux_warp == 0) {
            if (blockIdx.x == 0) {
                hs_announce(peers, base + 1);
            }
            hs_await(peers, base + 1, FU_ST_OPEN_TIMEOUT);
        }
        aux_barrier();
        const int units = p.tiles_m * peers.world;
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            const int mt   = u / peers.world;
            const int peer = (peers.rank + (u - mt * peers.world)) % peers.world;
            const int rows = min(BM, p.M - mt * BM);
            const uint32_t vpr  = static_cast<uint32_t>(p.heads_of[peer]) * 16u;  // 16-byte vectors per row
            const uint32_t nvec = vpr * rows;
            const uint8_t* src  = p.peer_o[peer];
            const int64_t  src_pitch = static_cast<int64_t>(p.heads_of[peer]) * 256;
            const int64_t  dst_pitch = static_cast<int64_t>(p.heads_total) * 256;
            uint8_t*       dst  = p.gather + static_cast<int64_t>(p.head_start[peer]) * 256;
            for (uint32_t v0 = tid; v0 < nvec; v0 += 8 * 128) {
                uint4    val[8];
                uint8_t* to[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t v = v0 + k * 128;
                    if (v < nvec) {
                        const uint32_t r     = v / vpr;
                        const uint32_t c     = v - r * vpr;
                        const int64_t  row   = static_cast<int64_t>(mt) * BM + r;
                        const int64_t  batch = row / p.s_local;
                        const int64_t  s     = row - batch * p.s_local;
                        val[k] = ptx::ld_v4(src + (batch * p.s_total + p.seq_off + s) * src_pitch + (c << 4));
                        to[k]  = dst + row * dst_pitch + (c << 4);
                    }
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (v0 + k * 128 < nvec) {
                        ptx::st_v4(to[k], val[k]);
                    }
                }
            }
            __threadfence();
            aux_barrier();
            if (tid == 0) {
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p.ready + mt * peers.world + peer), "r"(1u)
                             : "memory");
            }
        }
        // Closing: "I have finished reading everybody's output", so that the owners may overwrite
        // it; the last CTA also waits for the same word from all peers before the kernel ends.
        aux_barrier();
        if (tid == 0) {
            ticket = atomicAdd(&peers.own->arrive[0], 1u);
        }
        aux_barrier();
        if (ticket == gridDim.x - 1 && aux_warp == 0) {
            if (p.handshake) {
                ptx::fence_sys();
                hs_announce(peers, base + 2);
                hs_await(peers, base + 2, FU_ST_CLOSE_TIMEOUT);
            }
            if (lane == 0) {
                peers.own->arrive[0] = 0;
                __threadfence();
                *reinterpret_cast<volatile uint64_t*>(&peers.own->epoch) = base + 2;
            }
        }
    }
};

// The projection's epilogue: bias and residual. A lane is a row.
struct PullEpi {
    __nv_bfloat16*       c;
    const __nv_bfloat16* residual;
    const void*          bias;
    int64_t              ldc;
    int                  M, N, bias_bf16;

    __device__ void open(int) {}
    __device__ void close(int) {}

    __device__ void tile(uint32_t tmem_acc, int mt, int nt, int quarter, int lane)
    {
        const int  row    = mt * BM + quarter * 32 + lane;
        const bool row_ok = row < M;
#pragma unroll 1
        for (int chunk = 0; chunk < BN / 32; ++chunk) {
            const int col0 = nt * BN + chunk * 32;
            if (col0 >= N) {
                break;  // warp-uniform
            }
            uint32_t r[32];
            ptx::tmem_ld_32x32(tmem_acc + chunk * 32, r);
            ptx::tmem_ld_wait();
            if (!row_ok) {
                continue;
            }
            __nv_bfloat16*       dst = c + static_cast<int64_t>(row) * ldc + col0;
            const __nv_bfloat16* res = residual ? residual + static_cast<int64_t>(row) * ldc + col0 : nullptr;
#pragma unroll
            for (int g8 = 0; g8 < 4; ++g8) {
                float v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    v[j] = __uint_as_float(r[g8 * 8 + j]);
                    if (bias && col0 + g8 * 8 + j < N) {
                        v[j] += bias_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(bias)[col0 + g8 * 8 + j])
                                          : static_cast<const float*>(bias)[col0 + g8 * 8 + j];
                    }
                }
                if (col0 + g8 * 8 + 8 <= N) {
                    if (res) {
                        const uint4 rv = *reinterpret_cast<const uint4*>(res + g8 * 8);
                        const __nv_bfloat162* rp = reinterpret_cast<const __nv_bfloat162*>(&rv);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float2 f = __bfloat1622float2(rp[j]);
                            v[2 * j] += f.x;
                            v[2 * j + 1] += f.y;
                        }
                    }
                    *reinterpret_cast<uint4*>(dst + g8 * 8) =
                        make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
                }
                else {
                    for (int j = 0; j < 8; ++j) {
                        if (col0 + g8 * 8 + j < N) {
                            dst[g8 * 8 + j] = __float2bfloat16(v[j] + (res ? __bfloat162float(res[g8 * 8 + j]) : 0.0f));
                        }
                    }
                }
            }
        }
    }
};

struct PullArgs {
    Core       core;
    PullEpi    epi;
    PullParams pull;
};

__global__ void __launch_bounds__(THREADS + 128, 1) pull_outproj_kernel(const __grid_constant__ PullArgs a)
{
    PullEpi epi = a.epi;
    run(a.core, epi, PullSrc(a.pull), PullAux(a.pull));
}

int device_sms()
{
    static std::atomic<int> cached[64] = {};
    int                     dev        = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        return 148;
    }
    if (cached[dev] == 0) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cached[dev] = sms;
    }
    return cached[dev];
}

int launch_grid(int ctas, int tiles)
{
    const int sms = device_sms();
    const int g   = ctas > 0 ? std::min(ctas, sms) : sms;
    return std::max(1, std::min(g, tiles));
}

// How many CTA pairs of the wide kernels the device holds at once (GPCs with an odd number of SMs
// leave one SM without a partner). Asked once per device; all of them have the same shape.
int pair_capacity()
{
    static std::atomic<int> cached[64] = {};
    int                     dev        = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) {
        return 0;
    }
    if (cached[dev] == 0) {
        auto               kernel = gemm_wide_kernel<1, 2, 0>;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim          = dim3(2, 1, 1);
        cfg.blockDim         = dim3(WIDE_THREADS, 1, 1);
        cfg.dynamicSmemBytes = WIDE_SMEM_BYTES;
        cudaLaunchAttribute attr{};
        attr.id               = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs             = &attr;
        cfg.numAttrs          = 1;
        int n                 = 0;
        if (raise_smem_limit(kernel, WIDE_SMEM_BYTES) != FU_OK || cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess
            || n < 1) {
            (void)cudaGetLastError();
            // the kernel carries its cluster shape itself; ask again without naming it
            cfg.attrs    = nullptr;
            cfg.numAttrs = 0;
            n            = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
                (void)cudaGetLastError();
                // Pairs do not wait for one another, so a grid larger than what is resident at once
                // is merely scheduled in turns: assume every SM finds a partner.
                n = device_sms() / 2;
            }
        }
        cached[dev] = n > 0 ? n : -1;
    }
    return std::max(0, cached[dev].load());
}

// Which core and tile a problem gets, from its size alone: the one whose estimated time is lowest. The
// estimate is a start, per wave of CTAs a time per 64-wide K-block, and the epilogue. Fitted to products of 64 - 20000 rows,
// 64 - 13824 columns and K, each timed in up to 24 shapes behind a launch of itself (us, SM clock 1.9 GHz). On 450 others of up to 9000 rows
// the shape chosen takes 0.9 % more than the fastest one (geometric mean; 9 in 10 sizes less than 2 % more, one 30 %), on 200 of
// up to 75600 rows 1.3 % (5.3 %, 25 %). With the epilogue's time left out it was 5.4 % once, with half of it for two blocks and launches of
// nothing but halves of tiles 4.4 %. Small tiles and narrow blocks on few SMs are faster than this says since the producers look ahead.
// All constants fitted again took 0.5 % off most sizes, and put 10 - 26 % on ten of 1500, of 40 - 100 us, which L2 bounds then: left.
//   128 x 128 tiles on single CTAs   2.0 + 0.223 per K-block and wave of 148
//   two 256 x 256 blocks on pairs    2.6 + 0.622 per K-block and wave of 74, and the epilogue of both
//   one 256 x 256 block on pairs     2.6 + 0.328
// Rows of an operand that do not all start on a 32-byte sector (a pitch that is an odd multiple of 16 bytes)
// reach shared memory more slowly, see kSmallBlock and the next two (256 x 3328 x 4096 with small tiles and none, one or two such
// operands: 18.1, 21.3 and 28.6 us). The pair kernels' time per K-block shrinks with the width of the block, see block_clocks(). At
// most half as many tiles of two blocks as pairs left over are split into blocks.
// With one block (and with small tiles) the accumulators alternate and a wave takes the longer of the products and the epilogue with
// what it delays; with two, the second block waits in tensor memory until the first has been written, and the next tile with
// it. Two blocks and one: 6729 x 7632 x 2592 with a residual 205 and 184 us, 14493 x 3408 x 3472 with erf GELU 270 (of 192
// columns) and 246, 7478 x 10512 x 3248 with the derivative 412 and 375. Large products repeated for tenths of a second run at
// the power limit, and there two blocks, which read less from shared memory, win where the estimates are close: 7800 x 5120 x 13824
// with a residual 837 and 892 us, 7800 x 5120 x 5120 331 and 336, 7800 x 13824 x 5120 with GELU 854 and 860, with the derivative 912
// and 911; with one operand off the sectors 13645 x 5672 -> 2336 with GELU and a residual, both products, 630 and 672, with three of
// four 15717 x 6472 -> 3688 1320 and 1468. So beyond kLong (us) another shape has to be estimated 8 % faster than two whole
// blocks, 12 % with an operand off the sectors.
// A launch of nothing but halves of tiles of two blocks does what a launch of single blocks does, with a shorter ring: it is
// left out (143 x 10928 x 12416 76 -> 65 us, 4105 x 288 x 9032 with erf GELU 50.5 -> 48).
// What the widths and the single block gave, against two blocks of 256 columns or the small tiles: 1000 x 5120 x
// 5120 53.0 -> 41.8 us (two of 160), 512 x 5120 x 13824 81.6 -> 61.6 and 512 x 5120 x 5120 30.4 -> 25.8 (one of
// 160), 4100 x 1536 x 4096 58.9 -> 47.2 (two of 192).
enum class Shape { kSmall, kTall, kBroad, kOne };  // 128 x 128; 512 x width; 256 x 2 width; 256 x width
struct Choice {
    Shape  shape;
    int    tiles_m, tiles_n, full, items;
    double cost;
    int    width = 256;
    int    rest = 0, csize = 1;  // kBroad: blocks beyond `items`, shared by clusters of `csize` CTAs
};

// What bounds a K-block of a pair's tile of mb x nb blocks: the tensor pipe takes width / 2 clocks per MMA; shared
// memory moves 128 bytes a clock, 4 KiB of A and 16 * width bytes of B for each MMA and the operands' own
// 16 KiB per block row and 64 * width bytes per block column once.
double block_clocks(int mb, int nb, int width)
{
    const double tensor = 4.0 * mb * nb * width / 2;
    const double shared = (4.0 * mb * nb * (4096 + 16 * width) + 16384.0 * mb + 64.0 * width * nb) / 128;
    return std::max(tensor, shared);
}

// us per K-block, by how many of the two operands lie off the 32-byte sectors
constexpr double kSmallBlock[3] = {0.223, 0.27, 0.38}, kOneBlock[3] = {0.328, 0.34, 0.42}, kTwoBlocks[3] = {0.622, 0.65, 0.73};
constexpr double kSmallStart = 2.0, kPairStart = 2.6, kLong = 50.0;

// us that the epilogue of a block of 256 columns takes, of a 128 x 128 tile with eight warps and with four, which share it in clusters.
// Up to 16 K-blocks 146 products of 2000 - 75600 rows that small tiles with eight warps win from pairs take 17 % less so than with the
// four warps' figures (6043 x 5432 x 384 with the GELU's derivative 85.8 -> 63.7 us). 112 of them take more than 50 us and were repeated until
// the power limit held, and one takes more than 2 % longer: beyond kLong small tiles need no margin against two whole blocks. With
// more K-blocks the tiles' reads from L2, which are not counted here, make the estimate less sure: a small tile has to be faster than
// pairs by `doubt` of its time from 24 K-blocks on, twice that with an operand off the sectors, in proportion from 16. Of 600
// products beyond 16 K-blocks whose shape is another than with the four warps' figures, 279 take 3 - 24 % less and 77 3 - 14 % more.
// The projection's figures are fitted without.
struct Epilogue {
    double pair, small, shared, doubt;
    // A warp's share of a narrow block is half a unit, or more of it in pieces that are not whole.
    double block(int width) const { return width > 128 ? pair : 0.59 * pair; }
};
// Whether the pre-activation is saved (0.9 more) is left out: a forward pass has the same bits with gradients and without.
Epilogue epilogue_of(int act, bool residual)
{
    const double pair[4] = {2.4, 4.7, 7.3, 7.0}, small[4] = {1.2, 2.2, 4.4, 3.5}, shared[4] = {1.4, 3.2, 6.4, 5.5};
    return {pair[act] + (residual ? 1.7 : 0.0), small[act] + (residual ? 1.0 : 0.0), shared[act] + (residual ? 1.0 : 0.0), 0.04};
}
constexpr Epilogue kQkvEpilogue{7.0, 4.0, 4.0, 0.0};  // fitted to 100 projections of 64 - 75600 rows, 1 - 40 heads: 0.9 % above the fastest shape

// Waves of single blocks: an epilogue runs beside the next products and they delay it.
double alternating(double products, double epilogue, int64_t waves)
{
    return waves < 1 ? 0.0 : products + (waves - 1) * std::max(products, epilogue + 0.46 * products) + epilogue;
}

int off_sectors(const void* a, int64_t lda, const void* b, int64_t ldb)
{
    auto off = [](const void* p, int64_t ld) { return ld % 16 != 0 || (reinterpret_cast<uintptr_t>(p) & 31u) != 0; };
    return (off(a, lda) ? 1 : 0) + (off(b, ldb) ? 1 : 0);
}

Choice wide_choice(int64_t m, int64_t n, double kb, Shape shape, int width, int pairs, int off, Epilogue epi)
{
    const int     mb = shape == Shape::kTall ? 2 : 1, nb = shape == Shape::kBroad ? 2 : 1;
    const int64_t tm = (m + 256 * mb - 1) / (256 * mb), tn = (n + width * nb - 1) / (width * nb), tiles = tm * tn;
    const double  e = epi.block(width), block = kb * kOneBlock[off] / 512 * block_clocks(1, 1, width);
    if (shape == Shape::kOne) {
        return {shape, static_cast<int>(tm), static_cast<int>(tn), static_cast<int>(tiles), static_cast<int>(tiles),
                kPairStart + alternating(block, e, (tiles + pairs - 1) / pairs), width};
    }
    const int64_t left = tiles % pairs, full = 2 * left <= pairs ? tiles - left : tiles, items = full + 2 * (tiles - full);
    const double  whole = static_cast<double>((full + pairs - 1) / pairs);
    return {shape, static_cast<int>(tm), static_cast<int>(tn), static_cast<int>(full), static_cast<int>(items),
            kPairStart + whole * (kb * kTwoBlocks[off] / 1024 * block_clocks(mb, nb, width) + 2.0 * e)
                + alternating(block, e, (items - full + pairs - 1) / pairs), width};
}

// `narrow`: the epilogue takes blocks of any width (the heads of the QKV projection need 128 columns at once).
Choice choose_shape(int64_t m, int64_t n, int64_t k, int pairs, int sms, int flags, bool narrow, int off, Epilogue epi)
{
    const int64_t t128 = ((m + 127) / 128) * ((n + 127) / 128);
    const double  kb   = static_cast<double>((k + BK - 1) / BK);
    const double  products = kSmallBlock[off] * kb, waves = static_cast<double>((t128 + sms - 1) / sms);
    const Choice  small{Shape::kSmall, static_cast<int>((m + 127) / 128), static_cast<int>((n + 127) / 128), 0, static_cast<int>(t128),
                       kSmallStart + products + (waves - 1.0) * std::max(products + 0.35 * epi.small, epi.small) + epi.small};
    if (flags & FU_GEMM_SINGLE) {
        return small;
    }
    const Choice tall = wide_choice(m, n, kb, Shape::kTall, 256, pairs, off, epi), broad = wide_choice(m, n, kb, Shape::kBroad, 256, pairs, off, epi);
    if (flags & FU_GEMM_PAIR) {
        return tall.cost < broad.cost ? tall : broad;
    }
    const auto cheaper = [](const Choice& a, const Choice& b) { return b.cost < a.cost && (b.shape == Shape::kOne || b.full > 0) ? b : a; };
    Choice     two{}, best = wide_choice(m, n, kb, Shape::kOne, 256, pairs, off, epi);
    two.cost = std::numeric_limits<double>::infinity();
    two      = cheaper(cheaper(two, tall), broad);
    for (int width = narrow ? 224 : 0; width >= 96; width -= 32) {
        if ((flags & FU_GEMM_B_KN) && width % 128 != 0) {
            continue;  // such a B comes in blocks of 64 columns, half of them for each CTA
        }
        for (const Shape shape : {Shape::kTall, Shape::kBroad, Shape::kOne}) {
            best = cheaper(best, wide_choice(m, n, kb, shape, width, pairs, off, epi));
        }
    }
    if (best.cost >= (two.cost <= kLong ? 1.0 : off > 0 ? 0.88 : 0.92) * two.cost) {
        best = two;
    }
    const double doubt = (off > 0 ? 2.0 : 1.0) * epi.doubt * std::min(1.0, std::max(0.0, kb - 16.0) / 8.0);
    return small.cost * (1.0 + doubt) < best.cost ? small : best;
}

// The broad tiles with what whole waves leave over shared by clusters (gemm_wide_split_kernel), when that is
// estimated to be faster than `best`. Fitted with the others (us): a wave of clusters takes 7.0 (two pairs) or 7.3 (four), 0.32
// per K-block of a pair's share and 0.43 of an epilogue; behind another launch 1.5 of that are hidden. 2000 x 5120 x 5120 (80 tiles
// on 74 pairs): 83.5 -> 79.5, 1000 x 5120 x 13824 (40 tiles: a wave of blocks and six more): 130 -> 115.
Choice choose_wide_split(const Choice& best, int64_t m, int64_t n, int64_t k, int pairs, int off, Epilogue epi)
{
    static fu::ClusterCapacity capacity;
    const int64_t              kb = (k + BK - 1) / BK;
    Choice                     chosen = best;
    const Choice               broad  = wide_choice(m, n, static_cast<double>(kb), Shape::kBroad, 256, pairs, off, epi);
    const int64_t              tiles = static_cast<int64_t>(broad.tiles_m) * broad.tiles_n, full = tiles / pairs * pairs;
    const int64_t              blocks = 2 * (tiles - full), single = blocks / pairs * pairs, rest = blocks - single;
    int                        dev = 0;
    if (rest == 0 || cudaGetDevice(&dev) != cudaSuccess) {
        return best;
    }
    double       limit = 0.96 * best.cost;
    const double before = full + single > 0 ? kPairStart - 1.5 + (kb * kTwoBlocks[off] + 2.0 * epi.pair) * (full / pairs)
                                                  + alternating(kb * kOneBlock[off], epi.pair, single / pairs)
                                            : 0.0;
    for (const int csize : {4, 8}) {
        const int64_t parts = csize / 2, share = (kb + parts - 1) / parts;
        const double  wave  = (csize == 4 ? 7.0 : 7.3) + 0.97 * kOneBlock[off] * share + 0.43 * epi.pair;
        if ((kb + share - 1) / share != parts || before + wave >= limit) {
            continue;  // a pair would have nothing to do, or no gain beyond the estimate's error even in one wave
        }
        const int cap = capacity.of(gemm_wide_split_kernel<0>, csize, dev, WIDE_THREADS, WIDE_SMEM_BYTES);
        if (cap < 1) {
            continue;
        }
        const double cost = before + static_cast<double>((rest + cap - 1) / cap) * wave;
        if (cost < limit) {
            limit        = cost;
            chosen       = broad;
            chosen.full  = static_cast<int>(full);
            chosen.items = static_cast<int>(full + single);
            chosen.cost  = cost;
            chosen.rest  = static_cast<int>(rest);
            chosen.csize = csize;
        }
    }
    return chosen;
}

// How many CTAs share the K-blocks of a 128 x 128 tile (1: none do), see run_small, when that is estimated
// to be faster than `best`. The exchange takes 2.9, 3.2 and 3.5 us beyond the tile's own time (fitted with the others, for
// two, four and eight CTAs). 64 x 2000 x 8000: 30.6 -> 13.3 us with four, 64 x 512 x 2048: 10.6 -> 7.0 with eight,
// 512 x 1536 x 4096: 18.0 -> 13.2 with two; the 160 tiles of 512 x 5120 x 5120 stay as they are.
int choose_split(const Choice& best, int64_t m, int64_t n, int64_t k, int off, Epilogue epi)
{
    static fu::ClusterCapacity capacity;
    const int64_t              t128 = ((m + 127) / 128) * ((n + 127) / 128), kb = (k + BK - 1) / BK;
    int                        dev = 0, chosen = 1;
    double                     cost = best.cost;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        return 1;
    }
    for (const int csize : {2, 4, 8}) {
        const int64_t share = (kb + csize - 1) / csize;
        const double  once  = kSmallStart + (csize == 2 ? 2.9 : csize == 4 ? 3.2 : 3.5) + kSmallBlock[off] * share + epi.shared / csize;
        if ((kb + share - 1) / share != csize || once >= cost) {
            continue;  // a CTA would have nothing to do, or no gain even in one wave
        }
        const int cap = capacity.of(gemm_split_kernel<0>, csize, dev, small_threads(128), small_smem_bytes(128));
        if (cap < 1) {
            continue;
        }
        const double c = static_cast<double>((t128 + cap - 1) / cap) * once;
        if (c < cost) {
            cost   = c;
            chosen = csize;
        }
    }
    return chosen;
}

int fill_core(Core& core, const void* a, const void* b, int64_t m, int64_t n, int64_t k, int64_t lda, int64_t ldb, uint32_t* err)
{
    if (m <= 0 || n <= 0 || k <= 0) {
        return fu::fail(FU_E_ARG, "gemm: empty problem (m=%lld n=%lld k=%lld)", (long long)m, (long long)n, (long long)k);
    }
    int rc = make_map_2d(&core.map_a, a, 2, m, k, lda, BM, BK);
    if (rc != FU_OK) {
        return rc;
    }
    rc = make_map_2d(&core.map_b, b, 2, n, k, ldb, BN, BK);
    if (rc != FU_OK) {
        return rc;
    }
    core.M       = static_cast<int>(m);
    core.N       = static_cast<int>(n);
    core.K       = static_cast<int>(k);
    core.tiles_m = static_cast<int>((m + BM - 1) / BM);
    core.tiles_n = static_cast<int>((n + BN - 1) / BN);
    core.err     = err;
    return FU_OK;
}

int fill_wide(WideCore& core, const Choice& c, const void* a, const void* b, int64_t m, int64_t n, int64_t k, int64_t lda,
              int64_t ldb, uint32_t* err, int flags)
{
    // K itself may be anything (TMA zero-fills the part of a box that lies past it); what TMA needs
    // is a 16-byte row pitch, which make_map_2d checks on lda and ldb. Every box is 128 rows of one
    // operand (or a 64 x 64 block of one stored with the contraction along its rows).
    core.a_mn = (flags & FU_GEMM_A_KM) ? 1 : 0;
    core.b_mn = (flags & FU_GEMM_B_KN) ? 1 : 0;
    int rc = core.a_mn ? make_map_2d(&core.map_a, a, 2, k, m, lda, 64, 64) : make_map_2d(&core.map_a, a, 2, m, k, lda, 128, BK);
    if (rc != FU_OK) {
        return rc;
    }
    rc = core.b_mn ? make_map_2d(&core.map_b, b, 2, k, n, ldb, 64, 64) : make_map_2d(&core.map_b, b, 2, n, k, ldb, c.shape == Shape::kSmall ? 128 : c.width / 2, BK);
    if (rc != FU_OK) {
        return rc;
    }
    core.M       = static_cast<int>(m);
    core.N       = static_cast<int>(n);
    core.K       = static_cast<int>(k);
    core.tiles_m = c.tiles_m;
    core.tiles_n = c.tiles_n;
    core.full    = c.full;
    core.items   = c.items;
    core.width   = c.width;
    core.err     = err;
    return FU_OK;
}

int check_extents(int64_t m, int64_t n, int64_t k)
{
    if (m <= 0 || n <= 0 || k <= 0 || m > 0x7fffff00 || n > 0x7fffff00 || k > 0x7fffff00) {
        return fu::fail(FU_E_ARG, "gemm: empty problem or one too large (m=%lld n=%lld k=%lld)", (long long)m, (long long)n,
                        (long long)k);
    }
    return FU_OK;
}

// How many pairs a launch may use (`ctas` > 0 limits it), or 0 with the error set.
int pairs_for(int ctas)
{
    const int pairs = pair_capacity();
    if (pairs < 1) {
        fu::fail(FU_E_CUDA, "this device cannot hold a cluster of two CTAs of the pair kernels");
        return 0;
    }
    return ctas > 0 ? std::max(1, std::min(pairs, ctas / 2)) : pairs;
}

template <class Args>
cudaError_t launch(void (*kernel)(Args), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const Args& a)
{
    if (a.core.overlap) {
        return fu::launch_behind(kernel, grid, block, smem, stream, a);
    }
    kernel<<<grid, block, smem, stream>>>(a);
    return cudaGetLastError();
}

template <class Args>
int launch_pairs(void (*kernel)(Args), const Args& a, int pairs, cudaStream_t stream)
{
    const int rc = raise_smem_limit(kernel, WIDE_SMEM_BYTES);
    if (rc != FU_OK) {
        return rc;
    }
    FU_CUDA_OK(launch(kernel, dim3(static_cast<unsigned>(2 * std::max(1, std::min(pairs, a.core.items)))), dim3(WIDE_THREADS), WIDE_SMEM_BYTES, stream, a));
    return FU_OK;
}

template <class Args>
int launch_small(void (*kernel)(Args), const Args& a, int cols, int ctas, cudaStream_t stream)
{
    const int rc = raise_smem_limit(kernel, small_smem_bytes(cols));
    if (rc != FU_OK) {
        return rc;
    }
    FU_CUDA_OK(launch(kernel, dim3(static_cast<unsigned>(launch_grid(ctas, a.core.items))), dim3(static_cast<unsigned>(small_threads(cols))), static_cast<size_t>(small_smem_bytes(cols)), stream, a));
    return FU_OK;
}

template <int ACT>
int launch_clusters(void (*kernel)(PlainArgs<ACT>), const PlainArgs<ACT>& a, int clusters, int csize, int threads, int smem,
                    cudaStream_t stream)
{
    const int rc = raise_smem_limit(kernel, smem);
    if (rc != FU_OK) {
        return rc;
    }
    cudaLaunchConfig_t  cfg  = {};
    cudaLaunchAttribute attr = fu::cluster_attr(csize);
    cfg.gridDim              = dim3(static_cast<unsigned>(clusters * csize), 1, 1);
    cfg.blockDim             = dim3(static_cast<unsigned>(threads), 1, 1);
    cfg.dynamicSmemBytes     = static_cast<size_t>(smem);
    cfg.stream               = stream;
    cfg.attrs                = &attr;
    cfg.numAttrs             = 1;
    FU_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, a));
    return FU_OK;
}

template <int ACT>
int launch_plain(const FuGemmArgs* g, Choice c, int pairs, int flags, cudaStream_t stream)
{
    PlainArgs<ACT> a{};
    const int      off = off_sectors(g->a, g->lda, g->b, g->ldb);
    const Epilogue epi = epilogue_of(g->act, g->residual != nullptr);
    int            csize = 1;
    if (g->ctas <= 0 && !(flags & (FU_GEMM_SINGLE | FU_GEMM_PAIR))) {
        c     = choose_wide_split(c, g->m, g->n, g->k, pairs, off, epi);
        csize = choose_split(c, g->m, g->n, g->k, off, epi);
    }
    if (csize > 1) {
        c = choose_shape(g->m, g->n, g->k, pairs, 1, FU_GEMM_SINGLE, false, off, epi);
    }
    const int      rc = fill_wide(a.core, c, g->a, g->b, g->m, g->n, g->k, g->lda, g->ldb, g->err, flags);
    if (rc != FU_OK) {
        return rc;
    }
    a.core.overlap  = g->ctas <= 0;
    a.epi.c         = static_cast<__nv_bfloat16*>(g->c);
    a.epi.residual  = static_cast<const __nv_bfloat16*>(g->residual);
    a.epi.bias      = g->bias;
    a.epi.bias_bf16 = (flags & FU_GEMM_BIAS_BF16) ? 1 : 0;
    a.epi.ldc       = g->ldc;
    a.epi.M         = a.core.M;
    a.epi.N         = a.core.N;
    a.epi.aux       = static_cast<const __nv_bfloat16*>(g->aux);
    a.epi.c_pre     = static_cast<__nv_bfloat16*>(g->c_pre);
    if (csize > 1) {
        return launch_clusters<ACT>(gemm_split_kernel<ACT>, a, a.core.items, csize, small_threads(128), small_smem_bytes(128), stream);
    }
    if (c.rest > 0) {
        a.core.first = c.items;
        const int rc = c.items > 0 ? launch_pairs(gemm_wide_kernel<1, 2, ACT>, a, pairs, stream) : FU_OK;
        return rc != FU_OK ? rc
                           : launch_clusters<ACT>(gemm_wide_split_kernel<ACT>, a, c.rest, c.csize, WIDE_THREADS, WIDE_SMEM_BYTES, stream);
    }
    switch (c.shape) {
    case Shape::kTall: return launch_pairs(gemm_wide_kernel<2, 1, ACT>, a, pairs, stream);
    case Shape::kBroad: return launch_pairs(gemm_wide_kernel<1, 2, ACT>, a, pairs, stream);
    case Shape::kOne: return launch_pairs(gemm_wide_kernel<1, 1, ACT>, a, pairs, stream);
    default: return launch_small(gemm_small_kernel<ACT>, a, 64, g->ctas, stream);
    }
}

}  // namespace

extern "C" int fu_gemm_bf16(const FuGemmArgs* g, void* stream_v)
{
    if (!g || !g->a || !g->b || !g->c) {
        return fu::fail(FU_E_ARG, "fu_gemm_bf16: null operand");
    }
    if ((g->ldc % 8) || (reinterpret_cast<uintptr_t>(g->c) & 15u)
        || (g->residual && (reinterpret_cast<uintptr_t>(g->residual) & 15u))) {
        return fu::fail(FU_E_ARG, "fu_gemm_bf16: C (and the residual) need 16-byte aligned rows");
    }
    if (g->act < 0 || g->act > 3 || (g->act == 3 && !g->aux)) {
        return fu::fail(FU_E_ARG, "fu_gemm_bf16: act=%d (0..3; 3 needs aux)", g->act);
    }
    if ((g->aux || g->c_pre) && ((g->n % 8) || (reinterpret_cast<uintptr_t>(g->aux) & 15u)
                                 || (reinterpret_cast<uintptr_t>(g->c_pre) & 15u))) {
        return fu::fail(FU_E_ARG, "fu_gemm_bf16: aux / c_pre need n %% 8 == 0 and 16-byte aligned rows");
    }
    int rc = check_extents(g->m, g->n, g->k);
    if (rc != FU_OK) {
        return rc;
    }
    // The shape is chosen by size unless the call (FU_GEMM_PAIR / FU_GEMM_SINGLE) or, for calls that say
    // nothing, the environment variable FU_GEMM_PAIR (read once) asks for pairs.
    static const bool pair_default = [] {
        const char* e = std::getenv("FU_GEMM_PAIR");
        return e && e[0] == '1';
    }();
    const int pairs = pairs_for(g->ctas);
    if (pairs < 1) {
        return FU_E_CUDA;
    }
    const bool   forced = pair_default && !(g->flags & FU_GEMM_SINGLE);
    const int    flags  = forced ? (g->flags | FU_GEMM_PAIR) : g->flags;
    const int    sms    = g->ctas > 0 ? std::min(g->ctas, device_sms()) : device_sms();
    const Choice c      = choose_shape(g->m, g->n, g->k, pairs, sms, flags, true, off_sectors(g->a, g->lda, g->b, g->ldb),
                                      epilogue_of(g->act, g->residual != nullptr));
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    switch (g->act) {
    case 0: return launch_plain<0>(g, c, pairs, flags, stream);
    case 1: return launch_plain<1>(g, c, pairs, flags, stream);
    case 2: return launch_plain<2>(g, c, pairs, flags, stream);
    default: return launch_plain<3>(g, c, pairs, flags, stream);
    }
}

extern "C" int fu_qkv_rope_scatter_check(const FuQkvArgs* q)
{
    if (!q || !q->x || !q->w) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: null operand");
    }
    const int n_types  = q->n_types > 0 ? q->n_types : 3;
    const int n_normed = q->n_types > 0 ? q->n_normed : 2;
    if (n_types > 3 || n_normed > 2 || n_normed > n_types) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: %d projections, %d normed", n_types, n_normed);
    }
    if (n_normed > 0 && (!q->rope || !q->gamma_q || (n_normed > 1 && !q->gamma_k))) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: RMSNorm + RoPE need rope and gamma tables");
    }
    if (q->world < 1 || q->world > FU_MAX_WORLD || q->rank < 0 || q->rank >= q->world) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: rank %d / world %d", q->rank, q->world);
    }
    if (q->heads < 1 || q->heads > MAX_HEADS) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: heads=%d (need 1..%d)", q->heads, MAX_HEADS);
    }
    if (q->s_local <= 0 || q->m % q->s_local) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: m=%lld is not a multiple of s_local=%lld", (long long)q->m,
                        (long long)q->s_local);
    }
    int heads_seen = 0;
    for (int p = 0; p < q->world; ++p) {
        if (q->head_splits[p] < 0 || q->head_splits[p] > 255) {
            return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: head_splits[%d]=%d", p, q->head_splits[p]);
        }
        heads_seen += q->head_splits[p];
        if (!q->win_q[p] || (n_types > 1 && !q->win_k[p]) || (n_types > 2 && !q->win_v[p]) || !q->peer_ctrl[p]) {
            return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: no window for rank %d", p);
        }
    }
    if (heads_seen != q->heads) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: head_splits sum to %d, expected %d", heads_seen, q->heads);
    }
    // The epilogue stores row (batch, seq_off + s) of head `local` of rank p at
    // ((batch * s_total + seq_off + s) * head_splits[p] + local) * 256 bytes behind that rank's base.
    if (q->seq_off < 0 || q->s_total <= 0 || q->seq_off + q->s_local > q->s_total) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: rows %lld..%lld do not lie inside a sequence of %lld",
                        (long long)q->seq_off, (long long)(q->seq_off + q->s_local), (long long)q->s_total);
    }
    const int64_t batches = q->m / q->s_local;
    for (int p = 0; p < q->world; ++p) {
        const int64_t last = ((batches - 1) * q->s_total + q->seq_off + q->s_local) * q->head_splits[p] * 256;
        if (q->head_splits[p] > 0 && last > q->win_bytes) {
            return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: the stores to rank %d reach byte %lld of windows of %lld bytes",
                            p, (long long)last, (long long)q->win_bytes);
        }
    }
    return FU_OK;
}

extern "C" int fu_qkv_rope_scatter(const FuQkvArgs* q, void* stream_v)
{
    int rc = fu_qkv_rope_scatter_check(q);
    if (rc != FU_OK) {
        return rc;
    }
    const int n_types  = q->n_types > 0 ? q->n_types : 3;
    const int n_normed = q->n_types > 0 ? q->n_normed : 2;
    QkvArgs       a{};
    const int64_t n = static_cast<int64_t>(n_types) * q->heads * HEAD_DIM;
    rc              = check_extents(q->m, n, q->k);
    if (rc != FU_OK) {
        return rc;
    }
    const int pairs = pairs_for(q->ctas);
    if (pairs < 1) {
        return FU_E_CUDA;
    }
    const int    sms   = q->ctas > 0 ? std::min(q->ctas, device_sms()) : device_sms();
    const int    flags = (q->flags & FU_QKV_W_KN) ? FU_GEMM_B_KN : 0;
    const Choice c     = choose_shape(q->m, n, q->k, pairs, sms, flags, false, off_sectors(q->x, q->ldx, q->w, q->ldw), kQkvEpilogue);
    rc = fill_wide(a.core, c, q->x, q->w, q->m, n, q->k, q->ldx, q->ldw, q->err, flags);
    if (rc != FU_OK) {
        return rc;
    }
    QkvParams& e = a.epi;
    int     h = 0;
    for (int p = 0; p < q->world; ++p) {
        if (q->head_splits[p] < 0 || q->head_splits[p] > 255) {
            return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: head_splits[%d]=%d", p, q->head_splits[p]);
        }
        e.heads_of[p] = static_cast<uint8_t>(q->head_splits[p]);
        for (int i = 0; i < q->head_splits[p]; ++i, ++h) {
            if (h >= MAX_HEADS) {
                return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: too many heads");
            }
            e.owner[h] = static_cast<uint8_t>(p);
            e.local[h] = static_cast<uint8_t>(i);
        }
        if (!q->win_q[p] || (n_types > 1 && !q->win_k[p]) || (n_types > 2 && !q->win_v[p]) || !q->peer_ctrl[p]) {
            return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: no window for rank %d", p);
        }
        e.win[0][p]     = static_cast<uint8_t*>(q->win_q[p]);
        e.win[1][p]     = static_cast<uint8_t*>(q->win_k[p]);
        e.win[2][p]     = static_cast<uint8_t*>(q->win_v[p]);
        e.peers.ctrl[p] = q->peer_ctrl[p];
    }
    if (h != q->heads) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: head_splits sum to %d, expected %d", h, q->heads);
    }
    e.peers.own        = q->peer_ctrl[q->rank];
    e.peers.rank       = q->rank;
    e.peers.world      = q->world;
    e.peers.mute       = (q->flags & FU_A2A_MUTE) ? 1 : 0;
    e.peers.timeout_ns = static_cast<uint64_t>(q->timeout_ms ? q->timeout_ms : 10000) * 1000000ull;
    e.handshake        = (q->flags & FU_A2A_NO_HANDSHAKE) ? 0 : 1;
    e.rope             = reinterpret_cast<const float2*>(q->rope);
    e.gamma_q          = q->gamma_q;
    e.gamma_k          = q->gamma_k;
    e.tables_aligned   = ((reinterpret_cast<uintptr_t>(q->rope) | reinterpret_cast<uintptr_t>(q->gamma_q)
                         | reinterpret_cast<uintptr_t>(q->gamma_k)) & 15u) == 0;
    e.eps              = q->eps;
    e.M                = a.core.M;
    e.heads            = q->heads;
    e.s_local          = q->s_local;
    e.seq_off          = q->seq_off;
    e.s_total          = q->s_total;
    e.n_types          = n_types;
    e.n_normed         = n_normed;
    e.y_save           = static_cast<__nv_bfloat16*>(q->y_save);
    e.ld_y             = q->ld_y;
    if (q->y_save && ((q->ld_y % 8) || (reinterpret_cast<uintptr_t>(q->y_save) & 15u))) {
        return fu::fail(FU_E_ARG, "fu_qkv_rope_scatter: y_save needs 16-byte aligned rows");
    }
    a.core.overlap      = q->world == 1 && q->ctas <= 0;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    switch (c.shape) {
    case Shape::kTall: return launch_pairs(qkv_wide_kernel<2, 1>, a, pairs, stream);
    case Shape::kBroad: return launch_pairs(qkv_wide_kernel<1, 2>, a, pairs, stream);
    case Shape::kOne: return launch_pairs(qkv_wide_kernel<1, 1>, a, pairs, stream);
    default: return launch_small(qkv_small_kernel, a, 128, q->ctas, stream);
    }
}

extern "C" int fu_pull_outproj_check(const FuPullArgs* q)
{
    if (!q || !q->w || !q->c || !q->gather || !q->ready) {
        return fu::fail(FU_E_ARG, "fu_pull_outproj: null operand");
    }
    if (q->world < 1 || q->world > FU_MAX_WORLD || q->rank < 0 || q->rank >= q->world) {
        return fu::fail(FU_E_ARG, "fu_pull_outproj: rank %d / world %d", q->rank, q->world);
    }
    if (q->s_local <= 0 || q->m % q->s_local) {
        return fu::fail(FU_E_ARG, "fu_pull_outproj: m=%lld is not a multiple of s_local=%lld", (long long)q->m,
                        (long long)q->s_local);
    }
    if ((q->ldc % 8) || (reinterpret_cast<uintptr_t>(q->c) & 15u) || (reinterpret_cast<uintptr_t>(q->residual) & 15u)) {
        return fu::fail(FU_E_ARG, "fu_pull_outproj: C and the residual need 16-byte aligned rows");
    }
    int heads_seen = 0;
    for (int p = 0; p < q->world; ++p) {
        if (q->head_splits[p] < 0 || q->head_splits[p] > 255 || !q->peer_o[p] || !q->peer_ctrl[p]) {
            return fu::fail(FU_E_ARG, "fu_pull_outproj: bad shard or missing buffer for rank %d", p);
        }
        heads_seen += q->head_splits[p];
    }
    if (heads_seen < 1 || heads_seen > MAX_HEADS) {
        return fu::fail(FU_E_ARG, "fu_pull_outproj: %d heads (need 1..%d)", heads_seen, MAX_HEADS);
    }
    // The puller warps read row (batch, seq_off + s) of rank p's buffer at
    // ((batch * s_total + seq_off + s) * head_splits[p]) * 256 bytes, head_splits[p] * 256 bytes long.
    if (q->seq_off < 0 || q->s_total <= 0 || q->seq_off + q->s_local > q->s_total) {
        return fu::fail(FU_E_ARG, "fu_pull_outproj: rows %lld..%lld do not lie inside a sequence of %lld",
                        (long long)q->seq_off, (long long)(q->seq_off + q->s_local), (long long)q->s_total);
    }
    const int64_t batches = q->m / q->s_local;
    for (int p = 0; p < q->world; ++p) {
        const int64_t last = ((batches - 1) * q->s_total + q->seq_off + q->s_local) * q->head_splits[p] * 256;
        if (last > q->o_bytes) {
            return fu::fail(FU_E_ARG, "fu_pull_outproj: the loads from rank %d reach byte %lld of buffers of %lld bytes", p,
                            (long long)last, (long long)q->o_bytes);
        }
    }
    if (q->m * heads_seen * 256 > q->gather_bytes) {
        return fu::fail(FU_E_ARG, "fu_pull_outproj: the gathered operand needs %lld bytes, `gather` holds %lld",
                        (long long)(q->m * heads_seen * 256), (long long)q->gather_bytes);
    }
    if (((q->m + BM - 1) / BM) * q->world > q->ready_words) {
        return fu::fail(FU_E_ARG, "fu_pull_outproj: %lld flags needed, `ready` holds %lld",
                        (long long)(((q->m + BM - 1) / BM) * q->world), (long long)q->ready_words);
    }
    return FU_OK;
}

extern "C" int fu_pull_outproj(const FuPullArgs* q, void* stream_v)
{
    int rc = fu_pull_outproj_check(q);
    if (rc != FU_OK) {
        return rc;
    }
    PullArgs a{};
    PullParams& e = a.pull;
    int heads = 0;
    for (int p = 0; p < q->world; ++p) {
        if (q->head_splits[p] < 0 || q->head_splits[p] > 255 || !q->peer_o[p] || !q->peer_ctrl[p]) {
            return fu::fail(FU_E_ARG, "fu_pull_outproj: bad shard or missing buffer for rank %d", p);
        }
        e.heads_of[p]   = static_cast<uint8_t>(q->head_splits[p]);
        e.head_start[p] = static_cast<uint16_t>(heads);
        for (int i = 0; i < q->head_splits[p]; ++i, ++heads) {
            if (heads >= MAX_HEADS) {
                return fu::fail(FU_E_ARG, "fu_pull_outproj: too many heads");
            }
            e.owner[heads] = static_cast<uint8_t>(p);
        }
        e.peer_o[p]     = static_cast<const uint8_t*>(q->peer_o[p]);
        e.peers.ctrl[p] = q->peer_ctrl[p];
    }
    const int64_t k = static_cast<int64_t>(heads) * HEAD_DIM;
    rc = fill_core(a.core, q->gather, q->w, q->m, q->n, k, k, q->ldw, q->err);
    if (rc != FU_OK) {
        return rc;
    }
    e.peers.own        = q->peer_ctrl[q->rank];
    e.peers.rank       = q->rank;
    e.peers.world      = q->world;
    e.peers.mute       = (q->flags & FU_A2A_MUTE) ? 1 : 0;
    e.peers.timeout_ns = static_cast<uint64_t>(q->timeout_ms ? q->timeout_ms : 10000) * 1000000ull;
    e.handshake        = (q->flags & FU_A2A_NO_HANDSHAKE) ? 0 : 1;
    e.gather           = static_cast<uint8_t*>(q->gather);
    e.ready            = q->ready;
    e.M                = a.core.M;
    e.tiles_m          = a.core.tiles_m;
    e.heads_total      = heads;
    e.s_local          = q->s_local;
    e.seq_off          = q->seq_off;
    e.s_total          = q->s_total;
    e.err              = q->err;
    a.epi.c            = static_cast<__nv_bfloat16*>(q->c);
    a.epi.residual     = static_cast<const __nv_bfloat16*>(q->residual);
    a.epi.bias         = q->bias;
    a.epi.bias_bf16    = (q->flags & FU_PULL_BIAS_BF16) ? 1 : 0;
    a.epi.ldc          = q->ldc;
    a.epi.M            = a.core.M;
    a.epi.N            = a.core.N;
    rc                 = raise_smem_limit(pull_outproj_kernel, SMEM_BYTES);
    if (rc != FU_OK) {
        return rc;
    }
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    FU_CUDA_OK(cudaMemsetAsync(q->ready, 0, sizeof(uint32_t) * a.core.tiles_m * q->world, stream));
    // One CTA per SM and never more than the SM count: CTAs wait on flags other CTAs publish.
    const int grid = launch_grid(q->ctas, 1 << 30);
    pull_outproj_kernel<<<grid, THREADS + 128, SMEM_BYTES, stream>>>(a);
    FU_CUDA_OK(cudaGetLastError());
    return FU_OK;
}
