// Memory-bound companions of the fused GEMMs.
//
//   fu_qk_norm_rope_bwd   backward of "per-head RMSNorm -> RoPE" for q and k in one pass: takes the
//                         gradients that came back from the head owners, the pre-norm projections
//                         saved by the forward kernel, and writes the gradient of the projection
//                         output (ready to be the A operand of the dgrad/wgrad GEMMs) plus the
//                         gradients of the two norm weights.
//   fu_pull_qkv_grads     the same pass fused with the exchange that brings dq, dk and dv home
//                         (mode 1 of the all-to-all): every head-row is loaded straight from the
//                         rank that owns the head, over NVLink, transformed on the way (q, k) or
//                         passed through (v), and stored where the dgrad/wgrad GEMMs read it. One
//                         launch replaces the stand-alone exchange, this kernel's local form and a
//                         slice copy; the handshakes are those of every kernel that touches peers.
#include "fu_kernels.h"
#include "handshake.cuh"
#include "host_util.h"
#include "ptx.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <initializer_list>

namespace {

struct NormRopeBwd {
    const __nv_bfloat16* g[2];      // dq, dk: (m, heads, 128) dense
    const __nv_bfloat16* y;         // (m, 2 * heads * 128) pre-norm projections, leading dim ld_y
    __nv_bfloat16*       dy;        // (m, ...) output, leading dim ld_dy; q at column 0, k at heads * 128
    const float2*        rope;      // (s_local, 64)
    const float*         gamma[2];
    float*               dgamma[2];
    int64_t              ld_y, ld_dy;
    int64_t              m, s_local;
    int                  heads;
    float                eps;
};

// Both kernels below give a row of 128 values (one head of one token) to eight lanes, 16 values each:
// four rows per warp and instruction, three shuffles per reduction.
struct RowPart {
    uint2 w[4];  // 16 bf16 values
};
__device__ __forceinline__ RowPart load_part(const void* p)
{
    RowPart r;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        asm volatile("ld.global.v2.u32 {%0, %1}, [%2];"
                     : "=r"(r.w[k].x), "=r"(r.w[k].y)
                     : "l"(static_cast<const uint8_t*>(p) + k * 64));
    }
    return r;
}
__device__ __forceinline__ void store_part(void* p, const RowPart& r)
{
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        *reinterpret_cast<uint2*>(static_cast<uint8_t*>(p) + k * 64) = r.w[k];
    }
}
// Value k of lane `part` is element (k / 4) * 32 + part * 4 + k % 4 of its row (eight lanes move 64
// contiguous bytes per instruction and an 8-byte alignment is enough).
constexpr int kPartStride = 32;

__device__ __forceinline__ float sum_of_row(float v)
{
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, off);
    }
    return v;
}

// d(projection) of one row from the gradient behind RMSNorm -> RoPE; accumulates d(gamma) into dg.
__device__ __forceinline__ RowPart norm_rope_bwd(const RowPart& g, const RowPart& y, const float* rope, const float* gamma, float eps,
                                                 int part, float (&dg)[16])
{
    float yy[16], dx[16], ss = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 cs = *reinterpret_cast<const float4*>(rope + k * kPartStride + part * 4);  // (c0, s0, c1, s1)
        const float2 g0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g.w[k].x));
        const float2 g1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g.w[k].y));
        const float2 y0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&y.w[k].x));
        const float2 y1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&y.w[k].y));
        // undo the rotation: the transpose of a rotation is the opposite rotation
        dx[4 * k]     = g0.x * cs.x + g0.y * cs.y;
        dx[4 * k + 1] = -g0.x * cs.y + g0.y * cs.x;
        dx[4 * k + 2] = g1.x * cs.z + g1.y * cs.w;
        dx[4 * k + 3] = -g1.x * cs.w + g1.y * cs.z;
        yy[4 * k] = y0.x, yy[4 * k + 1] = y0.y, yy[4 * k + 2] = y1.x, yy[4 * k + 3] = y1.y;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            ss += yy[4 * k + i] * yy[4 * k + i];
        }
    }
    const float rstd = rsqrtf(sum_of_row(ss) * (1.0f / 128.0f) + eps);
    float       dot  = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 gm     = *reinterpret_cast<const float4*>(gamma + k * kPartStride + part * 4);
        const float  gmv[4] = {gm.x, gm.y, gm.z, gm.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int   e = 4 * k + i;
            const float n = yy[e] * rstd;
            dg[e] += dx[e] * n;
            dx[e] *= gmv[i];
            dot += dx[e] * n;
            yy[e] = n;
        }
    }
    dot = sum_of_row(dot) * (1.0f / 128.0f);
    RowPart out;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            o[i] = rstd * (dx[4 * k + i] - yy[4 * k + i] * dot);
        }
        out.w[k].x = fu::ptx::pack_bf16x2(o[0], o[1]);
        out.w[k].y = fu::ptx::pack_bf16x2(o[2], o[3]);
    }
    return out;
}

// Adds a CTA's d(gamma) to the result: the lanes that hold the same elements by shuffle, the warps through
// shared memory, one atomic per element and CTA. (All threads of the CTA.)
__device__ __forceinline__ void add_dgamma(float (&dg)[16], float* dgamma, float (*red)[128])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        dg[e] += __shfl_xor_sync(0xffffffffu, dg[e], 8);
        dg[e] += __shfl_xor_sync(0xffffffffu, dg[e], 16);
    }
    __syncthreads();
    if (lane < 8) {
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            red[warp][(e >> 2) * kPartStride + lane * 4 + (e & 3)] = dg[e];
        }
    }
    __syncthreads();
    if (dgamma && threadIdx.x < 128) {
        float s = 0.0f;
        for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) {
            s += red[w][threadIdx.x];
        }
        atomicAdd(dgamma + threadIdx.x, s);
    }
}

__global__ void __launch_bounds__(256) qk_norm_rope_bwd_kernel(const NormRopeBwd p)
{
    __shared__ float red[8][128];
    const int        sub    = (threadIdx.x >> 3) & 3, part = threadIdx.x & 7;
    const int64_t    warp0  = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t    nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    const int64_t    items  = p.m * p.heads;  // per projection
    for (int t = 0; t < 2; ++t) {
        float dg[16] = {};
        for (int64_t it0 = warp0 * 4; it0 < items; it0 += nwarps * 4) {
            const bool    here = it0 + sub < items;  // the warp stays together for the reductions
            const int64_t it   = here ? it0 + sub : items - 1;
            const int64_t row  = it / p.heads;
            const int64_t head = it - row * p.heads;
            const RowPart g    = load_part(p.g[t] + it * 128 + part * 4);
            const RowPart y    = load_part(p.y + row * p.ld_y + (t * p.heads + head) * 128 + part * 4);
            float         own[16] = {};
            const RowPart out  = norm_rope_bwd(g, y, reinterpret_cast<const float*>(p.rope + (row % p.s_local) * 64), p.gamma[t],
                                               p.eps, part, own);
            if (here) {
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    dg[e] += own[e];
                }
                store_part(p.dy + row * p.ld_dy + (t * p.heads + head) * 128 + part * 4, out);
            }
        }
        add_dgamma(dg, p.dgamma[t], red);
    }
}

// ---- LayerNorm without affine parameters ----------------------------------------------------------------
// A row is read once and stays in the registers of 1, 2, 4 or 8 warps, up to kRowUnits 16-byte units a lane, all of them on
// their way at once; statistics in fp32. Bound by HBM, and where L2 holds the matrix by what a CTA does before its first load: how many
// warps a row has is known when the kernel is compiled. With the number passed to the kernel, its divisions and the addresses they hold
// up took forward 75600 x 5120 (1.55 GB) from 230 us to 292, x 1536 from 70 to 87, 9450 x 1024 from 5.5 to 6.5; one warp for every row,
// which read it twice in a chain of short loops, took 342, 73 and 6.1. The backward that adds a gradient to rows of a matrix that L2 does
// not hold walks through them twice with the same warps and a third of the registers, so with three times the rows under way (its
// second pass finds the row in L1): 75600 x 5120 (3.1 GB) 488 us, in registers 576, one warp for every row 720. Without a gradient to add
// registers are faster (402 and 412, 574), and where L2 holds all of it (4000 x 2560 12.2 and 14.5, 20.9). Rows too long for the
// registers of eight warps are walked through twice as well: 2000 x 16384 54 -> 25 and 122 -> 51.
constexpr int kRowUnits = 5;

__device__ __forceinline__ float2 sum_of_warp(float2 v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
    }
    return v;
}

// The sums over the WARPS warps of a row, in their order. (All threads of the CTA.)
template <int WARPS>
__device__ __forceinline__ float2 sum_of_warps(float2 v)
{
    v = sum_of_warp(v);
    if (WARPS > 1) {
        __shared__ float2 part[8];
        const int         warp = threadIdx.x >> 5, first = warp & ~(WARPS - 1);
        if ((threadIdx.x & 31) == 0) {
            part[warp] = v;
        }
        __syncthreads();
        v = part[first];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) {
            v.x += part[first + w].x;
            v.y += part[first + w].y;
        }
    }
    return v;
}

// Where a thread works: its row and its first column of every `stride` columns.
template <int WARPS>
struct RowPlace {
    static constexpr int stride = 256 * WARPS;
    int64_t              row;
    int                  col;
    bool                 leads;
    __device__ __forceinline__ RowPlace()
        : row(static_cast<int64_t>(blockIdx.x) * (8 / WARPS) + (threadIdx.x >> 5) / WARPS), col((threadIdx.x & (32 * WARPS - 1)) * 8),
          leads(col == 0)
    {
    }
};

// The loaded values, not what was made of them for the sums, wait for the row's sums. It costs their conversion a second time and pays
// where the registers would keep a CTA away: backward without a gradient to add 75600 x 1024 91.1 -> 74.9 us, x 3584 345 -> 290.
// With five units there is none to gain (75600 x 1280 98.9 -> 105.8), with three only for rows of several warps (x 3072 250 -> 238).
__device__ __forceinline__ void keep_packed(uint4& v)
{
    asm volatile("" : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w));
}
constexpr bool keeps_packed(int warps, int units) { return units == 4 || (units == 3 && warps > 1); }

__device__ __forceinline__ uint4 ld_unit(const __nv_bfloat16* p)
{
    return *reinterpret_cast<const uint4*>(p);
}

__device__ __forceinline__ void add_moments(const uint4& v, float2& sum)
{
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        sum.x += f.x + f.y;
        sum.y += f.x * f.x + f.y * f.y;
    }
}
__device__ __forceinline__ uint4 normalised(const uint4& v, float mean, float rstd)
{
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
    uint32_t              o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        o[j]           = fu::ptx::pack_bf16x2((f.x - mean) * rstd, (f.y - mean) * rstd);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// UNITS: of a lane, 0 for rows of any length. Three units with several warps take 45 registers, which leaves room for five CTAs; with 40
// there are six (75600 x 1288 65.8 -> 64.3 us, 9450 x 2568 16.6 -> 15.8).
template <int WARPS, int UNITS>
__global__ void __launch_bounds__(256, WARPS > 1 && UNITS == 3 ? 6 : 0)
    layernorm_fwd_kernel(const __nv_bfloat16* x, __nv_bfloat16* y, float* stats, int64_t rows, int64_t cols, int64_t ldx, int64_t ldy, float eps)
{
    fu::ptx::grid_wait();
    fu::ptx::grid_trigger();
    const RowPlace<WARPS> at;
    const bool            here = at.row < rows;
    const __nv_bfloat16*  xr   = x + at.row * ldx;
    __nv_bfloat16*        yr   = y + at.row * ldy;
    uint4                 v[UNITS > 0 ? UNITS : 1];
    float2                sum = make_float2(0.0f, 0.0f);
    if (UNITS > 0) {
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int c = at.col + u * at.stride;
            v[u]        = here && c < cols ? fu::ptx::ld_once_v4(xr + c) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            add_moments(v[u], sum);
        }
    }
    else if (here) {
        for (int64_t c = at.col; c < cols; c += at.stride) {
            add_moments(ld_unit(xr + c), sum);
        }
    }
    sum              = sum_of_warps<WARPS>(sum);
    const float mean = sum.x / static_cast<float>(cols);
    const float rstd = rsqrtf(fmaxf(sum.y / static_cast<float>(cols) - mean * mean, 0.f) + eps);
    if (!here) {
        return;
    }
    if (at.leads && stats) {
        stats[2 * at.row]     = mean;
        stats[2 * at.row + 1] = rstd;
    }
    if (UNITS > 0) {
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int c = at.col + u * at.stride;
            if (c < cols) {
                fu::ptx::st_v4(yr + c, normalised(v[u], mean, rstd));
            }
        }
    }
    else {
        for (int64_t c = at.col; c < cols; c += at.stride) {
            fu::ptx::st_v4(yr + c, normalised(ld_unit(xr + c), mean, rstd));
        }
    }
}

__device__ __forceinline__ void add_products(const uint4& xv, const uint4& gv, float mean, float rstd, float2& sum)
{
    const __nv_bfloat162* xh = reinterpret_cast<const __nv_bfloat162*>(&xv);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 xf = __bfloat1622float2(xh[j]), gf = __bfloat1622float2(gh[j]);
        sum.x += gf.x + gf.y;
        sum.y += gf.x * (xf.x - mean) * rstd + gf.y * (xf.y - mean) * rstd;
    }
}
// `mg`, `mgx`: the row's means of the gradient and of its product with the normalised value; `av` is added where `add` says so
__device__ __forceinline__ uint4 norm_gradient(const uint4& xv, const uint4& gv, const uint4& av, bool add, float mean, float rstd, float mg,
                                               float mgx)
{
    const __nv_bfloat162* ah = reinterpret_cast<const __nv_bfloat162*>(&av);
    const __nv_bfloat162* xh = reinterpret_cast<const __nv_bfloat162*>(&xv);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv);
    uint32_t              o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 xf = __bfloat1622float2(xh[j]), gf = __bfloat1622float2(gh[j]);
        float2       d  = make_float2(rstd * (gf.x - mg - (xf.x - mean) * rstd * mgx),
                                      rstd * (gf.y - mg - (xf.y - mean) * rstd * mgx));
        if (add) {
            const float2 af = __bfloat1622float2(ah[j]);
            d.x += af.x;
            d.y += af.y;
        }
        o[j] = fu::ptx::pack_bf16x2(d.x, d.y);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

template <int WARPS, int UNITS>
__global__ void __launch_bounds__(256) layernorm_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* x,
                                                            const float* stats, const __nv_bfloat16* add,
                                                            __nv_bfloat16* dx, int64_t rows, int64_t cols, int64_t ld)
{
    fu::ptx::grid_wait();
    fu::ptx::grid_trigger();
    const RowPlace<WARPS> at;
    const bool            here = at.row < rows;
    const __nv_bfloat16 * xr = x + at.row * ld, *gr = dy + at.row * ld, *ar = add + at.row * ld;
    __nv_bfloat16*        dr   = dx + at.row * ld;
    const float           mean = here ? stats[2 * at.row] : 0.0f, rstd = here ? stats[2 * at.row + 1] : 0.0f;
    const uint4           none = make_uint4(0u, 0u, 0u, 0u);
    constexpr int         N    = UNITS > 0 ? UNITS : 1;
    uint4                 xv[N], gv[N];
    float2                sum = make_float2(0.0f, 0.0f);
    if (UNITS > 0) {
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int c = at.col + u * at.stride;
            xv[u] = gv[u] = none;
            if (here && c < cols) {
                xv[u] = fu::ptx::ld_once_v4(xr + c);
                gv[u] = fu::ptx::ld_once_v4(gr + c);
            }
        }
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            // Beyond the last column, which only the last unit reaches, 0 x (0 - 0): against a mean that has overflowed it would be NaN.
            const bool inside = u + 1 < UNITS || at.col + u * at.stride < cols;
            add_products(xv[u], gv[u], inside ? mean : 0.0f, inside ? rstd : 0.0f, sum);
        }
    }
    else if (here) {
        for (int64_t c = at.col; c < cols; c += at.stride) {
            add_products(ld_unit(xr + c), ld_unit(gr + c), mean, rstd, sum);
        }
    }
    sum            = sum_of_warps<WARPS>(sum);
    if (keeps_packed(WARPS, UNITS)) {
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            keep_packed(xv[u]);
            keep_packed(gv[u]);
        }
    }
    const float mg = sum.x / static_cast<float>(cols), mgx = sum.y / static_cast<float>(cols);
    if (!here) {
        return;
    }
    if (UNITS > 0) {
        uint4 av[N];  // not earlier: its registers would cost rows under way
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int c = at.col + u * at.stride;
            av[u]       = add && c < cols ? fu::ptx::ld_once_v4(ar + c) : none;
        }
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int c = at.col + u * at.stride;
            if (c < cols) {
                fu::ptx::st_v4(dr + c, norm_gradient(xv[u], gv[u], av[u], add != nullptr, mean, rstd, mg, mgx));
            }
        }
    }
    else {
        for (int64_t c = at.col; c < cols; c += at.stride) {
            const uint4 a = add ? ld_unit(ar + c) : none;
            fu::ptx::st_v4(dr + c, norm_gradient(ld_unit(xr + c), ld_unit(gr + c), a, add != nullptr, mean, rstd, mg, mgx));
        }
    }
}

// Values of a matrix beyond which the backward's four (x, dy, the gradient to add, dx) are more than L2 holds.
constexpr int64_t kNormInL2 = 12ll << 20;

// As few warps a row as its units allow, so that little rows need no meeting through shared memory.
struct RowShape {
    int      lg_warps, units;  // units: 0 for rows that no eight warps hold
    unsigned blocks;
    RowShape(int64_t rows, int64_t cols)
    {
        const int64_t pieces = cols / 8;
        for (lg_warps = 0; lg_warps < 3 && pieces > (32 << lg_warps) * kRowUnits;) {
            ++lg_warps;
        }
        const int64_t lanes = 32 << lg_warps, each = (pieces + lanes - 1) / lanes, at_once = 8 >> lg_warps;
        units               = each <= kRowUnits ? static_cast<int>(each) : 0;
        blocks              = static_cast<unsigned>((rows + at_once - 1) / at_once);
    }
};

// By the number of warps and of units; rows of two warps or more have at least three units a lane.
using NormForward  = decltype(&layernorm_fwd_kernel<8, 0>);
using NormBackward = decltype(&layernorm_bwd_kernel<1, 0>);
constexpr NormForward kNormForward[4][kRowUnits + 1] = {
    {nullptr, layernorm_fwd_kernel<1, 1>, layernorm_fwd_kernel<1, 2>, layernorm_fwd_kernel<1, 3>, layernorm_fwd_kernel<1, 4>, layernorm_fwd_kernel<1, 5>},
    {nullptr, nullptr, nullptr, layernorm_fwd_kernel<2, 3>, layernorm_fwd_kernel<2, 4>, layernorm_fwd_kernel<2, 5>},
    {nullptr, nullptr, nullptr, layernorm_fwd_kernel<4, 3>, layernorm_fwd_kernel<4, 4>, layernorm_fwd_kernel<4, 5>},
    {layernorm_fwd_kernel<8, 0>, nullptr, nullptr, layernorm_fwd_kernel<8, 3>, layernorm_fwd_kernel<8, 4>, layernorm_fwd_kernel<8, 5>}};
constexpr NormBackward kNormBackward[4][kRowUnits + 1] = {
    {layernorm_bwd_kernel<1, 0>, layernorm_bwd_kernel<1, 1>, layernorm_bwd_kernel<1, 2>, layernorm_bwd_kernel<1, 3>, layernorm_bwd_kernel<1, 4>,
     layernorm_bwd_kernel<1, 5>},
    {layernorm_bwd_kernel<2, 0>, nullptr, nullptr, layernorm_bwd_kernel<2, 3>, layernorm_bwd_kernel<2, 4>, layernorm_bwd_kernel<2, 5>},
    {layernorm_bwd_kernel<4, 0>, nullptr, nullptr, layernorm_bwd_kernel<4, 3>, layernorm_bwd_kernel<4, 4>, layernorm_bwd_kernel<4, 5>},
    {layernorm_bwd_kernel<8, 0>, nullptr, nullptr, layernorm_bwd_kernel<8, 3>, layernorm_bwd_kernel<8, 4>, layernorm_bwd_kernel<8, 5>}};

// ---- column sums (bias gradients) --------------------------------------------------------------------------
// A cluster of eight CTAs owns 64 columns and splits the rows; a warp reads four rows of 128 bytes per
// instruction. The CTAs' sums meet in the first one's shared memory, so there is no scratch buffer, no
// atomic and no second launch, and the order of the additions is fixed. Bound by HBM.
constexpr int kSumCluster = 8;
constexpr int kSumCols    = 64;
constexpr int kSumThreads = 256;

template <bool kVec>
__global__ void __cluster_dims__(kSumCluster, 1, 1) __launch_bounds__(kSumThreads)
    colsum_kernel(const __nv_bfloat16* x, __nv_bfloat16* out, int64_t rows, int64_t cols, int64_t ld)
{
    fu::ptx::grid_wait();
    fu::ptx::grid_trigger();
    constexpr int kGroups = kSumThreads / 8;  // rows a CTA reads at once; eight lanes of 8 columns each per row
    constexpr int kAhead  = 4;
    __shared__ float part[kGroups][kSumCols + 4];
    __shared__ float total[kSumCluster][kSumCols];
    // the first CTA's shared memory is written by the others: they say here that they have started
    // and wait for that just before they write
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
    const int     rank = static_cast<int>(fu::ptx::cluster_ctarank());
    const int     cg   = threadIdx.x & 7, rg = threadIdx.x >> 3;
    const int64_t c0   = static_cast<int64_t>(blockIdx.y) * kSumCols + cg * 8;
    float         acc[8] = {};
    const int64_t step = static_cast<int64_t>(kSumCluster) * kGroups;
    for (int64_t r0 = rank * kGroups + rg; r0 < rows; r0 += step * kAhead) {
        uint4 v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int64_t r = r0 + u * step;
            v[u]            = make_uint4(0u, 0u, 0u, 0u);
            if (r < rows) {
                if (kVec && c0 + 8 <= cols) {
                    v[u] = fu::ptx::ld_once_v4(x + r * ld + c0);
                }
                else {
                    __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&v[u]);
                    for (int k = 0; k < 8; ++k) {
                        if (c0 + k < cols) {
                            e[k] = x[r * ld + c0 + k];
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[u]);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 f = __bfloat1622float2(h[k]);
                acc[2 * k] += f.x;
                acc[2 * k + 1] += f.y;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        part[rg][cg * 8 + k] = acc[k];
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait;" ::: "memory");
    if (threadIdx.x < kSumCols) {
        float s = 0.f;
#pragma unroll 8
        for (int g = 0; g < kGroups; ++g) {
            s += part[g][threadIdx.x];
        }
        const uint32_t to = fu::ptx::cluster_addr(&total[rank][threadIdx.x], 0);
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to), "f"(s) : "memory");
    }
    fu::ptx::cluster_sync();
    const int64_t col = static_cast<int64_t>(blockIdx.y) * kSumCols + threadIdx.x;
    if (rank == 0 && threadIdx.x < kSumCols && col < cols) {
        float s = 0.f;
#pragma unroll
        for (int g = 0; g < kSumCluster; ++g) {
            s += total[g][threadIdx.x];
        }
        out[col] = __float2bfloat16(s);
    }
}

// ---- the same backward, fed by the head owners' memory ----------------------------------------------
constexpr int MAX_HEADS = 128;

struct PullGrads {
    const uint8_t*       src[3][FU_MAX_WORLD];  // dq, dk, dv of every rank: (b, s_total, heads_of[p], 128) bf16
    fu::Peers            peers;
    const __nv_bfloat16* y;                     // (m, 2 * heads * 128) pre-norm q | k, leading dim ld_y
    __nv_bfloat16*       dy;                    // (m, 3 * heads * 128): d(projection) for q | k | v
    const float2*        rope;                  // (s_local, 64)
    const float*         gamma[2];
    float*               dgamma[2];
    int64_t              ld_y, ld_dy;
    int64_t              m, s_local, seq_off, s_total;
    int                  heads, handshake;
    float                eps;
    uint8_t              owner[MAX_HEADS], local[MAX_HEADS], heads_of[FU_MAX_WORLD];
};

// Bound by HBM (or the link). 75600 tokens x 40 heads on one GPU, 6.2 GB: 1.6 ms; 5.0 with a warp per row,
// whose 64-bit index arithmetic filled the issue slots. 256 tokens x 2 heads: 11 us; 153 when every warp
// of a full grid added its d(gamma) with atomics of its own.
__global__ void __launch_bounds__(256, 2) pull_qkv_grads_kernel(const __grid_constant__ PullGrads p)
{
    fu::ptx::grid_wait();
    if (p.peers.world == 1) {
        fu::ptx::grid_trigger();
    }
    __shared__ uint32_t       ticket;
    __shared__ const uint8_t* from[3][MAX_HEADS];
    __shared__ uint32_t       pitch[MAX_HEADS];
    __shared__ float          red[8][128];
    constexpr int             kInFlight = 2;
    const int      lane = threadIdx.x & 31;
    const int      warp = threadIdx.x >> 5;
    const uint64_t base = *reinterpret_cast<volatile uint64_t*>(&p.peers.own->epoch);
    // Opening: every rank says "my dq, dk, dv are complete" (stream order put this kernel after its
    // attention backward); nobody reads a peer before that. Every CTA polls the local flags itself.
    if (p.handshake && warp == 0) {
        if (blockIdx.x == 0) {
            fu::hs_announce(p.peers, base + 1);
        }
        fu::hs_await(p.peers, base + 1, FU_ST_OPEN_TIMEOUT);
    }
    __syncthreads();

    // A warp takes four neighbouring heads of a token at a time, kInFlight such groups together: a load
    // from a peer takes microseconds, and with one group the kernel would wait on latency instead of
    // on the link. Where a head lives is looked up in shared memory (the lanes of a group may differ).
    for (int i = threadIdx.x; i < p.heads; i += blockDim.x) {
        const int peer = p.owner[i];
        pitch[i]       = static_cast<uint32_t>(p.heads_of[peer]) * 256u;
        for (int t = 0; t < 3; ++t) {
            from[t][i] = p.src[t][peer] + p.local[i] * 256;
        }
    }
    __syncthreads();
    const int      sub    = lane >> 3, part = lane & 7;
    const uint32_t warp0  = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t groups = (static_cast<uint32_t>(p.heads) + 3) / 4;
    const uint32_t s_loc  = static_cast<uint32_t>(p.s_local);
    const uint32_t items  = static_cast<uint32_t>(p.m) * groups;  // per projection
    for (int t = 0; t < 3; ++t) {
        float dg[16] = {};
        for (uint32_t it0 = warp0; it0 < items; it0 += nwarps * kInFlight) {
            RowPart  g[kInFlight], y[kInFlight];
            uint32_t rows[kInFlight], ss[kInFlight];
            int      hds[kInFlight];  // -1: nothing here for this lane
#pragma unroll
            for (int u = 0; u < kInFlight; ++u) {
                const uint32_t it = it0 + u * nwarps;
                hds[u]            = -1;
                if (it < items) {
                    const uint32_t row   = it / groups;
                    const int      head  = static_cast<int>(it - row * groups) * 4 + sub;
                    const uint32_t batch = row / s_loc;
                    rows[u]              = row;
                    ss[u]                = row - batch * s_loc;
                    if (head < p.heads) {
                        hds[u] = head;
                        g[u]   = load_part(from[t][head] + (batch * p.s_total + p.seq_off + ss[u]) * pitch[head] + part * 8);
                        if (t < 2) {
                            y[u] = load_part(p.y + row * p.ld_y + (t * p.heads + head) * 128 + part * 4);
                        }
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < kInFlight; ++u) {
                if (it0 + u * nwarps >= items) {
                    break;  // warp-uniform
                }
                RowPart out = g[u];  // dv needs no transformation
                if (t < 2) {
                    float own[16] = {};
                    out = norm_rope_bwd(g[u], y[u], reinterpret_cast<const float*>(p.rope + static_cast<int64_t>(ss[u]) * 64),
                                        p.gamma[t], p.eps, part, own);
                    if (hds[u] >= 0) {
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            dg[e] += own[e];
                        }
                    }
                }
                if (hds[u] >= 0) {
                    store_part(p.dy + rows[u] * p.ld_dy + (static_cast<int64_t>(t) * p.heads + hds[u]) * 128 + part * 4, out);
                }
            }
        }
        if (t < 2) {
            add_dgamma(dg, p.dgamma[t], red);
        }
    }
    // Closing: "I have finished reading everybody's gradients", so that their owners may overwrite
    // them; the CTA that finishes last says it and waits for the same word from every peer.
    __syncthreads();
    if (threadIdx.x == 0) {
        ticket = atomicAdd(&p.peers.own->arrive[0], 1u);
    }
    __syncthreads();
    if (ticket == gridDim.x - 1 && warp == 0) {
        if (p.handshake) {
            fu::ptx::fence_sys();
            fu::hs_announce(p.peers, base + 2);
            fu::hs_await(p.peers, base + 2, FU_ST_CLOSE_TIMEOUT);
        }
        if (lane == 0) {
            p.peers.own->arrive[0] = 0;
            __threadfence();
            *reinterpret_cast<volatile uint64_t*>(&p.peers.own->epoch) = base + 2;
        }
    }
}

// The tables are read four floats, the rows four bf16 values at a time.
bool misaligned(uintptr_t bytes, std::initializer_list<const void*> operands)
{
    return std::any_of(operands.begin(), operands.end(), [&](const void* p) { return reinterpret_cast<uintptr_t>(p) % bytes != 0; });
}

}  // namespace

extern "C" int fu_qk_norm_rope_bwd(const FuNormRopeBwdArgs* a, void* stream)
{
    if (!a || !a->dq || !a->dk || !a->y || !a->dy || !a->rope || !a->gamma_q || !a->gamma_k) {
        return fu::fail(FU_E_ARG, "fu_qk_norm_rope_bwd: null operand");
    }
    if (a->m <= 0 || a->heads <= 0 || a->s_local <= 0 || (a->ld_y % 4) || (a->ld_dy % 4)) {
        return fu::fail(FU_E_ARG, "fu_qk_norm_rope_bwd: bad shape");
    }
    if (misaligned(16, {a->rope, a->gamma_q, a->gamma_k}) || misaligned(8, {a->dq, a->dk, a->y, a->dy})) {
        return fu::fail(FU_E_ARG, "fu_qk_norm_rope_bwd: rope and norm weights need 16-byte alignment, rows 8-byte");
    }
    NormRopeBwd p{};
    p.g[0]      = static_cast<const __nv_bfloat16*>(a->dq);
    p.g[1]      = static_cast<const __nv_bfloat16*>(a->dk);
    p.y         = static_cast<const __nv_bfloat16*>(a->y);
    p.dy        = static_cast<__nv_bfloat16*>(a->dy);
    p.rope      = reinterpret_cast<const float2*>(a->rope);
    p.gamma[0]  = a->gamma_q;
    p.gamma[1]  = a->gamma_k;
    p.dgamma[0] = a->dgamma_q;
    p.dgamma[1] = a->dgamma_k;
    p.ld_y      = a->ld_y;
    p.ld_dy     = a->ld_dy;
    p.m         = a->m;
    p.s_local   = a->s_local;
    p.heads     = a->heads;
    p.eps       = a->eps;
    int dev = 0, sms = 0;
    FU_CUDA_OK(cudaGetDevice(&dev));
    FU_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    qk_norm_rope_bwd_kernel<<<static_cast<int>(std::min<int64_t>(sms * 8, (a->m * a->heads + 31) / 32)), 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
    FU_CUDA_OK(cudaGetLastError());
    return FU_OK;
}

extern "C" int fu_pull_qkv_grads_check(const FuPullGradsArgs* a)
{
    if (!a || !a->y || !a->dy || !a->rope || !a->gamma_q || !a->gamma_k) {
        return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: null operand");
    }
    if (a->world < 1 || a->world > FU_MAX_WORLD || a->rank < 0 || a->rank >= a->world) {
        return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: rank %d / world %d", a->rank, a->world);
    }
    if (a->m <= 0 || a->heads <= 0 || a->heads > MAX_HEADS || a->s_local <= 0 || a->m % a->s_local || (a->ld_y % 4)
        || (a->ld_dy % 4)) {
        return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: bad shape (m=%lld heads=%d s_local=%lld)", (long long)a->m, a->heads,
                        (long long)a->s_local);
    }
    if (a->seq_off < 0 || a->s_total <= 0 || a->seq_off + a->s_local > a->s_total) {
        return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: rows %lld..%lld do not lie inside a sequence of %lld",
                        (long long)a->seq_off, (long long)(a->seq_off + a->s_local), (long long)a->s_total);
    }
    if (misaligned(16, {a->rope, a->gamma_q, a->gamma_k}) || misaligned(8, {a->y, a->dy})) {
        return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: rope and norm weights need 16-byte alignment, y and dy 8-byte");
    }
    int heads_seen = 0;
    const int64_t batches = a->m / a->s_local;
    for (int p = 0; p < a->world; ++p) {
        if (a->head_splits[p] < 0 || a->head_splits[p] > 255 || !a->peer_dq[p] || !a->peer_dk[p] || !a->peer_dv[p]
            || !a->peer_ctrl[p]) {
            return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: bad shard or missing buffer for rank %d", p);
        }
        if (misaligned(8, {a->peer_dq[p], a->peer_dk[p], a->peer_dv[p]})) {
            return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: the buffers of rank %d need 8-byte alignment", p);
        }
        heads_seen += a->head_splits[p];
        // row (batch, seq_off + s) of rank p's buffers starts at ((batch * s_total + seq_off + s) * head_splits[p]) * 256
        const int64_t last = ((batches - 1) * a->s_total + a->seq_off + a->s_local) * a->head_splits[p] * 256;
        if (last > a->src_bytes) {
            return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: the loads from rank %d reach byte %lld of buffers of %lld bytes", p,
                            (long long)last, (long long)a->src_bytes);
        }
    }
    if (heads_seen != a->heads) {
        return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: head_splits sum to %d, expected %d", heads_seen, a->heads);
    }
    return FU_OK;
}

extern "C" int fu_pull_qkv_grads(const FuPullGradsArgs* a, void* stream)
{
    const int rc = fu_pull_qkv_grads_check(a);
    if (rc != FU_OK) {
        return rc;
    }
    PullGrads p{};
    int       h = 0;
    for (int r = 0; r < a->world; ++r) {
        p.src[0][r]     = static_cast<const uint8_t*>(a->peer_dq[r]);
        p.src[1][r]     = static_cast<const uint8_t*>(a->peer_dk[r]);
        p.src[2][r]     = static_cast<const uint8_t*>(a->peer_dv[r]);
        p.peers.ctrl[r] = a->peer_ctrl[r];
        p.heads_of[r]   = static_cast<uint8_t>(a->head_splits[r]);
        for (int i = 0; i < a->head_splits[r]; ++i, ++h) {
            p.owner[h] = static_cast<uint8_t>(r);
            p.local[h] = static_cast<uint8_t>(i);
        }
    }
    p.peers.own        = a->peer_ctrl[a->rank];
    p.peers.rank       = a->rank;
    p.peers.world      = a->world;
    p.peers.mute       = (a->flags & FU_A2A_MUTE) ? 1 : 0;
    p.peers.timeout_ns = static_cast<uint64_t>(a->timeout_ms ? a->timeout_ms : 10000) * 1000000ull;
    p.handshake        = (a->flags & FU_A2A_NO_HANDSHAKE) ? 0 : 1;
    p.y                = static_cast<const __nv_bfloat16*>(a->y);
    p.dy               = static_cast<__nv_bfloat16*>(a->dy);
    p.rope             = reinterpret_cast<const float2*>(a->rope);
    p.gamma[0]         = a->gamma_q;
    p.gamma[1]         = a->gamma_k;
    p.dgamma[0]        = a->dgamma_q;
    p.dgamma[1]        = a->dgamma_k;
    p.ld_y             = a->ld_y;
    p.ld_dy            = a->ld_dy;
    p.m                = a->m;
    p.s_local          = a->s_local;
    p.seq_off          = a->seq_off;
    p.s_total          = a->s_total;
    p.heads            = a->heads;
    p.eps              = a->eps;
    int dev = 0, sms = 0, per_sm = 0;
    FU_CUDA_OK(cudaGetDevice(&dev));
    FU_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // One wave: the CTA that finishes last waits for the peers, and CTAs that have not started yet
    // must not be what a peer is waiting for. Every CTA of the first wave gets to run whatever
    // else is on the device, and a resident grid keeps the closing handshake prompt.
    FU_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pull_qkv_grads_kernel, 256, 0));
    const int64_t warps = a->m * ((a->heads + 3) / 4);  // no more CTAs than there are groups of rows
    if (warps * 2 > 0xffffffffll - (1ll << 22)) {  // index arithmetic is 32 bits wide, one grid of items beyond the last included
        return fu::fail(FU_E_ARG, "fu_pull_qkv_grads: %lld tokens x %d heads", (long long)a->m, a->heads);
    }
    const int grid = static_cast<int>(std::min<int64_t>(sms * (per_sm > 0 ? per_sm : 1), (warps + 7) / 8));
    if (a->world == 1) {
        FU_CUDA_OK(fu::launch_behind(pull_qkv_grads_kernel, dim3(static_cast<unsigned>(grid)), dim3(256), 0, static_cast<cudaStream_t>(stream), p));
        return FU_OK;
    }
    pull_qkv_grads_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
    FU_CUDA_OK(cudaGetLastError());
    return FU_OK;
}

extern "C" int fu_layernorm_fwd(const void* x, void* y, float* stats, int64_t rows, int64_t cols, int64_t ldx, int64_t ldy,
                                float eps, void* stream)
{
    if (!x || !y || rows <= 0 || cols <= 0 || (cols % 8) || (ldx % 8) || (ldy % 8)
        || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15u)) {
        return fu::fail(FU_E_ARG, "fu_layernorm_fwd: needs 16-byte aligned rows of a multiple of 8 columns");
    }
    const RowShape shape(rows, cols);
    FU_CUDA_OK(fu::launch_behind(kNormForward[shape.lg_warps][shape.units], dim3(shape.blocks), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                 static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), stats, rows, cols, ldx, ldy, eps));
    return FU_OK;
}

extern "C" int fu_layernorm_bwd_add(const void* dy, const void* x, const float* stats, const void* add, void* dx, int64_t rows,
                                    int64_t cols, int64_t ld, void* stream)
{
    if (!dy || !x || !stats || !dx || rows <= 0 || cols <= 0 || (cols % 8) || (ld % 8)
        || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx)
             | reinterpret_cast<uintptr_t>(add)) & 15u)) {
        return fu::fail(FU_E_ARG, "fu_layernorm_bwd_add: needs 16-byte aligned rows of a multiple of 8 columns");
    }
    RowShape shape(rows, cols);
    if (add && rows * cols > kNormInL2) {
        shape.units = 0;
    }
    FU_CUDA_OK(fu::launch_behind(kNormBackward[shape.lg_warps][shape.units], dim3(shape.blocks), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                 static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x), stats,
                                 static_cast<const __nv_bfloat16*>(add), static_cast<__nv_bfloat16*>(dx), rows, cols, ld));
    return FU_OK;
}

extern "C" int fu_colsum_bf16(const void* x, void* out, int64_t rows, int64_t cols, int64_t ld, void* stream)
{
    if (!x || !out || rows <= 0 || cols <= 0) {
        return fu::fail(FU_E_ARG, "fu_colsum_bf16: null or empty operand");
    }
    const bool     vec    = (ld % 8) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    const dim3     grid(kSumCluster, static_cast<unsigned>((cols + kSumCols - 1) / kSumCols));
    auto           kernel = vec ? colsum_kernel<true> : colsum_kernel<false>;
    // Clusters of eight that come up beside the kernel before crowd on the SMs that it left first: with more than a little to read,
    // waiting for all SMs is faster. Between two GEMMs, launched behind the first and in the ordinary way (us): 300 x 1288 12.1 and
    // 12.6, 1100 x 640 14.6 and 14.9; 2640 x 640 25.5 and 24.5, 1000 x 5120 26.6 and 25.7, 2640 x 8832 68.0 and 64.8.
    if (rows * cols <= (1 << 20)) {
        FU_CUDA_OK(fu::launch_behind(kernel, grid, dim3(kSumThreads), 0, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(x),
                                     static_cast<__nv_bfloat16*>(out), rows, cols, ld));
        return FU_OK;
    }
    kernel<<<grid, kSumThreads, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(x),
                                                                        static_cast<__nv_bfloat16*>(out), rows, cols, ld);
    FU_CUDA_OK(cudaGetLastError());
    return FU_OK;
}
