// 3x3 "same" convolutions on bfloat16 activations with binary32
// accumulation on the tcgen05 tensor cores: forward (and data gradient, the
// same kernel with flipped, transposed weights) and weight gradient. These
// are the contractions of the learned relaxation surrogate; nothing here has
// a counterpart in the reference.
//
// Activation layout ("padded NHWC"): image b of H x W pixels with C channels
// is stored as (H + 2) x (W + 2) positions q = yp (W + 2) + xp, channels
// innermost, with a one-pixel zero border (yp = 0, H + 1 or xp = 0, W + 1).
// A tap (dy, dx) of the 3x3 stencil is then a constant offset
// off = dy (W + 2) + dx in q, and a run of 128 consecutive q is one GEMM
// M-tile whose rows keep a uniform stride even across image rows: outputs at
// the border columns are computed and discarded (2 of W + 2 columns).
//
// Forward: out[q][co] = sum_tap sum_ci in[q + off_tap][ci] W[co][ci][tap],
// an implicit GEMM with M = 128 positions, N = Cout, K = 9 Cin. The input
// rows of a CTA's M-tiles plus the stencil halo are staged once in shared
// memory, and one staged copy serves every tap: tap (dy, dx) only moves the
// descriptor's start row. Two kernels: k_conv3x3_fwd_ws (persistent, warps
// specialised; widths up to 124) stages with TMA, a position's channels in one
// swizzled row of 64 or 32 bytes; k_conv3x3_fwd (wider images) stages with
// cp.async as Cin/8 "chunk planes" (plane c holds channels 8c..8c+7 of every
// staged position, 16 B per position), the K-major core-matrix layout without
// swizzle. Weights are pre-packed in global memory in the latter layout.
//
// Weight gradient: dW[co][ci][tap] = sum_q dY[q][co] in[q + off_tap][ci],
// K = positions, both operands MN-major straight from TMA; persistent CTAs
// write one block of partial sums each, and a second kernel adds the blocks
// in a fixed order, so the result is deterministic.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <mutex>

#include "pfb_internal.h"
#include "tc_util.cuh"
#include "pfb200_surrogate.h"

namespace pfb {
namespace {

__device__ unsigned int g_conv_status = 0u;  // bit 0: an MMA completion wait gave up

using bf16 = __nv_bfloat16;

constexpr int kConvThreads = 128;  // 4 warps: one TMEM lane quadrant each
constexpr int kConvMT = 2;         // M-tiles (of 128 positions) per forward CTA

__host__ __device__ constexpr int round_up(int v, int m) { return (v + m - 1) / m * m; }

// Rows staged for a forward CTA: its MT x 128 positions plus the halo.
__host__ __device__ constexpr int fwd_rows(int W) { return kConvMT * 128 + 2 * (W + 2) + 2; }
// Chunk-plane stride in bytes; 32 mod 128 spreads the staging stores of the
// four planes of one position over distinct banks.
__host__ __device__ constexpr int fwd_plane(int W) { return round_up(fwd_rows(W) * 16, 128) + 32; }

template <int CIN, int COUT>
__host__ __device__ constexpr int fwd_smem(int W) {
    return (CIN / 8) * fwd_plane(W) + 9 * (CIN / 8) * COUT * 16 + 16;
}

template <int COUT>
__host__ __device__ constexpr uint32_t fwd_tmem_cols() {
    return kConvMT * COUT <= 32 ? 32u : kConvMT * COUT <= 64 ? 64u : 128u;
}

struct ConvFwdArgs {
    const bf16* x;     // [B][P2][CIN]
    bf16* y;           // [B][P2][COUT] or null
    float* yf;         // [B][P2][COUT] or null (binary32 copy of the output)
    float* y0;         // [B][H W] or null (channel 0 of the output, no border)
    const bf16* w;     // packed [9][CIN / 8][COUT][8]
    const float* bias; // [COUT] or null
    const bf16* gate;  // [B][P2][COUT] or null: output *= (gate > 0)
    int B, H, W;
    int relu;
    int tiles;  // CTAs per image
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kConvThreads) k_conv3x3_fwd(const __grid_constant__ ConvFwdArgs A) {
    static_assert(CIN % 16 == 0 && COUT % 16 == 0 && COUT <= 64, "channel counts");
    constexpr int NCA = CIN / 8;
    constexpr uint32_t NCOLS = fwd_tmem_cols<COUT>();
    extern __shared__ __align__(128) unsigned char smem[];
    const int W2 = A.W + 2;
    const int P2 = (A.H + 2) * W2;
    const int CH = fwd_plane(A.W);
    const int RA = fwd_rows(A.W);
    unsigned char* sA = smem;
    unsigned char* sW = smem + NCA * CH;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sW + 9 * NCA * COUT * 16);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 1);

    const int tid = (int)threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int b = (int)blockIdx.x / A.tiles;
    const int tile = (int)blockIdx.x - b * A.tiles;
    const int q0 = W2 + tile * (kConvMT * 128);  // first output position
    const int qa = q0 - (W2 + 1);                // first staged position
    const int q_end = (A.H + 1) * W2;            // one past the last interior row

    if (tid == 0) dev::mbar_init(bar, 1);
    if (warp == 0) {
        tc::tmem_alloc(slot, NCOLS);
        tc::tmem_relinquish();
    }
    // stage the input rows (zero outside the image) and the packed weights
    const bf16* xb = A.x + (size_t)b * P2 * CIN;
    const uint32_t sa = dev::smem_addr(sA);
    for (int u = tid; u < RA * NCA; u += kConvThreads) {
        const int row = u / NCA, c = u - row * NCA;
        const int q = qa + row;
        const bool ok = q >= 0 && q < P2;
        tc::cp_async16(sa + (uint32_t)(c * CH + row * 16), xb + (size_t)(ok ? q : 0) * CIN + c * 8,
                       ok ? 16u : 0u);
    }
    const uint32_t sw = dev::smem_addr(sW);
    for (int u = tid; u < 9 * NCA * COUT; u += kConvThreads)
        tc::cp_async16(sw + (uint32_t)u * 16u, A.w + (size_t)u * 8, 16u);
    tc::cp_async_wait_all();
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *slot;

    if (tid == 0) {
        constexpr uint32_t idesc = tc::idesc_bf16_f32(128, COUT, false, false);
        for (int m = 0; m < kConvMT; ++m) {
            for (int tap = 0; tap < 9; ++tap) {
                const int dy = tap / 3, dx = tap - 3 * (tap / 3);
                const int row = m * 128 + dy * W2 + dx;
                for (int ks = 0; ks < CIN / 16; ++ks) {
                    const uint64_t ad = tc::smem_desc(sa + (uint32_t)(2 * ks * CH + row * 16),
                                                      (uint32_t)CH, 128u);
                    const uint64_t bd = tc::smem_desc(
                        sw + (uint32_t)((tap * NCA + 2 * ks) * COUT * 16), (uint32_t)(COUT * 16), 128u);
                    tc::mma_bf16(tmem + (uint32_t)(m * COUT), ad, bd, idesc, (tap | ks) ? 1u : 0u);
                }
            }
        }
        tc::mma_commit(bar);
    }
    // every thread takes the same branch (the TMEM loads are warp-collective)
    const bool done = __syncthreads_and(dev::mbar_wait_bounded(bar, 0, tc::kMmaWaitPolls)) != 0;
    tc::fence_after_sync();
    if (!done) {
        if (tid == 0) atomicOr(&g_conv_status, 1u);
    } else {
        const int r = warp * 32 + lane;
        for (int m = 0; m < kConvMT; ++m) {
            float acc[COUT];
            __syncwarp();
#pragma unroll
            for (int h = 0; h < COUT / 16; ++h) {
                uint32_t v[16];
                tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(m * COUT + 16 * h), v);
                tc::tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[16 * h + j] = __uint_as_float(v[j]);
            }
            const int q = q0 + m * 128 + r;
            if (q < q_end) {
            const int xp = q % W2;
            const bool interior = xp >= 1 && xp <= A.W;
            const size_t o = ((size_t)b * P2 + q) * COUT;
            float g[COUT];
#pragma unroll
            for (int j = 0; j < COUT; ++j) g[j] = 1.0f;
            if (A.gate && interior) {
#pragma unroll
                for (int h = 0; h < COUT / 8; ++h) {
                    const uint4 gv = *reinterpret_cast<const uint4*>(A.gate + o + 8 * h);
                    const bf16* ge = reinterpret_cast<const bf16*>(&gv);
#pragma unroll
                    for (int j = 0; j < 8; ++j) g[8 * h + j] = __bfloat162float(ge[j]) > 0.0f ? 1.0f : 0.0f;
                }
            }
#pragma unroll
            for (int j = 0; j < COUT; ++j) {
                float v = acc[j];
                if (A.bias) v += A.bias[j];
                if (A.relu) v = fmaxf(v, 0.0f);
                v *= g[j];
                acc[j] = interior ? v : 0.0f;
            }
            if (A.y) {
#pragma unroll
                for (int h = 0; h < COUT / 8; ++h) {
                    uint4 pk;
                    __nv_bfloat162* p2 = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        p2[j] = __floats2bfloat162_rn(acc[8 * h + 2 * j], acc[8 * h + 2 * j + 1]);
                    *reinterpret_cast<uint4*>(A.y + o + 8 * h) = pk;
                }
            }
            if (A.yf) {
#pragma unroll
                for (int h = 0; h < COUT / 4; ++h)
                    *reinterpret_cast<float4*>(A.yf + o + 4 * h) =
                        make_float4(acc[4 * h], acc[4 * h + 1], acc[4 * h + 2], acc[4 * h + 3]);
            }
            if (A.y0 && interior) A.y0[((size_t)b * A.H + (q / W2 - 1)) * A.W + (xp - 1)] = acc[0];
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, NCOLS);
}

// ---- forward, persistent and warp-specialised ----------------------------------
// The same contraction as k_conv3x3_fwd with the three stages of a tile in
// separate warps so that they overlap across tiles: warp 0 loads a tile's
// positions with TMA (cp.async.bulk.tensor, channels x positions x images, so
// positions outside the image arrive as zeros; a position's channels are one
// row of 64 or 32 bytes, swizzled over that width) into a ring of stages; warp
// 1 issues the tile's tcgen05 MMAs into one of two TMEM accumulators and
// commits; eight epilogue warps (one TMEM lane quadrant of one M-tile each) drain
// the previous tile. One staged copy serves all nine taps: a tap only moves the
// descriptor's first row, and the swizzle, which works on shared-memory
// address bits, stays in step with what TMA wrote. The packed weights are
// staged once per CTA with one bulk copy. Each CTA walks tiles c, c + G,
// c + 2G, ... of the B x tiles work list.
//
// 256 crops of 64 x 64, 32 -> 32 channels take 45 us (55 us gated) against 74
// (84) of one tile per CTA. No unit is near its limit then: of 74 k clocks the
// MMAs need 48 k (36 a tile, 45 clocks each at N = 32; tensor pipe 23 % active),
// DRAM and L2 are 26 % busy, the schedulers issue on 37 % of cycles. The largest
// stalls, long scoreboard (6.6 per issue) and short scoreboard (4.4), are of the
// kind that the epilogue's TMEM loads and its 16-byte stores 64 bytes apart give.
// Side-by-side taps (N = 96, a third of the MMAs, neighbouring lanes added by
// shuffles) measured 128 us with one CTA per SM, where this form took 53.
constexpr int kWsThreads = 64 + 128 * kConvMT;  // producer, MMA, epilogue warps of each M-tile
constexpr int kWsStages = 2;
constexpr int kWsHeader = 1024;  // barriers, bias

// rows per TMA box: half the staged rows, rounded up to 8 (two boxes)
__host__ __device__ constexpr int ws_box(int W) { return round_up((fwd_rows(W) + 1) / 2, 8); }
template <int CIN>
__host__ __device__ constexpr int ws_stage(int W) { return round_up(2 * ws_box(W) * CIN * 2, 1024); }

template <int CIN, int COUT>
__host__ __device__ constexpr int ws_smem(int W) {
    return kWsHeader + kWsStages * ws_stage<CIN>(W) + 9 * CIN * COUT * 2;
}

struct WsHeader {
    uint64_t full[kWsStages], empty[kWsStages], acc_full[2], acc_empty[2], wbar;
    uint32_t tmem_slot;
    int fail;
    alignas(16) float bias[64];
};
static_assert(sizeof(WsHeader) <= kWsHeader, "header");

__device__ __forceinline__ void tma_load3(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2,
                                          uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(kWsThreads)
    k_conv3x3_fwd_ws(const __grid_constant__ ConvFwdArgs A, const __grid_constant__ CUtensorMap X) {
    static_assert(CIN % 16 == 0 && COUT % 16 == 0 && COUT <= 64, "channel counts");
    constexpr int NCA = CIN / 8;
    constexpr uint32_t NCOLS = 2 * fwd_tmem_cols<COUT>();  // two accumulators
    constexpr uint32_t ACC = fwd_tmem_cols<COUT>();
    extern __shared__ __align__(1024) unsigned char smem[];
    WsHeader& H = *reinterpret_cast<WsHeader*>(smem);
    const int W2 = A.W + 2;
    const int P2 = (A.H + 2) * W2;
    const int BOX = ws_box(A.W);
    const int STAGE = ws_stage<CIN>(A.W);
    constexpr int ROW = CIN * 2;  // bytes of a position
    unsigned char* sA = smem + kWsHeader;                // stages
    unsigned char* sW = sA + (size_t)kWsStages * STAGE;  // packed weights
    const uint32_t sa = dev::smem_addr(sA), sw = dev::smem_addr(sW);
    const uint32_t stage_bytes = (uint32_t)(2 * BOX * ROW);
    const uint32_t wbytes = (uint32_t)(9 * NCA * COUT * 16);

    const int tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int items = A.B * A.tiles;
    const int q_end = (A.H + 1) * W2;

    // the swizzle works on address bits: stages start on multiples of 1024
    // bytes when the dynamic shared memory does; refuse to run otherwise
    if (dev::smem_addr(smem) & 1023u) {
        if (tid == 0) atomicOr(&g_conv_status, 2u);
        return;
    }
    if (tid == 0) {
        for (int s = 0; s < kWsStages; ++s) {
            dev::mbar_init(&H.full[s], 1);
            dev::mbar_init(&H.empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            dev::mbar_init(&H.acc_full[a], 1);
            dev::mbar_init(&H.acc_empty[a], 4 * kConvMT);  // one arrival per epilogue warp
        }
        dev::mbar_init(&H.wbar, 1);
        H.fail = 0;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        dev::mbar_arrive_expect_tx(&H.wbar, wbytes);
        dev::bulk_g2s(sW, A.w, wbytes, &H.wbar);
    }
    if (warp == 0) {
        tc::tmem_alloc(&H.tmem_slot, NCOLS);
        tc::tmem_relinquish();
    }
    if (tid >= 64 && tid < 64 + COUT) H.bias[tid - 64] = A.bias ? A.bias[tid - 64] : 0.0f;
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = H.tmem_slot;
    auto give_up = [&]() {
        H.fail = 1;
        atomicOr(&g_conv_status, 1u);
    };

    if (warp == 0 && lane == 0) {
        // ---- producer: the positions of each tile, two boxes
        int k = 0;
        for (int it = (int)blockIdx.x; it < items && !H.fail; it += (int)gridDim.x, ++k) {
            const int s = k % kWsStages;
            if (!dev::mbar_wait_bounded(&H.empty[s], (uint32_t)(((k / kWsStages) & 1) ^ 1), tc::kMmaWaitPolls)) {
                give_up();
                break;
            }
            const int b = it / A.tiles, t = it - b * A.tiles;
            const int qa = t * (kConvMT * 128) - 1;  // first staged position (W2 + t 256 - (W2 + 1))
            const uint32_t bar = dev::smem_addr(&H.full[s]);
            dev::mbar_arrive_expect_tx(&H.full[s], stage_bytes);
            for (int h = 0; h < 2; ++h)
                tma_load3(sa + (uint32_t)(s * STAGE + h * BOX * ROW), &X, 0, qa + h * BOX, b, bar);
        }
        // no copy may still target shared memory at exit
        for (int j = (k > kWsStages ? k - kWsStages : 0); j < k; ++j)
            (void)dev::mbar_wait_bounded(&H.full[j % kWsStages], (uint32_t)((j / kWsStages) & 1),
                                         tc::kMmaWaitPolls);
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issue
        if (!dev::mbar_wait_bounded(&H.wbar, 0, tc::kMmaWaitPolls)) give_up();
        constexpr uint32_t idesc = tc::idesc_bf16_f32(128, COUT, false, false);
        const uint64_t w0 = tc::smem_desc(sw, (uint32_t)(COUT * 16), 128u);
        int k = 0;
        for (int it = (int)blockIdx.x; it < items && !H.fail; it += (int)gridDim.x, ++k) {
            const int s = k % kWsStages, a = k & 1;
            if (!dev::mbar_wait_bounded(&H.full[s], (uint32_t)((k / kWsStages) & 1), tc::kMmaWaitPolls) ||
                !dev::mbar_wait_bounded(&H.acc_empty[a], (uint32_t)(((k >> 1) & 1) ^ 1), tc::kMmaWaitPolls)) {
                give_up();
                break;
            }
            tc::fence_after_sync();
            const uint32_t st = sa + (uint32_t)(s * STAGE);
            // start-address fields advance by bytes / 16
            const uint64_t a0 = tc::smem_desc_k<CIN>(st);
#pragma unroll
            for (int m = 0; m < kConvMT; ++m) {
                const uint32_t d = tmem + (uint32_t)(a * ACC + m * COUT);
#pragma unroll
                for (int dy = 0; dy < 3; ++dy) {
                    const uint64_t ay = a0 + (uint64_t)(uint32_t)((m * 128 + dy * W2) * (ROW / 16));
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
                        for (int ks = 0; ks < CIN / 16; ++ks)
                            tc::mma_bf16(d, ay + (uint64_t)(dx * (ROW / 16) + 2 * ks),
                                         w0 + (uint64_t)(((3 * dy + dx) * NCA + 2 * ks) * COUT), idesc,
                                         (dy | dx | ks) ? 1u : 0u);
                }
            }
            tc::mma_commit(&H.empty[s]);     // the stage may be refilled
            tc::mma_commit(&H.acc_full[a]);  // the accumulator may be read
        }
        // no MMA may still be writing TMEM when it is released
        if (k > 0)
            (void)dev::mbar_wait_bounded(&H.acc_full[(k - 1) & 1], (uint32_t)(((k - 1) >> 1) & 1),
                                         tc::kMmaWaitPolls);
    } else if (warp >= 2) {
        // ---- epilogue: TMEM lane quadrant warp % 4 of M-tile (warp - 2) / 4
        const int quad = warp & 3, m = (warp - 2) >> 2;
        const int r = m * 128 + quad * 32 + lane;
        int k = 0;
        for (int it = (int)blockIdx.x; it < items; it += (int)gridDim.x, ++k) {
            const int a = k & 1;
            const int b = it / A.tiles, t = it - b * A.tiles;
            const int q = W2 + t * (kConvMT * 128) + r;
            const bool in = q < q_end;
            const int xp = q % W2;
            const bool interior = xp >= 1 && xp <= A.W;
            const size_t o = ((size_t)b * P2 + q) * COUT;
            // the gate arrives while the tile's MMAs run
            uint4 gv[COUT / 8];
            const bool gated = A.gate && in && interior;
            if (gated)
#pragma unroll
                for (int h = 0; h < COUT / 8; ++h)
                    gv[h] = __ldg(reinterpret_cast<const uint4*>(A.gate + o) + h);
            const bool ok = dev::mbar_wait_bounded(&H.acc_full[a], (uint32_t)((k >> 1) & 1), tc::kMmaWaitPolls);
            if (!__all_sync(0xFFFFFFFFu, ok) || H.fail) {
                if (lane == 0 && !ok) give_up();
                break;
            }
            tc::fence_after_sync();
#pragma unroll
            for (int h = 0; h < COUT / 16; ++h) {
                __syncwarp();  // the TMEM loads are warp-collective
                uint32_t u[16];
                tc::tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(a * ACC + m * COUT + 16 * h), u);
                tc::tmem_wait_ld();
                if (!in) continue;
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float4 bj = *reinterpret_cast<const float4*>(&H.bias[16 * h + j]);
                    v[j] = __uint_as_float(u[j]) + bj.x;
                    v[j + 1] = __uint_as_float(u[j + 1]) + bj.y;
                    v[j + 2] = __uint_as_float(u[j + 2]) + bj.z;
                    v[j + 3] = __uint_as_float(u[j + 3]) + bj.w;
                }
                if (A.relu)
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j], 0.0f);
                if (gated)
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const bf16* ge = reinterpret_cast<const bf16*>(&gv[2 * h + j / 8]);
                        v[j] *= __bfloat162float(ge[j % 8]) > 0.0f ? 1.0f : 0.0f;
                    }
                if (!interior)
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = 0.0f;
                if (A.y)
#pragma unroll
                    for (int k8 = 0; k8 < 2; ++k8) {
                        uint4 pk;
                        __nv_bfloat162* p2 = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            p2[j] = __floats2bfloat162_rn(v[8 * k8 + 2 * j], v[8 * k8 + 2 * j + 1]);
                        *reinterpret_cast<uint4*>(A.y + o + 16 * h + 8 * k8) = pk;
                    }
                if (A.yf)
#pragma unroll
                    for (int j = 0; j < 16; j += 4)
                        *reinterpret_cast<float4*>(A.yf + o + 16 * h + j) =
                            make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                if (A.y0 && h == 0 && interior) A.y0[((size_t)b * A.H + (q / W2 - 1)) * A.W + (xp - 1)] = v[0];
            }
            // the accumulator is free again
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(dev::smem_addr(&H.acc_empty[a])) : "memory");
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, NCOLS);
}

// ---- weight gradient --------------------------------------------------------
// dW[tap] = sum over positions p of dY[p - dx] x[p + dy (W + 2)]: both
// operands are MN-major tiles of kWgKT positions, channels innermost, exactly
// as TMA lays an activation box down (rows of one position, 64 or 32 bytes,
// swizzled over that width). The 128 rows of A are 128 / CY slots of CY
// channels, slot s the dY tile moved by s - 1 positions: one staged copy with
// a leading offset of one row (slots past the third are not used). B holds the
// x tiles of the three dy and a tile of ones side by side (N = 3 CX + 16: the
// last columns are the bias gradient), so 16 positions take one MMA. The width
// matters: a 128-row MMA of K = 16 takes 45 clocks up to N = 48 and 58 at
// N = 112 (measured), so three of N = 32 or nine of one tap each would be bound
// by their number.
//
// Warp-specialised and persistent, one CTA per SM: CTA c owns a contiguous
// range of the B x chunks tiles; warp 0 keeps a ring of kWgStages tiles in
// flight, warp 1 issues, and warps 2-5 take the accumulator out of TMEM after
// every run of `run` tiles, add it to the CTA's sums in registers and write
// those at the end. The tensor core adds into its accumulator with a bias
// towards zero, so the error of one-signed sums grows with the length of the
// chain: 2.7e-5 of the gradient over a CTA's whole range at 256 crops of
// 64 x 64 (457 additions), 5.6e-6 over half an image (132), 2.2e-6 over the 66
// of a run. Two accumulators keep the MMAs going meanwhile.
//
// 256 crops of 64 x 64, 32 -> 32 channels: 50.1 us a layer with the reduction,
// launches back to back (49.5 us with runs of half an image, 51.2 of 6 tiles),
// against about 200 of one CTA per half image that staged nine shifted copies of
// x with cp.async. Of the 86 k clocks of a launch the MMAs need 27 k (tensor
// pipe 30 % active); DRAM is 38 % and L2 27 % busy. What is left is the fill: 392 rows of 64 bytes a tile, 0.28
// GB a layer, one row per 2.9 clocks and SM.
constexpr int kWgStages = 6;
constexpr int kWgThreads = 192;
constexpr int kWgKT = 96;        // positions per tile: divides 64 x 66 exactly
constexpr int kWgHeader = 1024;  // barriers
constexpr uint32_t kWgCols = 128;  // TMEM columns of an accumulator: CX per dy, then 16 of the bias
constexpr int kWgRun = 11;       // most tiles summed in one accumulator

constexpr int kWgYRows = kWgKT + 8;  // dY rows staged: the last slot is moved by 7 at most
// A stage: the dY tile, three x tiles, a tile of ones.
template <int CY>
__host__ __device__ constexpr int wg_dy_bytes() { return round_up(kWgYRows * CY * 2, 1024); }
template <int CX, int CY>
__host__ __device__ constexpr int wg_stage_bytes() { return wg_dy_bytes<CY>() + 4 * kWgKT * CX * 2; }
template <int CX, int CY>
__host__ __device__ constexpr int wg_smem() {
    return kWgHeader + kWgStages * wg_stage_bytes<CX, CY>();
}

struct WgHeader {
    uint64_t full[kWgStages], empty[kWgStages], acc_full[2], acc_empty[2];
    uint32_t tmem_slot;
    int fail;
};

struct ConvWgradArgs {
    float* partial;  // [grid][9 * CY * CX + CY]
    int W2;          // padded row length
    int chunks;      // tiles per image
    int items;       // tiles of the batch
    int run;         // tiles summed in one accumulator
};

// DY covers image rows 1 .. H of the gradient (positions outside read as
// zeros), X the whole padded image.
template <int CX, int CY>
__global__ void __launch_bounds__(kWgThreads, 1)
    k_conv3x3_wgrad(const __grid_constant__ ConvWgradArgs A, const __grid_constant__ CUtensorMap X,
                    const __grid_constant__ CUtensorMap DY) {
    static_assert((CX == 16 || CX == 32) && (CY == 16 || CY == 32), "one swizzle atom per position");
    constexpr int AT = wg_dy_bytes<CY>(), BT = kWgKT * CX * 2;  // bytes of the dY and of an x tile
    constexpr int STAGE = wg_stage_bytes<CX, CY>();
    static_assert(AT % 1024 == 0 && BT % 1024 == 0 && kWgKT % 16 == 0, "tiles keep the swizzle phase");
    static_assert(kWgKT + 128 / CY - 1 <= kWgYRows, "every slot's rows are staged");
    extern __shared__ __align__(1024) unsigned char smem[];
    WgHeader& H = *reinterpret_cast<WgHeader*>(smem);
    const uint32_t base = dev::smem_addr(smem);
    const uint32_t st0 = base + kWgHeader;
    const int tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = (int)gridDim.x, c = (int)blockIdx.x;
    const int i0 = (int)((long long)A.items * c / G), i1 = (int)((long long)A.items * (c + 1) / G);

    // the swizzle works on address bits: refuse to run on an unaligned window
    const bool aligned = (base & 1023u) == 0u;
    if (tid == 0) {
        for (int s = 0; s < kWgStages; ++s) {
            dev::mbar_init(&H.full[s], 1);
            dev::mbar_init(&H.empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            dev::mbar_init(&H.acc_full[a], 1);
            dev::mbar_init(&H.acc_empty[a], 4);  // one arrival per epilogue warp
        }
        H.fail = aligned ? 0 : 1;
        if (!aligned) atomicOr(&g_conv_status, 2u);
    }
    for (int i = tid; i < kWgStages * (BT / 16); i += kWgThreads) {
        const int s = i / (BT / 16), j = i - s * (BT / 16);
        *reinterpret_cast<uint4*>(smem + kWgHeader + s * STAGE + AT + 3 * BT + j * 16) =
            make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);
    }
    if (warp == 0) {
        tc::tmem_alloc(&H.tmem_slot, 2 * kWgCols);
        tc::tmem_relinquish();
    }
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = H.tmem_slot;
    auto give_up = [&]() {
        *reinterpret_cast<volatile int*>(&H.fail) = 1;
        atomicOr(&g_conv_status, 1u);
    };
    auto failed = [&]() { return *reinterpret_cast<volatile int*>(&H.fail) != 0; };

    if (warp == 0 && lane == 0) {
        // ---- producer
        int k = 0;
        for (int it = i0; it < i1 && !failed(); ++it, ++k) {
            const int s = k % kWgStages;
            if (!dev::mbar_wait_bounded(&H.empty[s], (uint32_t)(((k / kWgStages) & 1) ^ 1), tc::kMmaWaitPolls)) {
                give_up();
                break;
            }
            const int b = it / A.chunks, p = (it - b * A.chunks) * kWgKT;
            const uint32_t bar = dev::smem_addr(&H.full[s]);
            const uint32_t st = st0 + (uint32_t)(s * STAGE);
            dev::mbar_arrive_expect_tx(&H.full[s], (uint32_t)(kWgYRows * CY * 2 + 3 * BT));
            tma_load3(st, &DY, 0, p - 1, b, bar);
            for (int d = 0; d < 3; ++d)
                tma_load3(st + (uint32_t)(AT + d * BT), &X, 0, p + d * A.W2, b, bar);
        }
        // no copy may still target shared memory at exit
        for (int j = (k > kWgStages ? k - kWgStages : 0); j < k; ++j)
            (void)dev::mbar_wait_bounded(&H.full[j % kWgStages], (uint32_t)((j / kWgStages) & 1),
                                         tc::kMmaWaitPolls);
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issue
        constexpr uint32_t id = tc::idesc_bf16_f32(128, 3 * CX + 16, true, true);
        constexpr uint32_t KS_A = 16 * CY * 2, KS_B = 16 * CX * 2;  // 16 positions
        int k = 0, u = 0, t = 0;  // tile of the range, run u, tile t of the run
        for (int it = i0; it < i1 && !failed(); ++it, ++k) {
            const int s = k % kWgStages, a = u & 1;
            if (!dev::mbar_wait_bounded(&H.full[s], (uint32_t)((k / kWgStages) & 1), tc::kMmaWaitPolls) ||
                (t == 0 &&
                 !dev::mbar_wait_bounded(&H.acc_empty[a], (uint32_t)(((u >> 1) & 1) ^ 1), tc::kMmaWaitPolls))) {
                give_up();
                break;
            }
            tc::fence_after_sync();
            const uint32_t st = st0 + (uint32_t)(s * STAGE);
            // a step adds its bytes / 16 to the start-address fields
            const uint64_t ad0 = tc::smem_desc_mn<CY>(st, (uint32_t)(CY * 2));
            const uint64_t bd0 = tc::smem_desc_mn<CX>(st + AT, (uint32_t)BT);
#pragma unroll
            for (int kk = 0; kk < kWgKT / 16; ++kk)
                tc::mma_bf16(tmem + (uint32_t)a * kWgCols, ad0 + (uint64_t)(kk * KS_A >> 4),
                             bd0 + (uint64_t)(kk * KS_B >> 4), id, (t | kk) ? 1u : 0u);
            tc::mma_commit(&H.empty[s]);
            if (++t == A.run || it + 1 == i1) {
                tc::mma_commit(&H.acc_full[a]);
                t = 0;
                ++u;
            }
        }
        // no MMA may still be writing TMEM when it is released; after a wait
        // that gave up, the run in hand is closed for the epilogue to see it
        if (t > 0) {
            tc::mma_commit(&H.acc_full[u & 1]);
            ++u;
        }
        if (u > 0)
            (void)dev::mbar_wait_bounded(&H.acc_full[(u - 1) & 1], (uint32_t)(((u - 1) >> 1) & 1),
                                         tc::kMmaWaitPolls);
    } else if (warp >= 2) {
        // ---- sums: row slot * CY + co of the accumulator is tap column
        // dx = 1 - slot (dY moved by slot - 1 meets x at the opposite offset)
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const int slot = row / CY, co = row % CY;
        const bool used = quad * 32 < 3 * CY;  // the warp holds rows of the three slots
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        float* out = A.partial + (size_t)c * (9 * CY * CX + CY);
        float sum[3 * CX], bias = 0.0f;
#pragma unroll
        for (int j = 0; j < 3 * CX; ++j) sum[j] = 0.0f;
        const int runs = (i1 - i0 + A.run - 1) / A.run;
#pragma unroll 1
        for (int u = 0; u < runs; ++u) {
            const int a = u & 1;
            const bool full = !failed() && dev::mbar_wait_bounded(&H.acc_full[a], (uint32_t)((u >> 1) & 1),
                                                                  tc::kMmaWaitPolls);
            if (!__all_sync(0xFFFFFFFFu, full && !failed())) {
                if (lane == 0) give_up();
                break;
            }
            tc::fence_after_sync();
            if (used) {
                const uint32_t acc = lanes + (uint32_t)a * kWgCols;
#pragma unroll
                for (int h = 0; h < 3 * CX / 16 + 1; ++h) {
                    uint32_t v[16];
                    tc::tmem_ld16(acc + (uint32_t)(16 * h), v);
                    tc::tmem_wait_ld();
                    if (h < 3 * CX / 16) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) sum[16 * h + j] += __uint_as_float(v[j]);
                    } else {
                        bias += __uint_as_float(v[0]);
                    }
                }
            }
            // the accumulator is free again
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(dev::smem_addr(&H.acc_empty[a]))
                             : "memory");
        }
        // the four warps agree on the outcome
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (failed()) {
            // a wait gave up: poison this CTA's block so the reduction yields
            // NaN instead of mixing in what the scratch held before
            for (int i = tid - 64; i < 9 * CY * CX + CY; i += 128) out[i] = __int_as_float(0x7fc00000);
        } else if (slot < 3) {
            // the lanes' output channels side by side
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int j = 0; j < CX; ++j) out[((3 * d + 2 - slot) * CX + j) * CY + co] = sum[d * CX + j];
            if (slot == 1) out[9 * CY * CX + co] = bias;
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 2 * kWgCols);
}

// dW[co][ci][tap] = sum over CTAs of partial[cta][tap][ci][co]; db[co] likewise.
// Two levels in a fixed order: thread row j of a CTA sums the blocks
// g = j, j + 16, j + 32, ... of 32 consecutive outputs (each warp reads 128
// contiguous bytes per block), then the 16 row sums are added in row order.
// The result does not depend on scheduling.
constexpr int kRedCols = 32, kRedRows = 16;

__global__ void __launch_bounds__(kRedCols * kRedRows)
    k_wgrad_reduce(const float* __restrict__ partial, int grid, int cx, int cy,
                   float* __restrict__ dw, float* __restrict__ db) {
    __shared__ float part[kRedRows][kRedCols + 1];
    const int per = 9 * cy * cx + cy;
    const int i = (int)blockIdx.x * kRedCols + (int)threadIdx.x;
    const int j = (int)threadIdx.y;
    float s = 0.0f;
    if (i < per) {
        int g = j;
        // four independent loads in flight, summed in order
        for (; g + 3 * kRedRows < grid; g += 4 * kRedRows) {
            const float a = partial[(size_t)g * per + i];
            const float b = partial[(size_t)(g + kRedRows) * per + i];
            const float c = partial[(size_t)(g + 2 * kRedRows) * per + i];
            const float d = partial[(size_t)(g + 3 * kRedRows) * per + i];
            s = (((s + a) + b) + c) + d;
        }
        for (; g < grid; g += kRedRows) s += partial[(size_t)g * per + i];
    }
    part[j][threadIdx.x] = s;
    __syncthreads();
    if (j != 0 || i >= per) return;
    float t = part[0][threadIdx.x];
#pragma unroll
    for (int r = 1; r < kRedRows; ++r) t += part[r][threadIdx.x];
    if (i < 9 * cy * cx) {
        const int tap = i / (cy * cx), rem = i - tap * cy * cx;
        const int ci = rem / cy, co = rem - ci * cy;
        dw[((size_t)co * cx + ci) * 9 + tap] = t;
    } else if (db) {
        db[i - 9 * cy * cx] = t;
    }
}

void launch_wgrad_reduce(const float* partial, int grid, int cx, int cy, float* dw, float* db,
                         cudaStream_t s) {
    const int per = 9 * cy * cx + cy;
    k_wgrad_reduce<<<(per + kRedCols - 1) / kRedCols, dim3(kRedCols, kRedRows), 0, s>>>(partial, grid, cx,
                                                                                        cy, dw, db);
}

// Packed weights from OIHW binary32 W[co][ci][3][3] (cout x cin):
//   forward  : P[tap][ci / 8][co][ci % 8] = W[co][ci][tap]
//   transpose: P[tap][co / 8][ci][co % 8] = W[co][ci][8 - tap]  (data gradient)
struct PackJobs {
    ConvPackJob job[16];
};

__global__ void k_pack_weights(const __grid_constant__ PackJobs J) {
    const ConvPackJob& job = J.job[blockIdx.y];
    const float* __restrict__ w = job.w;
    bf16* __restrict__ p = static_cast<bf16*>(job.packed);
    const int cin = job.cin, cout = job.cout, transpose = job.transpose;
    const int n = 9 * cin * cout;
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    const int ki = transpose ? cout : cin;  // K channels of the packed operand
    const int ni = transpose ? cin : cout;  // N rows
    const int j = i % 8, rest = i / 8;
    const int nrow = rest % ni, rest2 = rest / ni;
    const int kc = rest2 % (ki / 8), tap = rest2 / (ki / 8);
    const int kch = kc * 8 + j;
    float v;
    if (!transpose)
        v = w[((size_t)nrow * cin + kch) * 9 + tap];
    else
        v = w[((size_t)kch * cin + nrow) * 9 + (8 - tap)];
    p[i] = __float2bfloat16_rn(v);
}

template <int CIN, int COUT>
cudaError_t launch_fwd_ws(const ConvFwdArgs& a, cudaStream_t s, bool* used);

template <int CIN, int COUT>
cudaError_t launch_fwd(const ConvFwdArgs& a, cudaStream_t s) {
    bool used = false;
    cudaError_t e0 = launch_fwd_ws<CIN, COUT>(a, s, &used);
    if (e0 != cudaSuccess || used) return e0;
    const int smem = fwd_smem<CIN, COUT>(a.W);
    cudaError_t e = cudaFuncSetAttribute(k_conv3x3_fwd<CIN, COUT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k_conv3x3_fwd<CIN, COUT><<<a.B * a.tiles, kConvThreads, smem, s>>>(a);
    return cudaGetLastError();
}

// 0: one tile per CTA; 1 (2 is accepted as the same): the persistent
// warp-specialised forward where two TMA boxes hold a tile's rows (W <= 124).
int g_conv_pipeline = 1;

PFN_cuTensorMapEncodeTiled_v12000 encode_tiled() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// Activations [B][P2][C] (positions pos0 .. pos0 + npos of each image) as a
// C channels x positions x images map of boxes of `box` positions, swizzled
// over the C channels of a position.
bool position_map(CUtensorMap* map, const bf16* base, int C, int P2, int pos0, int npos, int B, int box) {
    const cuuint64_t dims[3] = {(cuuint64_t)C, (cuuint64_t)npos, (cuuint64_t)B};
    const cuuint64_t strides[2] = {(cuuint64_t)C * 2, (cuuint64_t)P2 * C * 2};
    const cuuint32_t boxd[3] = {(cuuint32_t)C, (cuuint32_t)box, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
                          const_cast<bf16*>(base + (size_t)pos0 * C), dims, strides, boxd, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE,
                          C == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The persistent forward; *used = false (nothing launched) when the shape or
// the driver does not allow it.
template <int CIN, int COUT>
cudaError_t launch_fwd_ws(const ConvFwdArgs& a, cudaStream_t s, bool* used) {
    *used = false;
    const int smem = ws_smem<CIN, COUT>(a.W);
    PFN_cuTensorMapEncodeTiled_v12000 encode = encode_tiled();
    if (!g_conv_pipeline || !encode ||
        ws_box(a.W) > 256 || smem > 227 * 1024)
        return cudaSuccess;
    const int P2 = (a.H + 2) * (a.W + 2);
    CUtensorMap map;
    if (!position_map(&map, a.x, CIN, P2, 0, P2, a.B, ws_box(a.W))) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_conv3x3_fwd_ws<CIN, COUT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_conv3x3_fwd_ws<CIN, COUT>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 100);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    cudaFuncAttributes fa;
    if ((e = cudaFuncGetAttributes(&fa, k_conv3x3_fwd_ws<CIN, COUT>)) != cudaSuccess ||
        (e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    // CTAs an SM holds by shared memory (1 KB of it reserved per CTA),
    // registers and TMEM columns. The runtime's occupancy query is not used:
    // it answers 1 for this kernel, and one CTA leaves the SM waiting on its
    // own epilogue.
    const int by_smem = 228 * 1024 / (smem + 1024);
    const int by_regs = 65536 / (round_up(fa.numRegs * 32, 256) * (kWsThreads / 32));
    const int by_tmem = 512 / (2 * (int)fwd_tmem_cols<COUT>());
    int per = by_smem < by_regs ? by_smem : by_regs;
    per = per < by_tmem ? per : by_tmem;
    if (per < 1) per = 1;
    const int items = a.B * a.tiles;
    const int grid = items < sms * per ? items : sms * per;
    k_conv3x3_fwd_ws<CIN, COUT><<<grid, kWsThreads, smem, s>>>(a, map);
    *used = true;
    return cudaGetLastError();
}

template <int CX, int CY>
cudaError_t launch_wgrad(const ConvWgradArgs& a, const bf16* x, const bf16* dy, int B, int H, int W,
                         int grid, cudaStream_t s) {
    constexpr int smem = wg_smem<CX, CY>();
    const int W2 = W + 2, P2 = (H + 2) * W2;
    CUtensorMap mx, my;
    if (!encode_tiled() || !position_map(&mx, x, CX, P2, 0, P2, B, kWgKT) ||
        !position_map(&my, dy, CY, P2, W2, H * W2, B, kWgYRows))
        return cudaErrorNotSupported;
    cudaError_t e = cudaFuncSetAttribute(k_conv3x3_wgrad<CX, CY>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k_conv3x3_wgrad<CX, CY><<<grid, kWgThreads, smem, s>>>(a, mx, my);
    return cudaGetLastError();
}

bool shape_ok(int B, int H, int W) {
    return B > 0 && H >= 2 && W >= 2 && H <= 1024 && W <= 1024 && fwd_smem<32, 64>(W) <= 227 * 1024;
}

}  // namespace

// ---- internal entry points ------------------------------------------------------

int conv3x3_fwd(const void* x, void* y, float* yf, const void* wp, const float* bias,
                const void* gate, int B, int H, int W, int cin, int cout, int relu,
                cudaStream_t s, float* y0) {
    if (!x || !wp || (!y && !yf && !y0)) return set_error(PFB_E_ARG, "conv3x3: null buffer");
    if (!shape_ok(B, H, W)) return set_error(PFB_E_ARG, "conv3x3: bad shape %dx%dx%d", B, H, W);
    if ((uintptr_t)x % 16 || (uintptr_t)wp % 16 || (y && (uintptr_t)y % 16) ||
        (yf && (uintptr_t)yf % 16) || (gate && (uintptr_t)gate % 16))
        return set_error(PFB_E_ARG, "conv3x3: buffers must be 16-byte aligned");
    ConvFwdArgs a;
    a.x = static_cast<const bf16*>(x);
    a.y = static_cast<bf16*>(y);
    a.yf = yf;
    a.y0 = y0;
    a.w = static_cast<const bf16*>(wp);
    a.bias = bias;
    a.gate = static_cast<const bf16*>(gate);
    a.B = B;
    a.H = H;
    a.W = W;
    a.relu = relu ? 1 : 0;
    a.tiles = (H * (W + 2) + kConvMT * 128 - 1) / (kConvMT * 128);
    cudaError_t e;
    if (cin == 16 && cout == 32)
        e = launch_fwd<16, 32>(a, s);
    else if (cin == 32 && cout == 32)
        e = launch_fwd<32, 32>(a, s);
    else if (cin == 32 && cout == 16)
        e = launch_fwd<32, 16>(a, s);
    else if (cin == 16 && cout == 16)
        e = launch_fwd<16, 16>(a, s);
    else
        return set_error(PFB_E_CONFIG, "conv3x3: channels %d -> %d not built", cin, cout);
    if (e != cudaSuccess) return set_error(PFB_E_CUDA, "conv3x3: %s", cudaGetErrorString(e));
    return PFB_OK;
}

size_t conv3x3_wgrad_workspace(int B, int H, int W, int cx, int cy) {
    const int total = (H * (W + 2) + 63) / 64;
    const int blocks = total < 8 ? 1 : 2;  // per image
    return (size_t)B * blocks * (size_t)(9 * cy * cx + cy) * sizeof(float);
}

// One block of partial sums per CTA; a CTA per SM, as many as the workspace
// holds blocks for and there are tiles.
int conv3x3_wgrad(const void* x, const void* dy, float* workspace, size_t workspace_bytes,
                  float* dw, float* db, int B, int H, int W, int cx, int cy, cudaStream_t s) {
    if (!x || !dy || !workspace || !dw) return set_error(PFB_E_ARG, "conv3x3_wgrad: null buffer");
    if (!shape_ok(B, H, W)) return set_error(PFB_E_ARG, "conv3x3_wgrad: bad shape");
    if ((uintptr_t)x % 16 || (uintptr_t)dy % 16)
        return set_error(PFB_E_ARG, "conv3x3_wgrad: buffers must be 16-byte aligned");
    if (workspace_bytes < conv3x3_wgrad_workspace(B, H, W, cx, cy))
        return set_error(PFB_E_ARG, "conv3x3_wgrad: workspace too small");
    ConvWgradArgs a;
    a.partial = workspace;
    a.W2 = W + 2;
    a.chunks = (H * (W + 2) + kWgKT - 1) / kWgKT;
    const long long items = (long long)B * a.chunks;
    if (items > 0x7FFFFFFFll) return set_error(PFB_E_ARG, "conv3x3_wgrad: bad shape");
    a.items = (int)items;
    // a run is no longer than half an image (a whole one below 512 positions)
    const int n = H * (W + 2), half = n > 448 ? n / (2 * kWgKT) : a.chunks;
    a.run = half < kWgRun ? half : kWgRun;
    int dev = 0, sms = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return set_error(PFB_E_CUDA, "conv3x3_wgrad: %s", cudaGetErrorString(e));
    const long long blocks = (long long)(workspace_bytes / ((size_t)(9 * cy * cx + cy) * sizeof(float)));
    long long g = sms;
    if (g > blocks) g = blocks;
    if (g > items) g = items;
    const int grid = (int)g;
    const bf16* xb = static_cast<const bf16*>(x);
    const bf16* yb = static_cast<const bf16*>(dy);
    if (cx == 16 && cy == 32)
        e = launch_wgrad<16, 32>(a, xb, yb, B, H, W, grid, s);
    else if (cx == 32 && cy == 32)
        e = launch_wgrad<32, 32>(a, xb, yb, B, H, W, grid, s);
    else if (cx == 32 && cy == 16)
        e = launch_wgrad<32, 16>(a, xb, yb, B, H, W, grid, s);
    else if (cx == 16 && cy == 16)
        e = launch_wgrad<16, 16>(a, xb, yb, B, H, W, grid, s);
    else
        return set_error(PFB_E_CONFIG, "conv3x3_wgrad: channels %d, %d not built", cx, cy);
    if (e != cudaSuccess) return set_error(PFB_E_CUDA, "conv3x3_wgrad: %s", cudaGetErrorString(e));
    launch_wgrad_reduce(workspace, grid, cx, cy, dw, db, s);
    e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(PFB_E_CUDA, "wgrad reduce: %s", cudaGetErrorString(e));
    return PFB_OK;
}

int conv3x3_pack_many(const ConvPackJob* jobs, int n, cudaStream_t s) {
    PackJobs J;
    if (!jobs || n < 1 || n > 16) return set_error(PFB_E_ARG, "conv3x3_pack: bad job list");
    int most = 0;
    for (int k = 0; k < n; ++k) {
        const ConvPackJob& j = jobs[k];
        if (!j.w || !j.packed) return set_error(PFB_E_ARG, "conv3x3_pack: null buffer");
        if (j.cin % 8 || j.cout % 8 || j.cin <= 0 || j.cout <= 0)
            return set_error(PFB_E_ARG, "conv3x3_pack: channels must be multiples of 8");
        J.job[k] = j;
        most = most > 9 * j.cin * j.cout ? most : 9 * j.cin * j.cout;
    }
    k_pack_weights<<<dim3((unsigned)((most + 255) / 256), (unsigned)n), 256, 0, s>>>(J);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(PFB_E_CUDA, "conv3x3_pack: %s", cudaGetErrorString(e));
    return PFB_OK;
}

int conv3x3_pack(const float* w, void* packed, int cin, int cout, int transpose, cudaStream_t s) {
    const ConvPackJob job{w, packed, cin, cout, transpose ? 1 : 0};
    return conv3x3_pack_many(&job, 1, s);
}

int conv_read_status(unsigned* out, int clear) {
    unsigned v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_conv_status, sizeof(v));
    if (e != cudaSuccess) return set_error(PFB_E_CUDA, "conv status: %s", cudaGetErrorString(e));
    if (clear) {
        const unsigned z = 0;
        e = cudaMemcpyToSymbol(g_conv_status, &z, sizeof(z));
        if (e != cudaSuccess) return set_error(PFB_E_CUDA, "conv status: %s", cudaGetErrorString(e));
    }
    if (out) *out = v;
    return PFB_OK;
}

}  // namespace pfb

// ---- C ABI (include/pfb200_surrogate.h) ----------------------------------------

extern "C" {

int pfb_conv3x3_forward(const void* x, void* y, float* y_f32, const void* w_packed,
                        const float* bias, const void* gate, int batch, int H, int W, int cin,
                        int cout, int relu, void* stream) {
    pfb::clear_error();
    return pfb::conv3x3_fwd(x, y, y_f32, w_packed, bias, gate, batch, H, W, cin, cout, relu,
                            static_cast<cudaStream_t>(stream));
}

int pfb_conv3x3_pack(const float* w_oihw, void* w_packed, int cin, int cout, int transpose,
                     void* stream) {
    pfb::clear_error();
    return pfb::conv3x3_pack(w_oihw, w_packed, cin, cout, transpose,
                             static_cast<cudaStream_t>(stream));
}

size_t pfb_conv3x3_wgrad_workspace(int batch, int H, int W, int cx, int cy) {
    return pfb::conv3x3_wgrad_workspace(batch, H, W, cx, cy);
}

int pfb_conv3x3_wgrad(const void* x, const void* dy, float* workspace, size_t workspace_bytes,
                      float* dw_oihw, float* db, int batch, int H, int W, int cx, int cy,
                      void* stream) {
    pfb::clear_error();
    // the split follows the stated size, not what the caller has to spare, so
    // that the result does not depend on it
    const size_t need = pfb::conv3x3_wgrad_workspace(batch, H, W, cx, cy);
    return pfb::conv3x3_wgrad(x, dy, workspace, workspace_bytes < need ? workspace_bytes : need,
                              dw_oihw, db, batch, H, W, cx, cy, static_cast<cudaStream_t>(stream));
}

int pfb_conv_status(unsigned* out, int clear) { return pfb::conv_read_status(out, clear); }

int pfb_conv_set_pipeline(int mode) {
    pfb::clear_error();
    if (mode < 0 || mode > 2) return pfb::set_error(PFB_E_ARG, "conv pipeline mode %d not in 0..2", mode);
    pfb::g_conv_pipeline = mode;
    return PFB_OK;
}

}  // extern "C"

// ---- weight gradient without caller workspace -----------------------------------
//
// Some callers cannot hand this library device memory for scratch: hosts
// whose device memory is owned by their own pool allocator (a training
// framework's caching allocator, a serving engine's preallocated arena) and
// that forbid a raw cudaMalloc, which would take memory outside their budget
// and, being synchronizing, stall their streams. For them the weight gradient
// keeps its partial sums in this fixed array instead, which every GPU that
// loads the library holds until the process exits. Calls that overlap on the
// GPU (two streams, or two host threads) share the array and race.

using namespace pfb;

namespace {

constexpr size_t kNoAllocScratchBytes = (size_t)4 << 20;  // 4 MiB per device
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) float g_wgrad_scratch[kNoAllocScratchBytes / sizeof(float)];

std::mutex g_scratch_mutex;
float* g_scratch_ptr[kNoAllocMaxDevices] = {};

// Device address of g_wgrad_scratch on the current device, looked up once per
// device (the host-side name of the array is not a device address). The
// address belongs to the device's primary context: a cudaDeviceReset in the
// same process makes the cached value stale, so such hosts must not call the
// entry point after a reset.
int scratch_on_current_device(float** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(PFB_E_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kNoAllocMaxDevices)
        return set_error(PFB_E_CONFIG, "device %d beyond the %d supported", dev, kNoAllocMaxDevices);
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_wgrad_scratch);
        if (e != cudaSuccess || !p)
            return set_error(PFB_E_CUDA, "scratch address: %s", cudaGetErrorString(e));
        g_scratch_ptr[dev] = static_cast<float*>(p);
    }
    *out = g_scratch_ptr[dev];
    return PFB_OK;
}

}  // namespace

extern "C" int pfb_conv3x3_wgrad_noalloc(const void* x, const void* dy, float* dw_oihw, float* db,
                                         int batch, int H, int W, int cx, int cy, void* stream) {
    clear_error();
    if (!x || !dy || !dw_oihw) return set_error(PFB_E_ARG, "conv3x3_wgrad_noalloc: null buffer");
    if (!shape_ok(batch, H, W))
        return set_error(PFB_E_ARG, "conv3x3_wgrad_noalloc: bad shape %dx%dx%d", batch, H, W);
    if (cx <= 0 || cy <= 0 || cx > 64 || cy > 64)
        return set_error(PFB_E_CONFIG, "conv3x3_wgrad_noalloc: channels %d, %d not built", cx, cy);
    const size_t need = conv3x3_wgrad_workspace(batch, H, W, cx, cy);
    if (need > kNoAllocScratchBytes)
        return set_error(PFB_E_ARG,
                         "conv3x3_wgrad_noalloc: %d images of %dx%d with %d -> %d channels need "
                         "%zu bytes of scratch, above its fixed %zu bytes (split the batch, or "
                         "use pfb_conv3x3_wgrad with a workspace)",
                         batch, H, W, cx, cy, need, kNoAllocScratchBytes);
    float* scratch = nullptr;
    const int rc = scratch_on_current_device(&scratch);
    if (rc) return rc;
    // every CTA overwrites its whole block of partial sums before the reduction
    // reads it (with NaN when its MMA wait gave up), so nothing in the shared
    // array has to start at zero
    return conv3x3_wgrad(x, dy, scratch, need, dw_oihw, db, batch, H, W, cx, cy,
                         static_cast<cudaStream_t>(stream));
}
