// Weight-only INT8 forward for 1..32 tokens: the weights streamed through a shared-memory ring by bulk copies
// (TMA, 1-D) and multiplied on warp-level MMA, sm_100a.
//
//   y[m,n] = scale[n] * sum_k q[n,k] * x[m,k] + bias[n]        (quantize.rs:463-476; the codes are exact in bf16,
// the products exact in the f32 accumulator, and one multiply applies the scale)
//
// HBM-bound: the INT8 matrix, N*K bytes, is read exactly once and a 4096 x 4096 layer is 2.6 us of stream, so
// what matters is that bytes are requested early, that many are in flight, and that the arithmetic per byte is
// small and independent of the batch.
//
//  - The grid is what fits the GPU at once and a CTA walks over blocks of 16 rows of W (gated: the gate rows and the up rows
//    of 8 channels), so that the producer runs on into the next block while this one is multiplied and reduced: gate/up
//    11008 x 4096 at 8 tokens 29.7 -> 21.1 us, 4096 x 11008 15.9 -> 12.8 us against one block per CTA.  A producer warp asks the copy
//    engine for them in stages of 16 rows x 2 KB, one bulk copy per row and stage, into a ring of two or three stages
//    (full / empty mbarriers).  Two stages are a whole K = 4096 row block, requested in the kernel's first hundred
//    cycles; no load instruction waits in a register scoreboard and the bytes in flight per SM (about 200 KB) do not
//    depend on how many warps are resident.
//  - Eight consumer warps split every stage by k (four 64-wide k-blocks each).  The weights are the A operand of
//    mma.sync.m16n8k16 (16 rows x 16 k), the activations the B operand (16 k x 8 tokens): widening a code to
//    bf16 costs 2.25 instructions whatever the batch (widen_bf16.cuh), and one to four MMAs per step cover 8 to 32 tokens with
//    the same converted fragment.  Lane (g = lane / 4, t = lane % 4) reads the 16 codes [16t, 16t + 16) of
//    rows g and g + 8 of the k-block and the 16 activations of the same k for tokens g (+ 8, 16, 24); MMA
//    step j uses codes and activations 4j .. 4j+3 of those runs for A and B alike (a dot product does not care
//    about the order of k).  Rows are 2112 bytes apart in shared memory, so the 16-byte reads of a quarter warp
//    fall into distinct banks.  Activations come straight from global memory (L1 keeps them: every CTA of
//    an SM reads the same few KB), requested half a k-block ahead and earlier.
//  - The eight warps' accumulators meet in shared memory; the 256 consumer threads apply scale, bias and the
//    epilogue to the 128 (gated: 64) x NT outputs and store to the local and the peer destinations.
//
// Programmatic dependent launch: the kernel lets its successor start at once, and its producer requests WEIGHTS
// without waiting for the predecessor (weights never depend on an earlier kernel); the consumers wait for it
// before they read activations or write outputs.  A chain of small-batch forwards thus keeps the weight stream
// going across kernel boundaries.  Launched without the attribute the two instructions do nothing.
//
// Every wait is bounded, and none that depends on the consumers starts before the previous kernel has completed.  A wait that
// runs out records itself in DeviceStatus (timeout code 4) and the CTA leaves without writing.
//
// Device code only (PTX behind ptx_small.cuh / ptx_tcgen05.cuh): also compiles against the CUDA stand-in of the
// CPU tests (tests/cpu_emu/).
#pragma once

#include "../../include/shrewq.h"
#include "dests.cuh"
#include "ptx_small.cuh"
#include "ptx_tcgen05.cuh"
#include "widen_bf16.cuh"

namespace shrewq {
namespace {

// W consumer warps (8 or 16) + one producer warp (warp W)
constexpr int kRingRows = 16;                          // rows of W per CTA
#ifndef SHREWQ_RING_SPIN_LIMIT
#define SHREWQ_RING_SPIN_LIMIT (1u << 22)
#endif
constexpr uint32_t kRingSpinLimit = SHREWQ_RING_SPIN_LIMIT;  // bounded wait: a few tenths of a second with the pauses
constexpr unsigned int kTimeoutRing = 4;               // DeviceStatus::timeout_flag of this kernel

// KC: bytes (= codes) of k per row and stage, i.e. the size of one bulk copy.  The copy engine's cost is per copy:
// measured on a B200 at 4096 x 4096, batch 1, the kernel takes 9.0 us with 512-byte, 7.3 us with 1 KB and 6.8 us
// with 2 KB copies.  Rows are KC + 64 bytes apart in shared memory, so the 16-byte reads of a quarter warp (rows
// g, g + 1; four 16-byte columns) fall into distinct banks.  Three stages of 2 KB rows are 99 KB: two CTAs per SM
// with ~200 KB of weights in flight, the choice for grids of up to two CTAs per SM; grids of several waves take two
// stages (66 KB, three CTAs per SM: the same bytes in flight, half as many more warps to widen codes).
constexpr int kRingMaxStages = 8;
template <int KC, int STAGES = (KC >= 2048 ? 3 : KC >= 1024 ? 5 : 8)>
struct RingCfg {
    static constexpr int kPitch = KC + 64;
    static constexpr int kStageBytes = kRingRows * kPitch;
    static constexpr int kStages = STAGES;
    static constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + 2 * kRingMaxStages * 8;
};
constexpr int kRingKC = 2048;     // what the launcher instantiates
constexpr int kRingConsumers = 8;

template <typename YT>
__device__ __forceinline__ void ring_store(YT *p, float v);
template <>
__device__ __forceinline__ void ring_store<float>(float *p, float v) { *p = v; }
template <>
__device__ __forceinline__ void ring_store<__nv_bfloat16>(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }

__device__ __forceinline__ bool ring_wait(uint32_t bar, uint32_t parity, DeviceStatus *st, uint32_t role, uint32_t stage) {
    for (uint32_t i = 0; i < kRingSpinLimit; ++i) {
        if (mbar_try(bar, parity)) return true;
        if (i > 256) __nanosleep(64);
    }
    if (atomicCAS(&st->timeout_flag, 0u, kTimeoutRing) == 0u) {
        st->where = (blockIdx.x << 8) | role;
        st->stage = stage;
        st->parity = parity;
    }
    return false;
}

// NT: token blocks of 8 (M <= 8 * NT).  K a multiple of 64; q, q_up and x 16-byte aligned.
// CHAINS: accumulators of a warp for one output, taking turns by MMA step (two halve the chain of dependent MMAs and of f32
// roundings).  One chain, with the epilogue rounding as gemv_mma_kernels.cuh's does (its compiler fuses scale and bias from 17
// tokens on), gives that kernel's results bit for bit.
// GATED: rows 0..7 of the CTA are gate rows, rows 8..15 the up rows of the same 8 channels.
template <int NT, int KC, int W, typename YT, bool GATED, int STAGES = RingCfg<KC>::kStages, int CHAINS = 2>
__global__ void __launch_bounds__((W + 1) * 32, NT >= 3 ? 2 : 3)
gemv_i8_ring_kernel(const int8_t *__restrict__ q, const float *__restrict__ scales, const float *__restrict__ bias,
                    const int8_t *__restrict__ q_up, const float *__restrict__ scales_up,
                    const float *__restrict__ bias_up, const uint16_t *__restrict__ x, YT *__restrict__ y, Dests extra,
                    int M, int N, int K, size_t ldy, int epilogue, DeviceStatus *status) {
    using C = RingCfg<KC, STAGES>;
    static_assert(KC / 64 >= W, "every consumer warp needs a k-block in every full stage");
    constexpr int kRingWarps = W;
    constexpr int NCH = GATED ? kRingRows / 2 : kRingRows;  // output channels per CTA
    SHREWQ_DYNAMIC_SMEM(uint8_t, smem);
    __shared__ float s_red[kRingWarps][NT][4][32];
    __shared__ volatile int s_bad;
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int S = C::kStages;
    constexpr uint32_t stage_bytes = C::kStageBytes;
    const uint32_t ring_u32 = smem_u32(smem);
    const uint32_t full_u32 = ring_u32 + S * stage_bytes;
    const uint32_t empty_u32 = full_u32 + kRingMaxStages * 8;
    const int nstages = (K + KC - 1) / KC;
    const int nblocks = (N + NCH - 1) / NCH;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(full_u32 + s * 8, 1);
            mbar_init(empty_u32 + s * 8, kRingWarps);
        }
        mbar_fence_init();
        s_bad = 0;
    }
    __syncthreads();

    bool ok = true;
    if (warp == kRingWarps) {
        // ---- producer: lane r brings row r of every stage ----
        int it = 0;
        for (int blk = blockIdx.x; blk < nblocks && ok; blk += gridDim.x) {
            const int8_t *src = nullptr;
            if (lane < kRingRows) {
                int n = blk * NCH + (GATED ? (lane & 7) : lane);
                n = n < N ? n : N - 1;  // clamp: duplicates are computed and dropped
                src = ((GATED && lane >= 8) ? q_up : q) + (size_t)n * K;
            }
            for (int s = 0; s < nstages; ++s, ++it) {
                const int slot = it % S;
                if (it >= S) {
                    // the consumers free a slot only after their own wait for the previous kernel, however long that takes
                    // (a barrier between GPUs tolerates a late peer): the time limit starts when it has completed
                    if (it == S) pdl_wait();
                    int good = 1;
                    if (lane == 0) good = ring_wait(empty_u32 + slot * 8, ((it / S) - 1) & 1, status, 1, s) ? 1 : 0;
                    ok = __shfl_sync(0xFFFFFFFFu, good, 0) != 0;
                    if (!ok) break;
                }
                const int k0 = s * KC;
                const uint32_t bytes = (uint32_t)(K - k0 < KC ? K - k0 : KC);
                if (lane == 0) mbar_expect_tx(full_u32 + slot * 8, bytes * kRingRows);
                __syncwarp();
                if (lane < kRingRows) bulk_load_1d(ring_u32 + slot * stage_bytes + lane * C::kPitch, src + k0, bytes, full_u32 + slot * 8);
            }
        }
        return;
    }

    // ---- consumers: warp w takes the k-blocks w, w + W, ... of every stage ----
    const int g = lane >> 2, t = lane & 3;
    // the activations may be the previous kernel's output, which may also still read our output buffer
    pdl_wait();
    const uint16_t *xrow[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) xrow[nt] = (8 * nt + g) < M ? x + (size_t)(8 * nt + g) * K + 16 * t : nullptr;

    // the activations of one k-block: half h of its 16-byte pieces is read again as soon as MMA steps 2h and 2h + 1 have used it,
    // so the next k-block's are on their way without a second set of registers
    uint4 xc[NT][2];
#define SHREWQ_RING_LOAD_X(koff, h)                                                               \
    _Pragma("unroll") for (int nt = 0; nt < NT; ++nt) {                                           \
        xc[nt][h] = make_uint4(0, 0, 0, 0);                                                       \
        if (xrow[nt] && (koff) < K) xc[nt][h] = __ldg(reinterpret_cast<const uint4 *>(xrow[nt] + (koff)) + (h)); \
    }
    SHREWQ_RING_LOAD_X(warp * 64, 0);
    SHREWQ_RING_LOAD_X(warp * 64, 1);
    int it = 0;
    for (int blk = blockIdx.x; blk < nblocks; blk += gridDim.x) {
        float acc[CHAINS][NT][4];
#pragma unroll
        for (int h = 0; h < CHAINS; ++h)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[h][nt][r] = 0.0f;
        for (int s = 0; s < nstages && ok; ++s, ++it) {
            const int slot = it % S;
            int good = 1;
            if (lane == 0) good = ring_wait(full_u32 + slot * 8, (it / S) & 1, status, 2 + warp, s) ? 1 : 0;
            ok = __shfl_sync(0xFFFFFFFFu, good, 0) != 0;
            // every lane observes the completed phase itself: its own acquire on the bytes the copies wrote
            if (ok) ok = __all_sync(0xFFFFFFFFu, mbar_try(full_u32 + slot * 8, (it / S) & 1) ? 1 : 0) != 0;
            if (!ok) break;
            const uint8_t *stage = smem + (size_t)slot * stage_bytes;
            const int k_end = K - s * KC < KC ? K - s * KC : KC;
            for (int kin = warp * 64; kin < k_end; kin += kRingWarps * 64) {
                // this warp's next k-block (after the last one: the first of the next row block), while this one is multiplied
                const int after = s * KC + kin + kRingWarps * 64, knext = after < K ? after : warp * 64;
                const uint8_t *wp = stage + (size_t)g * C::kPitch + kin + 16 * t;
                const uint4 wlo = *reinterpret_cast<const uint4 *>(wp);
                const uint4 whi = *reinterpret_cast<const uint4 *>(wp + 8 * C::kPitch);
                const uint32_t wl[4] = {wlo.x, wlo.y, wlo.z, wlo.w}, wh[4] = {whi.x, whi.y, whi.z, whi.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t a0, a1, a2, a3;
                    cvt_i8x4_bf16(wl[j], a0, a2);  // row g:     codes (4j, 4j+1) | (4j+2, 4j+3)
                    cvt_i8x4_bf16(wh[j], a1, a3);  // row g + 8
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const uint4 &xa = xc[nt][j >> 1];
                        const uint32_t b0 = (j & 1) ? xa.z : xa.x, b1 = (j & 1) ? xa.w : xa.y;
                        mma_bf16_16816(acc[j & (CHAINS - 1)][nt], a0, a1, a2, a3, b0, b1);
                    }
                    if (j & 1) SHREWQ_RING_LOAD_X(knext, j >> 1);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_u32 + slot * 8);  // this warp is done with the stage
        }
        if (!ok) s_bad = 1;  // a CTA with a wait that ran out still meets at the barriers; it writes nothing more
        if (blk != (int)blockIdx.x) named_bar_sync(1, kRingWarps * 32);  // the block before has been read out of s_red
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r) s_red[warp][nt][r][lane] = CHAINS == 2 ? acc[0][nt][r] + acc[CHAINS - 1][nt][r] : acc[0][nt][r];
        named_bar_sync(1, kRingWarps * 32);

        // accumulator element (lane, r) of block nt: row (lane / 4) + (r >= 2 ? 8 : 0), token 8 * nt + 2 * (lane % 4) + (r & 1)
        const int n0 = blk * NCH;
        if (!s_bad) {
            for (int i = threadIdx.x; i < NCH * 8 * NT; i += kRingWarps * 32) {
                const int c = i % NCH, m = i / NCH;
                const int n = n0 + c;
                if (m >= M || n >= N) continue;
                const int nt = m >> 3, mm = m & 7;
                const int ln = (c & 7) * 4 + (mm >> 1);
                float out;
                if constexpr (GATED) {
                    float gs = 0.0f, us = 0.0f;
#pragma unroll
                    for (int w = 0; w < kRingWarps; ++w) {
                        gs += s_red[w][nt][mm & 1][ln];
                        us += s_red[w][nt][2 + (mm & 1)][ln];
                    }
                    gs = __fadd_rn(__fmul_rn(gs, scales[n]), bias ? bias[n] : 0.0f);
                    us = __fadd_rn(__fmul_rn(us, scales_up[n]), bias_up ? bias_up[n] : 0.0f);
                    out = gs / (1.0f + __expf(-gs)) * us;
                } else {
                    float sum = 0.0f;
                    const int r = (mm & 1) + ((c & 8) ? 2 : 0);
#pragma unroll
                    for (int w = 0; w < kRingWarps; ++w) sum += s_red[w][nt][r][ln];
                    out = NT >= 3 ? __fmaf_rn(sum, scales[n], bias ? bias[n] : 0.0f) : __fadd_rn(__fmul_rn(sum, scales[n]), bias ? bias[n] : 0.0f);
                    if (epilogue == SHREWQ_EPILOGUE_RELU) out = fmaxf(out, 0.0f);
                }
                const size_t off = (size_t)m * ldy + n;
                ring_store<YT>(y + off, out);
                for (int d = 0; d < extra.n; ++d) ring_store<YT>(static_cast<YT *>(extra.p[d]) + off, out);
            }
        }
    }
#undef SHREWQ_RING_LOAD_X
}

}  // namespace
}  // namespace shrewq
