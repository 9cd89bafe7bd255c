// Quantized Linear forward for f32 activations on the 5th-generation tensor cores, persistent, sm_100a only.
//
//   y[m,n] = epi( scale[n] * sum_k q[n,k] * x[m,k] + bias[n] )       (quantize.rs:463-476)
//
// x is split in the kernel into hi = bf16(x) and lo = bf16(x - hi); both meet the same widened codes (exact in bf16) in
// one f32 accumulator, so the sum carries ~16 significand bits of x.
//
// What bounds these layers is not the tensor pipe but everything around it: with a few hundred input features a tile is
// a handful of MMAs between a prologue and an epilogue of 32 to 64 KB, and at 4096 tokens a vocabulary head is one
// long stream of output.  One CTA per tile with all tensor memory to itself (gemm_tcgen05_kernels.cuh) spends its time
// in launch, first loads and epilogue, one after the other, and needs a pass over x beforehand.  Hence:
//  - one CTA per SM walks a contiguous range of output tiles, channel tiles fastest; the accumulators are double
//    buffered, so the stores of a tile run under the loads, widening and MMAs of the next;
//  - the activations of a token tile are read as f32, split and swizzled into shared memory by the epilogue warps and
//    stay there for all channel tiles of the range while K fits (up to 768 features with 64-token
//    tiles, 384 with 128); wider layers run them through the same slots as a ring.  No pass over x, no copy of it;
//  - a warp stores its 32 accumulator lanes as 32 consecutive channels of one token straight from registers: 128-byte
//    segments whatever the alignment of the output row, no staging tile and no barrier.
//
// Roles: warp 0 TMA producer of the codes, warp 1 tensor-memory allocation and MMA issue, warps 2-9 widen codes into
// tensor memory (two groups of one warp per lane quadrant, taking turns by stage: one group is bound by the latency of its
// own chain, ~0.4 us a block), warps 10-17 load activations and store results.  Hand-offs by mbarrier, every
// wait bounded (timeout code 5); a wait that runs out raises the CTA's abort flag and every role leaves.
//
// Device code only: also compiles against the CUDA stand-in of the CPU tests (tests/cpu_emu/).
#pragma once

#include "../../include/shrewq.h"
#include "dests.cuh"
#include "ptx_small.cuh"
#include "ptx_tcgen05.cuh"
#include "tcgen05_common.cuh"

namespace shrewq {
namespace {

constexpr int kF32Threads = 18 * 32;
constexpr int kF32Chan = 128;  // output channels per tile = tensor-memory lanes
constexpr int kF32BlockK = 64;

// XKB: kilobytes of shared memory for activations.  The rest of 224 KB are stages for codes, which come from L2 while the
// results load it: four stages are one tile of 256 features ahead, twelve are three (gemm_tcgen05_f32.cu has what each gives).
template <int TOK, int XKB>
struct F32Cfg {
    static_assert(TOK == 64 || TOK == 128, "two accumulators of TOK columns below the operand columns");
    static constexpr int kXTile = TOK * kF32BlockK * 2;  // one bf16 tile of a 64-wide block
    static constexpr int kXSlot = 2 * kXTile;            // hi, then lo
    static constexpr int kXSlots = XKB * 1024 / kXSlot;
    static constexpr int kWBytes = kF32Chan * kF32BlockK;
    static constexpr int kWStages = (224 - XKB) * 1024 / kWBytes;
    static_assert(kWStages % 2 == 0, "a converter group owns every second stage");
    static constexpr int kABase = 256;                   // tensor-memory columns of the widened codes
    static constexpr int kACols = kF32BlockK / 2;
    static constexpr int kAStages = (512 - kABase) / kACols;
    static constexpr int kWOff = kXSlots * kXSlot;
    static constexpr int kBarOff = kWOff + kWStages * kWBytes;
    static constexpr int kSmemBytes = kBarOff + 1024 + 1024 /* alignment slack */;
    static constexpr int kUnits = TOK * 8 / 256;         // 8-float pieces per loader thread and block
    static constexpr int kBatch = 4 / kUnits;            // blocks loaded together: 32 floats in registers
    // barriers (8 bytes each)
    static constexpr uint32_t kWFull = 0, kWEmpty = kWFull + 8 * kWStages, kAReady = kWEmpty + 8 * kWStages,
                              kAEmpty = kAReady + 8 * kAStages, kXReady = kAEmpty + 8 * kAStages,
                              kXEmpty = kXReady + 8 * kXSlots, kAccFull = kXEmpty + 8 * kXSlots, kAccEmpty = kAccFull + 16;
    static_assert(kAccEmpty + 16 <= 512, "barriers fit below the control block");
    // above kChain features a 64-token tile sums the halves of K in two accumulators and adds them in the epilogue, as
    // the two-way split along K of gemm_tcgen05_launch.cuh would (an accumulator loses up to an ulp per MMA)
    static constexpr int kParts = TOK == 64 ? 2 : 1;
    static constexpr int kChain = 512;
    static_assert(2 * kParts * TOK <= kABase && kSmemBytes <= 227 * 1024, "tensor memory, shared memory");
};

__device__ __forceinline__ bool f32_wait(uint32_t bar, uint32_t parity, Ctl *ctl, DeviceStatus *st, uint32_t role, uint32_t stage) {
    return mbar_wait_c<5>(bar, parity, ctl, st, role, stage);
}
__device__ __forceinline__ bool f32_wait_warp(uint32_t bar, uint32_t parity, Ctl *ctl, DeviceStatus *st, uint32_t role,
                                              uint32_t stage) {
    return mbar_wait_warp_c<5>(bar, parity, ctl, st, role, stage);
}

// resident: the activations of a token tile stay in shared memory for all its channel tiles (K <= kXSlots * 64).
// x 16-byte aligned, K a multiple of 16; y any f32 rows of stride ldy.
template <int TOK, int XKB>
__global__ void __launch_bounds__(kF32Threads, 1)
linear_i8_tcgen05_f32_kernel(const __grid_constant__ CUtensorMap tmap_w, const float *__restrict__ scales,
                             const float *__restrict__ bias, const float *__restrict__ x, float *__restrict__ y, int M, int N,
                             int K, size_t ldy, int epilogue, int n_tiles, int tiles, int resident, DeviceStatus *status) {
    using C = F32Cfg<TOK, XKB>;
    pdl_launch_dependents();
    SHREWQ_DYNAMIC_SMEM(uint8_t, smem_raw);
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    Ctl *ctl = reinterpret_cast<Ctl *>(smem + C::kBarOff + 512);
    const uint32_t smem_base = smem_u32(smem), bars = smem_base + C::kBarOff;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int begin = (int)((long long)tiles * blockIdx.x / gridDim.x), end = (int)((long long)tiles * (blockIdx.x + 1) / gridDim.x);
    const int nkb = (K + kF32BlockK - 1) / kF32BlockK;
    const int kb_part = C::kParts == 2 && K > C::kChain ? (nkb + 1) / 2 : nkb;  // the block the second accumulator begins with

    if (threadIdx.x == 0) {
        ctl->abort_flag = 0;
        ctl->tmem_base = 0;
        for (int s = 0; s < C::kWStages; ++s) {
            mbar_init(bars + C::kWFull + 8 * s, 1);
            mbar_init(bars + C::kWEmpty + 8 * s, 4);
        }
        for (int s = 0; s < C::kAStages; ++s) {
            mbar_init(bars + C::kAReady + 8 * s, 4);
            mbar_init(bars + C::kAEmpty + 8 * s, 1);
        }
        for (int s = 0; s < C::kXSlots; ++s) {
            mbar_init(bars + C::kXReady + 8 * s, 8);
            mbar_init(bars + C::kXEmpty + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(bars + C::kAccFull + 8 * s, 1);
            mbar_init(bars + C::kAccEmpty + 8 * s, 4);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        tc_alloc_512(smem_u32(&ctl->tmem_base));
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;

    if (warp == 0) {
        // ---------------- codes: one 128 x 64 box per block (weights never depend on an earlier kernel) ----------------
        if (elect_one()) {
            int it = 0;
            bool ok = true;
            for (int tile = begin; tile < end && ok; ++tile) {
                const int n0 = (tile % n_tiles) * kF32Chan;
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const int s = it % C::kWStages;
                    // the converters free this many stages before they need the first MMA, which needs activations
                    if (it == C::kWStages + C::kAStages) pdl_wait();
                    if (it >= C::kWStages) ok = f32_wait(bars + C::kWEmpty + 8 * s, ((it / C::kWStages) - 1) & 1, ctl, status, 0, s);
                    if (!ok) break;
                    mbar_expect_tx(bars + C::kWFull + 8 * s, C::kWBytes);
                    tma_load_2d(smem_base + C::kWOff + s * C::kWBytes, &tmap_w, kb * kF32BlockK, n0, bars + C::kWFull + 8 * s);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issue ----------------
        if (elect_one()) {
            // D=f32, A=bf16 (K-major, tensor memory), B=bf16 (K-major), M=128, N=TOK
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TOK >> 3) << 17) | ((uint32_t)(kF32Chan >> 4) << 24);
            pdl_wait();  // the first activations come after it: a time limit must not run while the previous kernel does
            int it = 0, li = 0, visit_load = 0;  // visit_load: index of the first activation block of this token tile
            bool ok = true;
            for (int tile = begin; tile < end && ok; ++tile, ++li) {
                const int buf = li & 1;
                const bool last_of_visit = !resident || tile + 1 == end || (tile + 1) % n_tiles == 0;
                if (li >= 2) ok = f32_wait(bars + C::kAccEmpty + 8 * buf, ((li >> 1) - 1) & 1, ctl, status, 1, buf);
                for (int kb = 0; kb < nkb && ok; ++kb, ++it) {
                    const int as = it % C::kAStages, xl = visit_load + kb, xs = xl % C::kXSlots;
                    ok = f32_wait(bars + C::kAReady + 8 * as, (it / C::kAStages) & 1, ctl, status, 2, as) &&
                         f32_wait(bars + C::kXReady + 8 * xs, (xl / C::kXSlots) & 1, ctl, status, 3, xs);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t bdesc = make_b_desc(smem_base + xs * C::kXSlot);
                    const uint32_t d = tmem + (buf * C::kParts + (kb >= kb_part ? 1 : 0)) * TOK;
                    const bool fresh = kb == 0 || kb == kb_part;
#pragma unroll
                    for (int j = 0; j < kF32BlockK / 16; ++j) {
                        const uint32_t a = tmem + C::kABase + as * C::kACols + j * 8;
                        tc_mma_ts(d, a, bdesc + (uint64_t)((j * 32) >> 4), idesc, (!fresh || j > 0) ? 1u : 0u);
                        tc_mma_ts(d, a, bdesc + (uint64_t)((C::kXTile + j * 32) >> 4), idesc, 1u);
                    }
                    tc_commit(bars + C::kAEmpty + 8 * as);
                    if (last_of_visit) tc_commit(bars + C::kXEmpty + 8 * xs);
                }
                if (ok) tc_commit(bars + C::kAccFull + 8 * buf);
                if (last_of_visit) visit_load += nkb;
            }
        }
        __syncwarp();
    } else if (warp < 10) {
        // ---------------- codes -> bf16 in tensor memory: one row per thread ----------------
        const int quad = warp & 3, row = quad * 32 + lane, swz = (row >> 1) & 3;
        const uint32_t a0 = tmem + ((uint32_t)(quad * 32) << 16) + C::kABase;
        const int total = (end - begin) * nkb;
        for (int it = (warp - 2) >> 2; it < total; it += 2) {
            const int s = it % C::kWStages, as = it % C::kAStages;
            if (!f32_wait_warp(bars + C::kWFull + 8 * s, (it / C::kWStages) & 1, ctl, status, 4, s)) break;
            uint32_t packed[32];
            convert_row64(smem + C::kWOff + s * C::kWBytes + row * kF32BlockK, swz, packed);
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + C::kWEmpty + 8 * s);
            // as far as the free operand columns reach the codes are widened while the previous kernel still runs
            if (it == C::kAStages || it == C::kAStages + 1) pdl_wait();
            if (it >= C::kAStages && !f32_wait_warp(bars + C::kAEmpty + 8 * as, ((it / C::kAStages) - 1) & 1, ctl, status, 5, as)) break;
            tc_fence_after();
            tc_st32(a0 + as * C::kACols, packed);
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + C::kAReady + 8 * as);
        }
    } else {
        // ---------------- activations in, results out ----------------
        const int ew = warp - 10, group = ew >> 2, quad = warp & 3, et = ew * 32 + lane;
        const bool relu = (epilogue & 0xFF) == SHREWQ_EPILOGUE_RELU;
        // x may be the previous kernel's output, and y may still be read by it
        pdl_wait();
        int li = 0, xl0 = 0;
        bool ok = true;
        for (int tile = begin; tile < end && ok; ++tile, ++li) {
            const int m0 = (tile / n_tiles) * TOK, n = (tile % n_tiles) * kF32Chan + quad * 32 + lane;
            if (!resident || tile == begin || tile % n_tiles == 0) {
                for (int kb0 = 0; kb0 < nkb && ok; kb0 += C::kBatch) {
                    float v[C::kBatch][C::kUnits][8];
#pragma unroll
                    for (int b = 0; b < C::kBatch; ++b)
#pragma unroll
                        for (int u = 0; u < C::kUnits; ++u) {
                            const int unit = et + u * 256, m = m0 + (unit >> 3), k = (kb0 + b) * kF32BlockK + (unit & 7) * 8;
                            float4 lo4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi4 = lo4;
                            if (m < M && k < K) {
                                const float4 *p = reinterpret_cast<const float4 *>(x + (size_t)m * K + k);
                                lo4 = __ldg(p);
                                hi4 = __ldg(p + 1);
                            }
                            v[b][u][0] = lo4.x; v[b][u][1] = lo4.y; v[b][u][2] = lo4.z; v[b][u][3] = lo4.w;
                            v[b][u][4] = hi4.x; v[b][u][5] = hi4.y; v[b][u][6] = hi4.z; v[b][u][7] = hi4.w;
                        }
#pragma unroll
                    for (int b = 0; b < C::kBatch; ++b) {
                        if (kb0 + b >= nkb || !ok) continue;
                        const int xl = xl0 + kb0 + b, xs = xl % C::kXSlots;
                        if (xl >= C::kXSlots) ok = f32_wait_warp(bars + C::kXEmpty + 8 * xs, ((xl / C::kXSlots) - 1) & 1, ctl, status, 6, xs);
                        if (!ok) continue;
#pragma unroll
                        for (int u = 0; u < C::kUnits; ++u) {
                            const int unit = et + u * 256, r = unit >> 3, c = unit & 7;
                            uint32_t h[4], l[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const float v0 = v[b][u][2 * e], v1 = v[b][u][2 * e + 1];
                                h[e] = pack_bf16x2_rn(v1, v0);
                                l[e] = pack_bf16x2_rn(v1 - __uint_as_float(h[e] & 0xFFFF0000u), v0 - __uint_as_float(h[e] << 16));
                            }
                            // 128-byte swizzle: 16-byte piece c of row r sits at piece c ^ (r & 7)
                            uint8_t *dst = smem + xs * C::kXSlot + r * 128 + ((c ^ (r & 7)) << 4);
                            *reinterpret_cast<uint4 *>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
                            *reinterpret_cast<uint4 *>(dst + C::kXTile) = make_uint4(l[0], l[1], l[2], l[3]);
                        }
                        fence_proxy_async_smem();  // the MMA reads the tile through the async proxy
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bars + C::kXReady + 8 * xs);
                    }
                }
                xl0 += nkb;
            }
            // the two groups of four warps take turns by tile (and accumulator), so that the stores of one run under the waits and
            // the tensor-memory loads of the other (4096 x 50257 x 256: 284 -> 275 us)
            if ((li & 1) != group) continue;
            const bool n_ok = n < N;
            const float sc = n_ok ? scales[n] : 0.0f, bs = (n_ok && bias) ? bias[n] : 0.0f;
            const int buf = li & 1;
            if (ok) ok = f32_wait_warp(bars + C::kAccFull + 8 * buf, (li >> 1) & 1, ctl, status, 7, buf);
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < TOK / 32; ++c) {
                const int col = c * 32;
                uint32_t r[32];
                const uint32_t acc = tmem + ((uint32_t)(quad * 32) << 16) + buf * C::kParts * TOK + col;
                tc_ld32(acc, r);
                if constexpr (C::kParts == 2) {
                    if (kb_part < nkb) {
                        uint32_t r2[32];
                        tc_ld32(acc + TOK, r2);
                        tc_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + __uint_as_float(r2[i]));
                    }
                }
                tc_wait_ld();
                if (c == TOK / 32 - 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bars + C::kAccEmpty + 8 * buf);
                }
                if (n_ok) {
                    float *p = y + (size_t)(m0 + col) * ldy + n;
                    const int rows = M - (m0 + col) < 32 ? M - (m0 + col) : 32;
                    if (rows == 32) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            float o = __uint_as_float(r[i]) * sc + bs;
                            if (relu) o = fmaxf(o, 0.0f);
                            *p = o;
                            p += ldy;
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            float o = __uint_as_float(r[i]) * sc + bs;
                            if (relu) o = fmaxf(o, 0.0f);
                            if (i < rows) *p = o;
                            p += ldy;
                        }
                    }
                }
                __syncwarp();
            }
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        if (ctl->abort_flag) {
            // give in-flight copies / MMAs a bounded moment to land before tensor memory is released
            for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        }
        tc_fence_after();
        __syncwarp();
        tc_dealloc_512(tmem);
    }
}

}  // namespace
}  // namespace shrewq
