// Launcher of the persistent f32-activation forward (device code and its description: gemm_tcgen05_f32_kernels.cuh).
#include <cuda.h>

#include <atomic>

#include "common.cuh"
#include "gemm_tcgen05_f32_kernels.cuh"

namespace shrewq {
namespace {

template <int TOK, int XKB>
int launch_f32(shrewq_ctx *ctx, const ForwardArgs &a, const CUtensorMap &tw) {
    using C = F32Cfg<TOK, XKB>;
    auto kern = linear_i8_tcgen05_f32_kernel<TOK, XKB>;
    static std::atomic<unsigned long long> attr_done{0};  // per instantiation: bit d = device d has the attribute
    const int d = ctx->device;
    if (d < 0 || d >= 64 || !((attr_done.load(std::memory_order_acquire) >> d) & 1ull)) {
        SHREWQ_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
        if (d >= 0 && d < 64) attr_done.fetch_or(1ull << d, std::memory_order_release);
    }
    const int n_tiles = (int)((a.N + kF32Chan - 1) / kF32Chan), m_tiles = (int)((a.M + TOK - 1) / TOK);
    const int tiles = n_tiles * m_tiles;
    const int resident = a.K <= (size_t)C::kXSlots * kF32BlockK;
    const int grid = tiles < ctx->sm_count ? tiles : ctx->sm_count;
    SHREWQ_CUDA_TRY(ctx, launch_maybe_pdl(kern, dim3((unsigned)grid), dim3(kF32Threads), (size_t)C::kSmemBytes, ctx->stream, a.pdl, tw,
                                          a.scales, a.bias, static_cast<const float *>(a.x), static_cast<float *>(a.y), (int)a.M,
                                          (int)a.N, (int)a.K, a.ldy, a.epilogue, n_tiles, tiles, resident, ctx->dev_status));
    ctx->launches += 1;
    SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
    return SHREWQ_OK;
}

}  // namespace

bool tcgen05_f32_wins(const ForwardArgs &a, const Tuning &t) {
    const size_t n_tiles = (a.N + kF32Chan - 1) / kF32Chan, tiles = n_tiles * ((a.M + 63) / 64);
    if (a.x_dtype != SHREWQ_F32 || a.y_dtype != SHREWQ_F32 || a.q_up || a.extra.n != 0 || tiles > 0x3FFFFFFF) return false;
    if (t.tc_f32 != 1) return t.tc_f32 == 2;
    // Beyond a thousand features a tile is all main loop, which the pipeline over a split copy of x runs faster (and splits
    // along K): 1024 x 1000 x 2048 22.6 against 23.3 us, 1024 x 4096 x 4096 79 against 100 us; 4096 x 256 x 1024 21.2 against 12.8.
    return a.K <= 1024;
}

int launch_gemm_tcgen05_f32(shrewq_ctx *ctx, const ForwardArgs &a, const void *w_tmap) {
    const CUtensorMap &tw = *static_cast<const CUtensorMap *>(w_tmap);
    const size_t n_tiles = (a.N + kF32Chan - 1) / kF32Chan, tiles128 = n_tiles * ((a.M + 127) / 128);
    // 128-token tiles as soon as 64-token ones would take two rounds of the SMs: 4096 x 256 x 256 (128 of 64 tokens) 5.6 against
    // 6.4 us, 4096 x 512 x 512 (256) 13.3 against 9.9 us, 4096 x 50257 x 256 327 against 275 us.  Option tc_tok overrides.
    const bool wide = ctx->tuning.tc_tok == 128 || (ctx->tuning.tc_tok != 64 && 2 * tiles128 > (size_t)ctx->sm_count);
    // 128 KB for activations (and the rest for a deeper ring of codes) as long as those of a token tile fit there, else 192 KB.
    // With 128-token tiles only where output rows start on 32-byte sectors: 4096 x 50304 x 256 243 -> 219 us, but at 50257
    // channels, where every store splits sectors and L2 is the limit, 275 against 292 us.
    const bool sectors = (a.ldy * sizeof(float)) % 32 == 0 && (reinterpret_cast<uintptr_t>(a.y) & 31) == 0;
    if (wide) return sectors && a.K <= (size_t)F32Cfg<128, 128>::kXSlots * kF32BlockK ? launch_f32<128, 128>(ctx, a, tw) : launch_f32<128, 192>(ctx, a, tw);
    return a.K <= (size_t)F32Cfg<64, 128>::kXSlots * kF32BlockK ? launch_f32<64, 128>(ctx, a, tw) : launch_f32<64, 192>(ctx, a, tw);
}

}  // namespace shrewq
