// Host side of the CTA-pair forward (device code and its description: gemm_tcgen05_2cta_kernels.cuh).
#include <cuda.h>

#include <atomic>
#include <cstdlib>

#include "common.cuh"
#include "gemm_tcgen05_2cta_kernels.cuh"

namespace shrewq {
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode_x_half(shrewq_ctx *ctx, CUtensorMap *out, const void *x, size_t K, size_t M, int tok_half) {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
            qres != cudaDriverEntryPointSuccess)
            return set_err(ctx, SHREWQ_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
        fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    cuuint32_t box[2] = {(cuuint32_t)kBlockK, (cuuint32_t)tok_half};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(x), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_err(ctx, SHREWQ_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return SHREWQ_OK;
}

// What a launch of the kernel needs besides the operands, prepared for one token tile.
template <typename YT, bool GATED, int TOKP>
struct PairLaunch {
    CUtensorMap tx;

    int prepare(shrewq_ctx *ctx, const ForwardArgs &a) {
        int rc = encode_x_half(ctx, &tx, a.x, a.K, a.M, PairCfg<TOKP>::kTokHalf);
        if (rc != SHREWQ_OK) return rc;
        static std::atomic<unsigned long long> attr_done{0};  // per instantiation: bit d = device d has the attribute
        if (ctx->device < 0 || ctx->device >= 64 || !((attr_done.load(std::memory_order_acquire) >> ctx->device) & 1ull)) {
            SHREWQ_CUDA_TRY(ctx, cudaFuncSetAttribute(linear_i8_tcgen05_pair_kernel<YT, GATED, TOKP>,
                                                      cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<TOKP>::kSmemBytes));
            if (ctx->device >= 0 && ctx->device < 64) attr_done.fetch_or(1ull << ctx->device, std::memory_order_release);
        }
        return SHREWQ_OK;
    }
    int run(shrewq_ctx *ctx, const ForwardArgs &a, const CUtensorMap &tw, const CUtensorMap &tw2, dim3 grid, const SplitK2 &sk) const {
        const Operands ops{a.scales, a.bias, a.scales_up, a.bias_up};
        SHREWQ_CUDA_TRY(ctx, launch_maybe_pdl(linear_i8_tcgen05_pair_kernel<YT, GATED, TOKP>, grid, dim3(kThreads),
                                              (size_t)PairCfg<TOKP>::kSmemBytes, ctx->stream, a.pdl, tw, tw2, tx, ops,
                                              static_cast<YT *>(a.y), a.extra, (int)a.M, (int)a.N, (int)a.K, a.ldy, a.epilogue, sk,
                                              ctx->dev_status));
        ctx->launches += 1;
        SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
        return SHREWQ_OK;
    }
};

// K splits of `ctas` output tiles that leave SMs idle: as many as fit in one wave, each of at least 8 rounds
int pair_splits(const shrewq_ctx *ctx, long ctas, int rounds) {
    int want = ctas <= 1024 ? (int)(ctx->sm_count / ctas) : 1;
    if (want > rounds / 8) want = rounds / 8;
    if (want < 2) return 1;
    const int rps = (rounds + want - 1) / want;
    return (rounds + rps - 1) / rps;  // no empty split
}

// context scratch as in the single-CTA launcher: tile counters at 4096, partial sums from 8192
int split_scratch(shrewq_ctx *ctx, size_t cta_tiles, int splits, int tokp, SplitK2 *sk) {
    int rc = ensure_scratch(ctx, 8192 + cta_tiles * splits * tokp * kLanes * sizeof(float));
    if (rc != SHREWQ_OK) return rc;
    sk->counters = reinterpret_cast<unsigned int *>(static_cast<char *>(ctx->scratch) + 4096);
    sk->partials = reinterpret_cast<float *>(static_cast<char *>(ctx->scratch) + 8192);
    return SHREWQ_OK;
}

template <typename YT, bool GATED>
int launch_pair(shrewq_ctx *ctx, const ForwardArgs &a, const CUtensorMap &tw, const CUtensorMap &tw2) {
    int rc;
    constexpr int kChanPair = GATED ? kLanes : 2 * kLanes;  // output channels per CTA pair
    const unsigned pairs = (unsigned)((a.N + kChanPair - 1) / kChanPair);
    const int rounds = (int)((a.K + kBlockK * kSub - 1) / (kBlockK * kSub));
    const int per_wave = ctx->sm_count / 2;  // pair tiles resident at once, one CTA per SM
    const unsigned m_tiles = (unsigned)((a.M + 255) / 256), m_halves = (unsigned)((a.M + 127) / 128);
    const int tiles = (int)(pairs * m_tiles), halves = (int)(pairs * m_halves);
    const int splits = pair_splits(ctx, 2L * tiles, rounds);

    // 128-token pair tiles where 256-token ones would be split along K and their halves still fit in one wave: twice the output
    // tiles, half (or none) of the partial sums.  4096 x 11008 at 200 tokens 32.3 -> 28.3 us, at 384 41.4 -> 38.8, at 512
    // equal.  (bf16 results only: fewer splits are longer f32 sums, which an f32 result would show.)
    if (ctx->tuning.tc_tok == 128 || (ctx->tuning.tc_tok == 0 && sizeof(YT) == 2 && splits >= 2 && halves <= per_wave)) {
        PairLaunch<YT, GATED, 128> half;
        if ((rc = half.prepare(ctx, a)) != SHREWQ_OK) return rc;
        const int sp = pair_splits(ctx, 2L * halves, rounds);
        SplitK2 sk{nullptr, nullptr, (rounds + sp - 1) / sp, 0, 0};
        if (sp > 1 && (rc = split_scratch(ctx, (size_t)2 * halves, sp, 128, &sk)) != SHREWQ_OK) return rc;
        return half.run(ctx, a, tw, tw2, dim3(2 * pairs, m_halves, (unsigned)sp), sk);
    }
    PairLaunch<YT, GATED, 256> full;
    if ((rc = full.prepare(ctx, a)) != SHREWQ_OK) return rc;
    // A short last wave of pair tiles (at most a quarter of a wave): the full waves go out as one launch of whole-K tiles, the
    // tail as a second launch split along K, so that it fills the SMs too.  Measured on the MLP block at batch 512: a tail of
    // 12 of 74 pair tiles (the 2-GPU shard) 57.6 -> 53.4 us; a tail of 24 (one GPU) gains nothing, split or as 128-token halves
    // (85.0 without, 86.8 us as halves).  Option tc_tailsplit: 1 = whenever a tail exists, 2 = never.
    const int rem = per_wave > 0 ? tiles % per_wave : 0;
    if (ctx->tuning.tc_tailsplit != 2 && splits == 1 && tiles > per_wave && rem > 0) {
        int s_tail = per_wave / rem;
        if (s_tail > 4) s_tail = 4;
        if (s_tail > rounds / 8) s_tail = rounds / 8;
        // (the tail launch may start under the head launch's last wave: the two write disjoint tiles)
        if (s_tail >= 2 && (ctx->tuning.tc_tailsplit == 1 || rem * 4 <= per_wave)) {
            const int rps = (rounds + s_tail - 1) / s_tail, sp = (rounds + rps - 1) / rps;
            SplitK2 head{nullptr, nullptr, rounds, 0, (int)pairs}, tail{nullptr, nullptr, rps, tiles - rem, (int)pairs};
            if ((rc = split_scratch(ctx, (size_t)2 * rem, sp, 256, &tail)) != SHREWQ_OK) return rc;
            if ((rc = full.run(ctx, a, tw, tw2, dim3(2u * (unsigned)(tiles - rem)), head)) != SHREWQ_OK) return rc;
            return full.run(ctx, a, tw, tw2, dim3(2u * (unsigned)rem, 1, (unsigned)sp), tail);
        }
    }
    SplitK2 sk{nullptr, nullptr, (rounds + splits - 1) / splits, 0, 0};
    if (splits > 1 && (rc = split_scratch(ctx, (size_t)2 * tiles, splits, 256, &sk)) != SHREWQ_OK) return rc;
    return full.run(ctx, a, tw, tw2, dim3(2 * pairs, m_tiles, (unsigned)splits), sk);
}

}  // namespace

#ifdef SHREWQ_TRACE
extern "C" __attribute__((visibility("default"))) int shrewq_debug_set_trace_pair(long long *dev_buf) {
    return (int)cudaMemcpyToSymbol(g_trace_pair, &dev_buf, sizeof(dev_buf));
}
#endif

// Plain forward: w_tmap = the handle's 128-row INT8 boxes, w_up_tmap = nullptr.  Gate/up pair: the
// 64-row boxes of the gate and of the up handle (the descriptors the single-CTA kernel uses).
int launch_gemm_tcgen05_2cta(shrewq_ctx *ctx, const ForwardArgs &a, const void *w_tmap, const void *w_up_tmap) {
    const CUtensorMap &tw = *static_cast<const CUtensorMap *>(w_tmap);
    if (a.q_up) {
        if (!w_up_tmap) return set_err(ctx, SHREWQ_ERR_INVALID_ARG, "tcgen05-2cta: the up matrix has no tensor map");
        const CUtensorMap &tw2 = *static_cast<const CUtensorMap *>(w_up_tmap);
        if (a.y_dtype == SHREWQ_BF16) return launch_pair<__nv_bfloat16, true>(ctx, a, tw, tw2);
        return launch_pair<float, true>(ctx, a, tw, tw2);
    }
    if (a.y_dtype == SHREWQ_BF16) return launch_pair<__nv_bfloat16, false>(ctx, a, tw, tw);
    return launch_pair<float, false>(ctx, a, tw, tw);
}

}  // namespace shrewq
