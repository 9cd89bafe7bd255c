// Host-side launch of the tcgen05 forward, shared by its translation units (one per number of converter groups: the
// instantiations are what the build spends its time on).
#pragma once

#include <cuda.h>

#include <atomic>
#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "gemm_tcgen05_kernels.cuh"

namespace shrewq {

// every token tile, plain and gated, with G converter groups (gemm_tcgen05_g1.cu, _g2.cu, _g3.cu)
int launch_tcgen05_groups1(shrewq_ctx *ctx, const ForwardArgs &a, int tok, const CUtensorMap &tw, const CUtensorMap &tw2, void *fs, size_t fsb);
int launch_tcgen05_groups2(shrewq_ctx *ctx, const ForwardArgs &a, int tok, const CUtensorMap &tw, const CUtensorMap &tw2, void *fs, size_t fsb);
int launch_tcgen05_groups3(shrewq_ctx *ctx, const ForwardArgs &a, int tok, const CUtensorMap &tw, const CUtensorMap &tw2, void *fs, size_t fsb);

namespace {

// ---- host side ------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

int encode_2d(shrewq_ctx *ctx, CUtensorMap *out, CUtensorMapDataType dt, int elem_bytes, const void *base,
              size_t inner, size_t outer, int box_inner, int box_outer, CUtensorMapSwizzle sw) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return set_err(ctx, SHREWQ_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
    cuuint64_t strides[1] = {(cuuint64_t)inner * elem_bytes};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, dt, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_err(ctx, SHREWQ_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return SHREWQ_OK;
}

// ---- launch ---------------------------------------------------------------------------
constexpr size_t kScratchCounterOff = 4096, kScratchPartialOff = 8192;

struct LaunchPlan {
    int n_tiles, m_tiles, splits, rounds_per_split;
};

// Split-K when the output tiles alone leave most SMs idle: as many splits as fit in one wave, each with at
// least 2 pipeline rounds (token tiles up to 64, whose partial sums are small) or 8 (larger tiles).
// split_max_tok: the widest token tile that may be split (the no-allocation entry point keeps its
// partial sums in a fixed array and splits the small tiles only).
template <int TOK, int KSUB>
LaunchPlan plan_launch(const ForwardArgs &a, int chan_per_tile, int sm_count, bool allow_split, int split_max_tok = 256) {
    LaunchPlan p;
    p.n_tiles = (int)((a.N + chan_per_tile - 1) / chan_per_tile);
    p.m_tiles = (int)((a.M + TOK - 1) / TOK);
    const int rounds = (int)((a.K + kBlockK * KSUB - 1) / (kBlockK * KSUB));
    int splits = 1;
    const long tiles = (long)p.n_tiles * p.m_tiles;
    const int min_rounds = TOK <= 64 ? 2 : 8;
    if (allow_split && TOK <= split_max_tok && tiles <= 1024) {
        int want = (int)(sm_count / tiles);
        if (want > rounds / min_rounds) want = rounds / min_rounds;
        if (want > 1) splits = want;
    }
    p.rounds_per_split = (rounds + splits - 1) / splits;
    p.splits = (rounds + p.rounds_per_split - 1) / p.rounds_per_split;  // no empty split
    return p;
}

// cudaFuncSetAttribute once per kernel instantiation and device (bit d of `done`: device d has it)
template <typename Kern>
int set_smem_attr_once(shrewq_ctx *ctx, Kern kern, int bytes, std::atomic<unsigned long long> &done) {
    const int d = ctx->device;
    if (d >= 0 && d < 64 && ((done.load(std::memory_order_acquire) >> d) & 1ull)) return SHREWQ_OK;
    SHREWQ_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    if (d >= 0 && d < 64) done.fetch_or(1ull << d, std::memory_order_release);
    return SHREWQ_OK;
}

// scratch == nullptr: use (and grow) the context's scratch; otherwise a caller-provided
// region of scratch_bytes laid out as [0,4096) counters, partial sums from 4096.
// XSPLIT: a.x is the bf16 hi/lo pair of f32 activations, lo rows stacked under the M hi rows
template <int TOK, int KSUB, int G, bool GATED, typename YT, bool XSPLIT = false>
int launch_cfg(shrewq_ctx *ctx, const ForwardArgs &a, const CUtensorMap &tw, const CUtensorMap &tw2, bool allow_split,
               void *fixed_scratch, size_t fixed_scratch_bytes) {
    using C = Cfg<TOK, KSUB, XSPLIT>;
    CUtensorMap tx;
    int rc = encode_2d(ctx, &tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.x, a.K, XSPLIT ? 2 * a.M : a.M, kBlockK, TOK,
                       CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != SHREWQ_OK) return rc;
    auto kern = linear_i8_tcgen05_kernel<TOK, KSUB, G, GATED, YT, XSPLIT>;
    static std::atomic<unsigned long long> attr_done{0};  // per instantiation
    if ((rc = set_smem_attr_once(ctx, kern, C::kSmemRequest, attr_done)) != SHREWQ_OK) return rc;
    const LaunchPlan p = plan_launch<TOK, KSUB>(a, GATED ? 64 : 128, ctx->sm_count, allow_split, fixed_scratch ? 64 : 256);
    SplitK sk{nullptr, nullptr, p.rounds_per_split, 0, 0};
    Operands ops{a.scales, a.bias, a.scales_up, a.bias_up};
    // Option tc_tailsplit: when large tiles leave a short last wave, issue the full waves as one
    // launch and the tiles of the last wave as a second launch split along K so that it also fills
    // the SMs.  Not by default: it would make shapes that need no workspace share the context's (between streams,
    // under capture).
    const bool tail_split = ctx->tuning.tc_tailsplit == 1;
    if (tail_split && !fixed_scratch && TOK >= 128 && p.splits == 1) {
        const int tiles = p.n_tiles * p.m_tiles, rem = tiles % ctx->sm_count;
        const int rounds = p.rounds_per_split;
        int s_tail = rem > 0 ? ctx->sm_count / rem : 0;
        if (s_tail > 4) s_tail = 4;
        if (s_tail > rounds / 8) s_tail = rounds / 8;
        if (tiles > ctx->sm_count && rem > 0 && s_tail >= 2) {
            const size_t part_bytes = (size_t)rem * s_tail * TOK * kTileN * sizeof(float);
            if ((rc = ensure_scratch(ctx, kScratchPartialOff + part_bytes)) != SHREWQ_OK) return rc;
            SplitK head{nullptr, nullptr, rounds, 0, p.n_tiles};
            SHREWQ_CUDA_TRY(ctx, launch_maybe_pdl(kern, dim3((unsigned)(tiles - rem), 1, 1), dim3(64 + 128 * G), (size_t)C::kSmemRequest,
                                                  ctx->stream, a.pdl, tw, tw2, tx, ops, static_cast<YT *>(a.y), a.extra, (int)a.M,
                                                  (int)a.N, (int)a.K, a.ldy, a.epilogue, head, ctx->dev_status));
            const int rps = (rounds + s_tail - 1) / s_tail;
            const int splits = (rounds + rps - 1) / rps;
            SplitK tail{reinterpret_cast<float *>(static_cast<char *>(ctx->scratch) + kScratchPartialOff),
                        reinterpret_cast<unsigned int *>(static_cast<char *>(ctx->scratch) + kScratchCounterOff), rps,
                        tiles - rem, p.n_tiles};
            SHREWQ_CUDA_TRY(ctx, launch_maybe_pdl(kern, dim3((unsigned)rem, 1, (unsigned)splits), dim3(64 + 128 * G),
                                                  (size_t)C::kSmemRequest, ctx->stream, a.pdl, tw, tw2, tx, ops, static_cast<YT *>(a.y),
                                                  a.extra, (int)a.M, (int)a.N, (int)a.K, a.ldy, a.epilogue, tail, ctx->dev_status));
            ctx->launches += 2;
            SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
            return SHREWQ_OK;
        }
    }
    if (p.splits > 1) {
        const size_t tiles = (size_t)p.n_tiles * p.m_tiles;
        const size_t part_bytes = tiles * p.splits * TOK * kTileN * sizeof(float);
        if (fixed_scratch) {
            const size_t need = 4096 + part_bytes;
            if (need > fixed_scratch_bytes)
                return set_err(ctx, SHREWQ_ERR_UNSUPPORTED,
                               "forward_noalloc: this shape needs %zu bytes of split-K scratch, the built-in array holds %zu "
                               "(use shrewq_linear_forward, which allocates)", need, fixed_scratch_bytes);
            // the array keeps whatever the previous call left: the counters must start at zero
            SHREWQ_CUDA_TRY(ctx, cudaMemsetAsync(fixed_scratch, 0, 4096, ctx->stream));
            sk.counters = static_cast<unsigned int *>(fixed_scratch);
            sk.partials = reinterpret_cast<float *>(static_cast<unsigned char *>(fixed_scratch) + 4096);
        } else {
            // context scratch: [0,4096) quantizer words, [4096,8192) tile counters (at most one
            // per SM is ever in use), partial sums from 8192
            if ((rc = ensure_scratch(ctx, kScratchPartialOff + part_bytes)) != SHREWQ_OK) return rc;
            sk.counters = reinterpret_cast<unsigned int *>(static_cast<char *>(ctx->scratch) + kScratchCounterOff);
            sk.partials = reinterpret_cast<float *>(static_cast<char *>(ctx->scratch) + kScratchPartialOff);
        }
    }
    dim3 grid((unsigned)p.n_tiles, (unsigned)p.m_tiles, (unsigned)p.splits);
    SHREWQ_CUDA_TRY(ctx, launch_maybe_pdl(kern, grid, dim3(64 + 128 * G), (size_t)C::kSmemRequest, ctx->stream, a.pdl, tw, tw2, tx, ops,
                                          static_cast<YT *>(a.y), a.extra, (int)a.M, (int)a.N, (int)a.K, a.ldy, a.epilogue, sk,
                                          ctx->dev_status));
    ctx->launches += 1;
    SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
    return SHREWQ_OK;
}

template <bool GATED, int G, typename YT>
int launch_tok(shrewq_ctx *ctx, const ForwardArgs &a, int tok, const CUtensorMap &tw, const CUtensorMap &tw2, void *fs, size_t fsb) {
    const bool sk = ctx->tuning.tc_splitk != 0;
    switch (tok) {
        // small token tiles are HBM-bound: 2 sub-blocks per stage keeps the pipeline 6-7 stages
        // deep (TMEM columns limit the depth), i.e. ~100 KB of codes in flight per SM
        case 16: return launch_cfg<16, 2, G, GATED, YT>(ctx, a, tw, tw2, sk, fs, fsb);
        case 32: return launch_cfg<32, 2, G, GATED, YT>(ctx, a, tw, tw2, sk, fs, fsb);
        case 64: return launch_cfg<64, 2, G, GATED, YT>(ctx, a, tw, tw2, sk, fs, fsb);
        case 128: return launch_cfg<128, 2, G, GATED, YT>(ctx, a, tw, tw2, sk, fs, fsb);
        default: return launch_cfg<256, 1, G, GATED, YT>(ctx, a, tw, tw2, sk, fs, fsb);
    }
}

template <int G>
int launch_groups(shrewq_ctx *ctx, const ForwardArgs &a, int tok, const CUtensorMap &tw, const CUtensorMap &tw2, void *fs, size_t fsb) {
    if (a.y_dtype == SHREWQ_BF16)
        return a.q_up ? launch_tok<true, G, __nv_bfloat16>(ctx, a, tok, tw, tw2, fs, fsb) : launch_tok<false, G, __nv_bfloat16>(ctx, a, tok, tw, tw2, fs, fsb);
    return a.q_up ? launch_tok<true, G, float>(ctx, a, tok, tw, tw2, fs, fsb) : launch_tok<false, G, float>(ctx, a, tok, tw, tw2, fs, fsb);
}

}  // namespace
}  // namespace shrewq
