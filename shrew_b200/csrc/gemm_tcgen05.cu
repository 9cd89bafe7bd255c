// Host side of the tcgen05 forward: tensor maps, choice of the token tile, entry points (launch plan and launchers:
// gemm_tcgen05_launch.cuh; device code and its description: gemm_tcgen05_kernels.cuh).
#include "gemm_tcgen05_launch.cuh"

namespace shrewq {
namespace {

// Token tile: the smallest tile that covers M up to 128.  Above that a gate/up launch takes 256 tokens
// (twice the tokens per converted weight byte; measured 12 % shorter on the 4096 -> 11008 block at batch 512),
// a plain launch 256 tokens unless 128-token tiles fill the SMs markedly better (few channel tiles, e.g.
// N = 4096 at M = 512: 128 CTAs instead of 64).
int choose_tok(const ForwardArgs &a, bool gated, int sm_count, const Tuning &t) {
    const int forced = (gated && t.tc_tok_gated) ? t.tc_tok_gated : t.tc_tok;
    if (forced == 16 || forced == 32 || forced == 64 || forced == 128 || forced == 256) return forced;
    if (a.M <= 16) return 16;
    if (a.M <= 32) return 32;
    if (a.M <= 64) return 64;
    if (a.M <= 128) return 128;
    if (gated) return 256;
    const long n_tiles = (long)((a.N + 127) / 128);
    auto fill = [&](int tok) {
        const long tiles = n_tiles * (long)((a.M + tok - 1) / tok);
        const long waves = (tiles + sm_count - 1) / sm_count;
        return (double)tiles / (double)(waves * sm_count);
    };
    return fill(128) * 0.85 > fill(256) ? 128 : 256;
}

int launch_forward(shrewq_ctx *ctx, const ForwardArgs &a, const CUtensorMap &tw, const CUtensorMap &tw2, void *fs, size_t fsb) {
    const int tok = choose_tok(a, a.q_up != nullptr, ctx->sm_count, ctx->tuning);
    if (ctx->tuning.tc_groups == 1) return launch_tcgen05_groups1(ctx, a, tok, tw, tw2, fs, fsb);
    if (ctx->tuning.tc_groups == 2) return launch_tcgen05_groups2(ctx, a, tok, tw, tw2, fs, fsb);
    return launch_tcgen05_groups3(ctx, a, tok, tw, tw2, fs, fsb);
}

// ---- forward without any allocation ---------------------------------------------------
// Split-K scratch for shrewq_linear_forward_noalloc: a fixed array inside the library image
// instead of a cudaMalloc'd buffer.  Every GPU that loads the library holds these 4 MiB
// until the process exits.  Layout: [0,4096) tile counters, partial sums from 4096.
constexpr size_t kStaticScratchBytes = 4u << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// In host code the array's name is only a handle for the runtime, not a device address:
// the address is looked up once per device (with that device current) and cached.
constexpr int kMaxDevices = 64;
static std::atomic<void *> g_static_scratch_addr[kMaxDevices];

int static_scratch_for_device(shrewq_ctx *ctx, void **out) {
    if (ctx->device < 0 || ctx->device >= kMaxDevices)
        return set_err(ctx, SHREWQ_ERR_UNSUPPORTED, "forward_noalloc: device index %d above %d", ctx->device, kMaxDevices - 1);
    if (!g_static_scratch_addr[ctx->device].load(std::memory_order_acquire)) {
        void *p = nullptr;
        SHREWQ_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess || !p)
            return set_err(ctx, SHREWQ_ERR_CUDA, "forward_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        g_static_scratch_addr[ctx->device].store(p, std::memory_order_release);  // every thread looks up the same address
    }
    *out = g_static_scratch_addr[ctx->device].load(std::memory_order_acquire);
    return SHREWQ_OK;
}

}  // namespace

bool tcgen05_supported(const ForwardArgs &a) {
    return a.x_dtype == SHREWQ_BF16 && a.K >= 16 && (a.K % 16) == 0 && a.M >= 1 && a.N >= 1 &&
           (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.q) & 15) == 0 &&
           (!a.q_up || (reinterpret_cast<uintptr_t>(a.q_up) & 15) == 0) && a.K < (1u << 31) && a.N < (1u << 31) &&
           a.M < (1u << 31) && (a.M + 15) / 16 <= 65535 * 16;
}

// box_rows = 128 for plain tiles, 64 for the gate / up halves of a gated tile
int encode_weight_tmap(shrewq_ctx *ctx, const int8_t *q, size_t n, size_t k, int box_rows, void *tmap_out) {
    return encode_2d(ctx, static_cast<CUtensorMap *>(tmap_out), CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, q, k, n, kBlockK,
                     box_rows, CU_TENSOR_MAP_SWIZZLE_64B);
}

// f32 activations: a.x points at the bf16 hi matrix [M,K] with the lo matrix right behind it
int launch_gemm_tcgen05_xsplit(shrewq_ctx *ctx, const ForwardArgs &a, const void *w_tmap) {
    const CUtensorMap &tw = *static_cast<const CUtensorMap *>(w_tmap);
    const bool sk = ctx->tuning.tc_splitk != 0;
    // token tile: 256 (half the tiles, twice the work per prologue and per byte of weights) when such tiles still
    // keep three quarters of the SMs busy, 128 otherwise; option tc_tok overrides.  Measured at 4096 tokens:
    // 50257 x 256: 666 against 910 us; 1024 x 256: 14.8 against 19.6 us; 256 x 1024 (32 tiles): 28.4 against 21.5 us.
    const size_t tiles256 = ((a.N + kTileN - 1) / kTileN) * ((a.M + 255) / 256);
    const int tok = ctx->tuning.tc_tok == 128 || ctx->tuning.tc_tok == 256 ? ctx->tuning.tc_tok
                    : (tiles256 * 4 >= (size_t)ctx->sm_count * 3 ? 256 : 128);
    if (tok == 256) {
        if (a.y_dtype == SHREWQ_BF16) return launch_cfg<256, 1, 3, false, __nv_bfloat16, true>(ctx, a, tw, tw, sk, nullptr, 0);
        return launch_cfg<256, 1, 3, false, float, true>(ctx, a, tw, tw, sk, nullptr, 0);
    }
    if (a.y_dtype == SHREWQ_BF16) return launch_cfg<128, 1, 3, false, __nv_bfloat16, true>(ctx, a, tw, tw, sk, nullptr, 0);
    return launch_cfg<128, 1, 3, false, float, true>(ctx, a, tw, tw, sk, nullptr, 0);
}

int launch_gemm_tcgen05_noalloc(shrewq_ctx *ctx, const ForwardArgs &a, const void *w_tmap) {
    const CUtensorMap &tw = *static_cast<const CUtensorMap *>(w_tmap);
    void *base = nullptr;
    int rc = static_scratch_for_device(ctx, &base);
    if (rc != SHREWQ_OK) return rc;
    return launch_forward(ctx, a, tw, tw, base, kStaticScratchBytes);
}

// w_tmap: 128-row boxes of the weight (plain) or 64-row boxes of the gate matrix (gated, with
// w_up_tmap the 64-row boxes of the up matrix)
// The launch plan of the tcgen05 forward for a shape, without launching anything (pure host arithmetic:
// token tile, tile grid, K splits, pipeline rounds per split).
int plan_gemm_tcgen05(size_t M, size_t N, size_t K, bool gated, int sm_count, int *tok, int *n_tiles, int *m_tiles,
                      int *splits, int *rounds_per_split) {
    ForwardArgs a{};
    a.M = M; a.N = N; a.K = K;
    const Tuning t;  // the defaults
    const int chan = gated ? 64 : 128;
    const int tk = choose_tok(a, gated, sm_count, t);
    LaunchPlan p;
    switch (tk) {
        case 16: p = plan_launch<16, 2>(a, chan, sm_count, true); break;
        case 32: p = plan_launch<32, 2>(a, chan, sm_count, true); break;
        case 64: p = plan_launch<64, 2>(a, chan, sm_count, true); break;
        case 128: p = plan_launch<128, 2>(a, chan, sm_count, true); break;
        case 256: p = plan_launch<256, 1>(a, chan, sm_count, true); break;
        default: return SHREWQ_ERR_INVALID_ARG;
    }
    *tok = tk; *n_tiles = p.n_tiles; *m_tiles = p.m_tiles; *splits = p.splits; *rounds_per_split = p.rounds_per_split;
    return SHREWQ_OK;
}

int launch_gemm_tcgen05(shrewq_ctx *ctx, const ForwardArgs &a, const void *w_tmap, const void *w_up_tmap) {
    const CUtensorMap &tw = *static_cast<const CUtensorMap *>(w_tmap);
    return launch_forward(ctx, a, tw, a.q_up ? *static_cast<const CUtensorMap *>(w_up_tmap) : tw, nullptr, 0);
}

}  // namespace shrewq
