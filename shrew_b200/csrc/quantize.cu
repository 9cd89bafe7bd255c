// Launchers of the quantize / dequantize kernels (device code and its description:
// quantize_kernels.cuh).
#include <cuda_fp16.h>

#include "common.cuh"
#include "quantize_kernels.cuh"
#include "quantize_launch.cuh"

namespace shrewq {

namespace {

constexpr size_t kMaxGridRows = 0x7FFFFFFF;

template <int GROUP, int NV, typename T, bool ASYM>
void rows_reg(shrewq_ctx *ctx, const T *w, size_t rows, size_t cols, int8_t *q, double *scales, double *zps, int bits) {
    constexpr int THREADS = GROUP == 32 ? 256 : GROUP;
    constexpr size_t kRows = GROUP == 32 ? 8 * (8 / NV) : 1;  // rows per CTA
    const size_t grid = (rows + kRows - 1) / kRows;
    launch_maybe_pdl(quantize_rows_reg_kernel<GROUP, NV, T, ASYM>, dim3((unsigned)grid), dim3(THREADS), 0, ctx->stream, ctx->tuning.pdl != 0, w, rows, cols, q, scales, zps,
                     bits);
}

template <int GROUP, int NE, typename T, bool ASYM>
void rows_elem(shrewq_ctx *ctx, const T *w, size_t rows, size_t cols, int8_t *q, double *scales, double *zps, int bits) {
    const unsigned grid = (unsigned)(GROUP == 32 ? (rows + 7) / 8 : rows);
    launch_maybe_pdl(quantize_rows_elem_kernel<GROUP, NE, T, ASYM>, dim3(grid), dim3(GROUP == 32 ? 256 : GROUP), 0, ctx->stream, ctx->tuning.pdl != 0, w, rows, cols, q,
                     scales, zps, bits);
}

// Per-channel rows through registers.  false: the row is too long for it.
template <typename T, bool ASYM>
bool rows_in_registers(shrewq_ctx *ctx, const T *w, size_t rows, size_t cols, int bits, int8_t *q, double *scales, double *zps) {
    constexpr int EPV = Vec16<T>::kElems;
    const bool vec = cols % EPV == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & (EPV - 1)) == 0;
    const size_t nvec = cols / EPV;
    // Tile widths by the vectors of a row: a warp up to 256 of them, then whole CTAs.  f32 rows of more than 1024 vectors keep
    // eight per thread (94 % of the copy rate); the 16-bit types, with twice the elements in a vector, keep four.
    constexpr bool k16 = sizeof(T) == 2;
    if (vec && nvec <= 32) rows_reg<32, 1, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (vec && nvec <= 64) rows_reg<32, 2, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (vec && nvec <= 128) rows_reg<32, 4, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (vec && nvec <= 256) rows_reg<32, 8, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (vec && nvec <= 512) rows_reg<k16 ? 128 : 256, k16 ? 4 : 2, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (vec && nvec <= 1024) rows_reg<256, 4, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (vec && nvec <= 2048) rows_reg<k16 ? 512 : 256, k16 ? 4 : 8, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (vec && nvec <= 4096) rows_reg<k16 ? 1024 : 512, k16 ? 4 : 8, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (vec && nvec <= 8192) rows_reg<1024, 8, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    // element tiles: the narrowest that holds the row (its unused slots cost as much as used ones)
    else if (cols <= 256) rows_elem<32, 8, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (cols <= 512) rows_elem<32, 16, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (cols <= 1024) rows_elem<128, 8, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (cols <= 2048) rows_elem<256, 8, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (cols <= 4096) rows_elem<256, 16, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else if (cols <= 8192) rows_elem<512, 16, T, ASYM>(ctx, w, rows, cols, q, scales, zps, bits);
    else return false;
    ctx->launches += 1;
    return true;
}

// Per-tensor in two launches (extrema and parameters, codes), the second one allowed to start under the first one's tail.
template <typename T, bool ASYM>
int tensor_two_pass(shrewq_ctx *ctx, const T *w, size_t n, int bits, int8_t *q, double *scales, double *zps) {
    static_assert(sizeof(TensorGroup) <= kTensorSlotBytes && kTensorSlotBytes % 64 == 0, "a slot holds one call's words");
    TensorGroup *g = reinterpret_cast<TensorGroup *>(static_cast<char *>(ctx->tensor_slots) +
                                                     ctx->tensor_calls.fetch_add(1, std::memory_order_relaxed) % kTensorSlots * kTensorSlotBytes);
    const size_t vecs = n / Vec16<T>::kElems;
    const size_t cap = (size_t)ctx->sm_count * 8 < (size_t)kMaxPartials ? (size_t)ctx->sm_count * 8 : (size_t)kMaxPartials;
    const size_t want = (vecs + 1023) / 1024;
    SHREWQ_CUDA_TRY(ctx, launch_maybe_pdl(extrema_partials_kernel<T, ASYM>, dim3((unsigned)(want < 1 ? 1 : (want > cap ? cap : want))), dim3(256), 0,
                                          ctx->stream, ctx->tuning.pdl != 0, w, n, bits, g, scales, zps));
    ctx->launches += 1;
    if (n > 0) {
        constexpr int U = sizeof(T) == 2 ? 2 : 4;
        SHREWQ_CUDA_TRY(ctx, launch_maybe_pdl(quantize_tensor_kernel<T, ASYM, U>, dim3((unsigned)(want < 1 ? 1 : (vecs + 256 * U - 1) / (256 * U))),
                                              dim3(256), 0, ctx->stream, ctx->tuning.pdl != 0, w, n, g, q));
        ctx->launches += 1;
    }
    return SHREWQ_OK;
}

template <typename T, bool ASYM>
int quantize_t(shrewq_ctx *ctx, const T *w, size_t rows, size_t cols, int granularity, int bits, int8_t *q, double *scales,
               double *zps, bool *taken) {
    *taken = true;
    if (granularity == SHREWQ_PER_CHANNEL) {
        if (rows == 0) return SHREWQ_OK;
        if (rows > kMaxGridRows) {  // a CTA per row or more: left to the kernels whose grid strides over the rows
            *taken = false;
            return SHREWQ_OK;
        }
        *taken = rows_in_registers<T, ASYM>(ctx, w, rows, cols, bits, q, scales, zps);
    } else {
        int rc = tensor_two_pass<T, ASYM>(ctx, w, rows * cols, bits, q, scales, zps);
        if (rc != SHREWQ_OK) return rc;
    }
    SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
    return SHREWQ_OK;
}

}  // namespace

// f32, bf16 or f16 tensors in any mode.  *taken false: per-channel rows too long, or too many, for the register kernels.
int launch_quantize_tuned(shrewq_ctx *ctx, const void *w, int w_dtype, size_t rows, size_t cols, int granularity, int bits,
                          int mode, int8_t *q, double *scales, double *zps, bool *taken) {
    const bool asym = mode == SHREWQ_ASYMMETRIC;
#define SHREWQ_QUANT(T)                                                                                                          \
    return asym ? quantize_t<T, true>(ctx, static_cast<const T *>(w), rows, cols, granularity, bits, q, scales, zps, taken)     \
                : quantize_t<T, false>(ctx, static_cast<const T *>(w), rows, cols, granularity, bits, q, scales, zps, taken)
    if (w_dtype == SHREWQ_F32) SHREWQ_QUANT(float);
    if (w_dtype == SHREWQ_BF16) SHREWQ_QUANT(__nv_bfloat16);
    if (w_dtype == SHREWQ_F16) SHREWQ_QUANT(__half);
#undef SHREWQ_QUANT
    *taken = false;
    return SHREWQ_OK;
}

int launch_quantize(shrewq_ctx *ctx, const float *w, size_t rows, size_t cols, int granularity,
                    int8_t *q, double *scales) {
    if (granularity == SHREWQ_PER_CHANNEL && rows > kMaxGridRows)
        return set_err(ctx, SHREWQ_ERR_UNSUPPORTED, "quantize: more than 2^31-1 channels");
    bool taken = false;
    int rc = launch_quantize_tuned(ctx, w, SHREWQ_F32, rows, cols, granularity, 8, SHREWQ_SYMMETRIC, q, scales, nullptr, &taken);
    if (rc != SHREWQ_OK || taken) return rc;
    const unsigned grid = (unsigned)(rows < (size_t)ctx->sm_count * 32 ? rows : (size_t)ctx->sm_count * 32);
    quantize_rows_generic_kernel<<<grid, 256, 0, ctx->stream>>>(w, rows, cols, q, scales);
    ctx->launches += 1;
    SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
    return SHREWQ_OK;
}

// ---- per-tensor quantization of a row shard ---------------------------------------------------
// A tensor split over several GPUs has ONE per-tensor scale, defined by the amax of the whole
// tensor (quantize.rs:349-351).  Each rank takes the amax of its shard, the ranks take the max of
// those (one float through an all-reduce, done by the caller), and every rank quantizes its shard
// with the global value.  Same kernels as the single-GPU per-tensor path.
int launch_absmax(shrewq_ctx *ctx, const float *w, size_t n, float *amax_dev) {
    SHREWQ_CUDA_TRY(ctx, cudaMemsetAsync(amax_dev, 0, sizeof(float), ctx->stream));  // +0.0f
    if (n > 0) {
        size_t want = (n / 4 + 255) / 256;
        const size_t cap = (size_t)ctx->sm_count * 16;
        const unsigned grid = (unsigned)(want < 1 ? 1 : (want > cap ? cap : want));
        absmax_flat_kernel<<<grid, 256, 0, ctx->stream>>>(w, n, reinterpret_cast<unsigned int *>(amax_dev));
        ctx->launches += 1;
    }
    SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
    return SHREWQ_OK;
}

int launch_quantize_given_amax(shrewq_ctx *ctx, const float *w, size_t n, const float *amax_dev, int8_t *q,
                               double *scale) {
    int rc = ensure_scratch(ctx, 256);
    if (rc != SHREWQ_OK) return rc;
    TensorParams *tp = reinterpret_cast<TensorParams *>(reinterpret_cast<char *>(ctx->scratch) + 64);
    // the scale always derives from the supplied amax, also for an empty shard
    finalize_tensor_scale_kernel<<<1, 1, 0, ctx->stream>>>(reinterpret_cast<const unsigned int *>(amax_dev), scale, tp);
    ctx->launches += 1;
    if (n > 0) {
        size_t want = (n / 4 + 255) / 256;
        const size_t cap = (size_t)ctx->sm_count * 16;
        const unsigned grid = (unsigned)(want < 1 ? 1 : (want > cap ? cap : want));
        quantize_flat_kernel<<<grid, 256, 0, ctx->stream>>>(w, n, tp, q);
        ctx->launches += 1;
    }
    SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
    return SHREWQ_OK;
}

int launch_dequantize(shrewq_ctx *ctx, const int8_t *q, const double *scales, size_t rows,
                      size_t cols, int granularity, int out_dtype, void *out) {
    const size_t n = rows * cols;
    if (n == 0) return SHREWQ_OK;
    const int per_channel = granularity == SHREWQ_PER_CHANNEL;
    const int vec_ok = ((reinterpret_cast<uintptr_t>(q) & 3) == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
    const size_t words = 256 * (out_dtype == SHREWQ_F32 ? DequantWords<float>::kPerThread : DequantWords<uint16_t>::kPerThread);
    const size_t want = vec_ok ? (n / 4 + words - 1) / words : (n + 255) / 256;
    const size_t cap = vec_ok ? 0x7FFFFFFF : (size_t)ctx->sm_count * 32;
    unsigned grid = (unsigned)(want < 1 ? 1 : (want > cap ? cap : want));
    if (out_dtype == SHREWQ_F32)
        SHREWQ_CUDA_TRY(ctx, launch_maybe_pdl(dequantize_kernel<float>, dim3(grid), dim3(256), 0, ctx->stream, ctx->tuning.pdl != 0, q, scales, rows, cols, per_channel,
                                              static_cast<float *>(out), vec_ok));
    else
        SHREWQ_CUDA_TRY(ctx, launch_maybe_pdl(dequantize_kernel<uint16_t>, dim3(grid), dim3(256), 0, ctx->stream, ctx->tuning.pdl != 0, q, scales, rows, cols, per_channel,
                                              static_cast<uint16_t *>(out), vec_ok));
    ctx->launches += 1;
    SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
    return SHREWQ_OK;
}

int launch_split_f32(shrewq_ctx *ctx, const float *x, size_t n, void *hi_bf16, void *lo_bf16) {
    if (n == 0) return SHREWQ_OK;
    size_t want = (n + 255) / 256;
    const size_t cap = (size_t)ctx->sm_count * 32;
    split_f32_kernel<<<(unsigned)(want > cap ? cap : want), 256, 0, ctx->stream>>>(
        x, n, static_cast<__nv_bfloat16 *>(hi_bf16), static_cast<__nv_bfloat16 *>(lo_bf16));
    ctx->launches += 1;
    SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
    return SHREWQ_OK;
}

int launch_scales_to_f32(shrewq_ctx *ctx, const double *scales, int granularity, size_t n, float *out) {
    if (n == 0) return SHREWQ_OK;
    scales_to_f32_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(
        scales, granularity == SHREWQ_PER_CHANNEL, n, out);
    ctx->launches += 1;
    SHREWQ_CUDA_TRY(ctx, cudaGetLastError());
    return SHREWQ_OK;
}

}  // namespace shrewq
