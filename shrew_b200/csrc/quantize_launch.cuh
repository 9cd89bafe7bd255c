// Declaration shared by the quantizers' launchers.
#pragma once

#include "common.cuh"

namespace shrewq {

// f32, bf16 or f16 tensors in any mode (quantize.cu).  *taken false: nothing launched, the rows are too long or
// too many for the register kernels or the storage type is f64.
int launch_quantize_tuned(shrewq_ctx *ctx, const void *w, int w_dtype, size_t rows, size_t cols, int granularity, int bits,
                          int mode, int8_t *q, double *scales, double *zps, bool *taken);

}  // namespace shrewq
