// Quantize / dequantize kernels (sm_100a): per-channel rows of f32, bf16 or f16 in every mode, per-tensor, and back.
//
// The arithmetic, and why the f32 shortcut gives the reference's f64 codes bit for bit: quantize_common.cuh.
//
// Memory plan (HBM-bound; f32 5 B/element, bf16 and f16 3 B/element): a row is read ONCE into registers as 16-byte
// vectors, reduced (warp shuffles, then shared memory across warps), and quantized from registers; codes are
// written as packed words.  Rows that are not whole aligned vectors are held in registers element by element; rows
// too long for registers take a two-pass kernel whose second read normally hits L2.  Per-tensor: one pass for the
// extrema of every block, a second one for the codes.
//
// The kernels are launched with programmatic stream serialization and wait for the previous kernel before they touch
// memory: the next launch's start-up lies under the tail of the one before.
//
// This header holds the device code only (no launch syntax, no runtime calls), so that it also
// compiles as plain C++ against a small CUDA stand-in: the CPU tests run these kernels thread by
// thread and compare them with the golden vectors (tests/cpu_emu/).
#pragma once

#include "ptx_small.cuh"
#include "quantize_common.cuh"

namespace shrewq {
namespace {

struct RowParams {
    double inv64;
    float inv32;
    int exact_only;  // 1: every element must take the f64 path
};

__device__ __forceinline__ void make_params(float amax, double *scale_out, RowParams *p) {
    double a = (double)amax;
    double scale = a < 1e-30 ? 1.0 : a / 127.0;
    double inv = fabs(scale) < 1e-30 ? 0.0 : 1.0 / scale;
    *scale_out = scale;
    p->inv64 = inv;
    p->inv32 = (float)inv;
    // f32 fast path needs an ordinary reciprocal: finite, normal in f32, not zero
    p->exact_only = !(inv > 1e-30 && inv < 1e30);
}

// The reference's element map, operation for operation, in f64.
__device__ __forceinline__ int quant_exact(float v, double inv64) {
    double t = __dadd_rn(__dmul_rn((double)v, inv64), 0.0);
    if (t != t) return 0;  // NaN as i8 == 0
    double r = trunc(t);
    if (fabs(t - r) >= 0.5) r += copysign(1.0, t);  // round half away from zero
    r = fmin(fmax(r, -127.0), 127.0);
    return (int)r;
}

// for scales that do not come from the elements themselves (a supplied amax): the f32 candidate is clamped
__device__ __forceinline__ int quant_one(float v, const RowParams &p) {
    if (!p.exact_only) {
        const float t = v * p.inv32, a = t + kRoundMagic;
        if (fabsf(t - (a - kRoundMagic)) <= kSafeSym && fabsf(t) < 1000.0f)  // false for NaN
            return max(-127, min(127, (int)(__float_as_uint(a) - __float_as_uint(kRoundMagic))));
    }
    return quant_exact(v, p.inv64);
}

__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d) {
    return (uint32_t)(a & 0xFF) | ((uint32_t)(b & 0xFF) << 8) | ((uint32_t)(c & 0xFF) << 16) |
           ((uint32_t)(d & 0xFF) << 24);
}

__device__ __forceinline__ float abs4max(float4 v) {
    // fmaxf drops a NaN operand, as f64::max does in the reference's fold
    return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}

// ---- per-channel, row held in registers ---------------------------------------------
// The extrema of a row from those of its threads.  GROUP threads own a row; with several warps per row they meet in
// shared memory (one barrier; every thread reads the partial results itself, so no second one is needed).
template <int GROUP, bool ASYM>
__device__ __forceinline__ void extrema_group(Extrema &e, int t) {
    constexpr int W = GROUP / 32;
    __shared__ Extrema s_part[W];
    extrema_warp<ASYM>(e);
    if ((t & 31) == 0) s_part[t >> 5] = e;
    __syncthreads();
    if constexpr (W <= 8) {
        e = s_part[0];
#pragma unroll
        for (int i = 1; i < W; ++i) extrema_merge<ASYM>(e, s_part[i]);
    } else {
        e = s_part[(t & 31) < W ? (t & 31) : 0];
        extrema_warp<ASYM>(e);
    }
}

// GROUP = 32: a warp takes 8 / NV consecutive rows at a time.  Otherwise the GROUP threads of a CTA own one row, NV
// 16-byte vectors each.  cols is a multiple of the vector's elements, w is 16-byte and q 4-byte (f32) or 8-byte aligned
// (checked by the launcher).  Thread 0 forms the f64 parameters while the others already write codes; the undecided
// elements wait for them at the end (symmetric; an asymmetric row's zero point is needed for every code).
// 8192 x 8192 f32: 54 us (6.2 TB/s); 66.9 us with two barriers a row, two f64 divisions on the way to the codes and ~20
// instructions an element.  (CTAs that walk over rows with the next row's loads in flight were slower: 33 against 29 us
// for 8192 x 4096, the registers cost more resident rows than the look-ahead gave.)
template <int GROUP, int NV, typename T = float, bool ASYM = false>
__global__ void __launch_bounds__(GROUP == 32 ? 256 : GROUP)
quantize_rows_reg_kernel(const T *__restrict__ w, size_t rows, size_t cols, int8_t *__restrict__ q, double *__restrict__ scales,
                         double *__restrict__ zps = nullptr, int bits = 8) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int EPV = Vec16<T>::kElems;
    if constexpr (GROUP == 32) {
        constexpr int R = NV >= 8 ? 1 : 8 / NV;
        const size_t row = ((size_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * R;
        if (row >= rows) return;
        const int count = rows - row < (size_t)R ? (int)(rows - row) : R;
        quantize_rows_by_warp<R, NV, T, ASYM>(w + row * cols, cols, count, bits, q + row * cols, scales + row, zps ? zps + row : zps,
                                              threadIdx.x & 31);
    } else {
        const int t = threadIdx.x;
        const size_t row = blockIdx.x;
        const int nvec = (int)(cols / EPV);
        const T *src = w + row * cols;
        int8_t *dst = q + row * cols;
        __shared__ GroupParams s_p;
        uint4 v[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = t + i * GROUP;
            v[i] = c < nvec ? __ldcs(reinterpret_cast<const uint4 *>(src) + c) : make_uint4(0, 0, 0, 0);
        }
        Extrema e = extrema_none<ASYM>();
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (!ASYM || t + i * GROUP < nvec) extrema_add16<T, ASYM>(e, v[i]);  // (amax does not mind the zeros)
        extrema_group<GROUP, ASYM>(e, t);
        if (t == 0) {
            s_p = group_of<ASYM>(e, cols, bits);
            scales[row] = s_p.scale;
            if (zps) zps[row] = s_p.zp;
        }
        if constexpr (ASYM) __syncthreads();
        const FastGroup f = fast_of<ASYM>(e, bits, ASYM ? s_p.zp : 0.0);
        constexpr int H = (NV * EPV + 31) / 32;
        uint32_t redo[H] = {0};
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = t + i * GROUP;
            if (c >= nvec) break;
            float x[EPV];
            uint32_t word[EPV / 4];
            unpack16(v[i], static_cast<const T *>(nullptr), x);
            redo[i * EPV / 32] |= quant_words<ASYM, EPV>(x, f, word) << (i * EPV % 32);
            store_codes<EPV>(dst, c, word);
            if (f.exact) redo[i * EPV / 32] |= ((1u << EPV) - 1u) << (i * EPV % 32);
        }
        if constexpr (!ASYM) __syncthreads();
#pragma unroll
        for (int h = 0; h < H; ++h) {
#pragma unroll 1
            for (uint32_t left = redo[h]; left != 0; left &= left - 1) {
                const int k = h * 32 + lowest_bit(left);
                const size_t at = (size_t)(t + k / EPV * GROUP) * EPV + k % EPV;
                dst[at] = (int8_t)quant_ex(widen(src[at]), s_p);
            }
        }
    }
}

// Rows that are not whole aligned vectors: the same with NE elements per thread, consecutive threads on consecutive
// elements (a warp's loads are 32 elements, its stores 32 bytes).  GROUP = 32: a row per warp, else a row per CTA.
template <int GROUP, int NE, typename T, bool ASYM>
__global__ void __launch_bounds__(GROUP == 32 ? 256 : GROUP)
quantize_rows_elem_kernel(const T *__restrict__ w, size_t rows, size_t cols, int8_t *__restrict__ q, double *__restrict__ scales,
                          double *__restrict__ zps, int bits) {
    pdl_launch_dependents();
    pdl_wait();
    static_assert(NE <= 32, "one mask bit per element");
    constexpr int kRows = GROUP == 32 ? 8 : 1;  // rows per CTA
    const int t = threadIdx.x % GROUP;
    const size_t row = (size_t)blockIdx.x * kRows + threadIdx.x / GROUP;
    if (GROUP == 32 && row >= rows) return;
    const int n = (int)cols;
    const T *src = w + row * cols;
    int8_t *dst = q + row * cols;
    __shared__ GroupParams s_p[kRows];
    float v[NE];
    Extrema e = extrema_none<ASYM>();
#pragma unroll
    for (int i = 0; i < NE; ++i) {
        const int c = t + i * GROUP;
        v[i] = c < n ? storage_to_f32(__ldcs(src + c)) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < NE; ++i)
        if (!ASYM || t + i * GROUP < n) extrema_add<ASYM>(e, v[i]);
    GroupParams &p = s_p[threadIdx.x / GROUP];
    if constexpr (GROUP == 32) extrema_warp<ASYM>(e);
    else extrema_group<GROUP, ASYM>(e, t);
    if (t == 0) {
        p = group_of<ASYM>(e, cols, bits);
        scales[row] = p.scale;
        if (zps) zps[row] = p.zp;
    }
    if constexpr (ASYM) {
        if constexpr (GROUP == 32) __syncwarp();
        else __syncthreads();
    }
    const FastGroup f = fast_of<ASYM>(e, bits, ASYM ? p.zp : 0.0);
    uint32_t redo = f.exact ? ~0u : 0u;
#pragma unroll
    for (int i = 0; i < NE; ++i) {
        const int c = t + i * GROUP;
        uint32_t m;
        if (undecided<ASYM>(quant_candidate<ASYM>(v[i], f, m))) redo |= 1u << i;
        if (c < n) dst[c] = (int8_t)m;
    }
    if constexpr (!ASYM) {
        if constexpr (GROUP == 32) __syncwarp();
        else __syncthreads();
    }
#pragma unroll 1
    for (uint32_t left = redo; left != 0; left &= left - 1) {
        const int i = lowest_bit(left), c = t + i * GROUP;
        if (i < NE && c < n) dst[c] = (int8_t)quant_ex(widen(src[c]), p);
    }
}

// ---- per-channel, any shape (two passes, scalar accesses) ----------------------------
__global__ void __launch_bounds__(256)
quantize_rows_generic_kernel(const float *__restrict__ w, size_t rows, size_t cols,
                             int8_t *__restrict__ q, double *__restrict__ scales) {
    __shared__ float s_part[8];
    __shared__ RowParams s_p;
    for (size_t row = blockIdx.x; row < rows; row += gridDim.x) {
        const float *src = w + row * cols;
        float amax = 0.0f;
        for (size_t c = threadIdx.x; c < cols; c += blockDim.x) amax = fmaxf(amax, fabsf(src[c]));
        amax = warp_max(amax);
        if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = amax;
        __syncthreads();
        if (threadIdx.x == 0) {
            float m = 0.0f;
            for (int i = 0; i < 8; ++i) m = fmaxf(m, s_part[i]);
            double scale;
            RowParams pp;
            make_params(m, &scale, &pp);
            s_p = pp;
            scales[row] = scale;
        }
        __syncthreads();
        const RowParams p = s_p;
        int8_t *dst = q + row * cols;
        for (size_t c = threadIdx.x; c < cols; c += blockDim.x) dst[c] = (int8_t)quant_one(src[c], p);
        __syncthreads();  // s_part / s_p are reused by the next row
    }
}

// ---- per-tensor: amax over everything, then the element map --------------------------
// `amax_bits` is a zero-initialised word of scratch; non-negative floats order like their
// bit patterns, so atomicMax on the bits is a float max.
__global__ void __launch_bounds__(256)
absmax_flat_kernel(const float *__restrict__ w, size_t n, unsigned int *amax_bits) {
    float amax = 0.0f;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t nthreads = (size_t)gridDim.x * blockDim.x;
    const bool aligned = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
    const size_t nvec = aligned ? (n >> 2) : 0;
    const float4 *w4 = reinterpret_cast<const float4 *>(w);
    for (size_t i = tid; i < nvec; i += nthreads) amax = fmaxf(amax, abs4max(__ldg(w4 + i)));
    for (size_t i = (nvec << 2) + tid; i < n; i += nthreads) amax = fmaxf(amax, fabsf(w[i]));
    amax = warp_max(amax);
    __shared__ float s_part[8];
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = amax;
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = 0.0f;
        for (int i = 0; i < 8; ++i) m = fmaxf(m, s_part[i]);
        atomicMax(amax_bits, __float_as_uint(m));  // m is never NaN: fmaxf dropped them
    }
}

// Per-tensor in two launches.  Every block leaves the extrema of its contiguous part; the block that finishes last
// reduces them and forms the tensor's parameters, so no kernel of one thread sits between the passes.  The second pass leaves the
// counter at zero for the slot's next call, whatever calls that overlapped on other streams made of it.  The second pass takes the tensor from its end, where the
// first one stopped: that much of it may still be in L2.
constexpr int kMaxPartials = 2048;

struct TensorGroup {
    GroupParams p;
    FastGroup f;
    unsigned int arrived;
    alignas(16) Extrema partials[kMaxPartials];  // read as float2
};
static_assert(sizeof(Extrema) == 8, "an Extrema is two floats");

template <typename T, bool ASYM>
__global__ void __launch_bounds__(256)
extrema_partials_kernel(const T *__restrict__ w, size_t n, int bits, TensorGroup *g, double *__restrict__ scales,
                        double *__restrict__ zps) {
    // in this order: the second launch reads w before its own wait, so none of it may start before w is complete
    pdl_wait();
    pdl_launch_dependents();
    constexpr int EPV = Vec16<T>::kElems;
    __shared__ unsigned int s_last;
    Extrema e = extrema_none<ASYM>();
    const size_t nvec = (reinterpret_cast<uintptr_t>(w) & 15) == 0 ? n / EPV : 0;
    const uint4 *w4 = reinterpret_cast<const uint4 *>(w);
    const size_t stride = (size_t)gridDim.x * 256;
    size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    for (; i + 3 * stride < nvec; i += 4 * stride) {
        uint4 r[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) r[k] = __ldg(w4 + i + k * stride);
#pragma unroll
        for (int k = 0; k < 4; ++k) extrema_add16<T, ASYM>(e, r[k]);
    }
    for (; i < nvec; i += stride) extrema_add16<T, ASYM>(e, __ldg(w4 + i));
    for (size_t j = nvec * EPV + (size_t)blockIdx.x * 256 + threadIdx.x; j < n; j += (size_t)gridDim.x * 256)
        extrema_add<ASYM>(e, storage_to_f32(w[j]));
    extrema_group<256, ASYM>(e, threadIdx.x);
    if (threadIdx.x == 0) {
        g->partials[blockIdx.x] = e;
        __threadfence();
        s_last = gridDim.x == 1 || atomicAdd(&g->arrived, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    e = extrema_none<ASYM>();
    for (unsigned int k = threadIdx.x; k < gridDim.x; k += 256) {
        const float2 o = __ldcg(reinterpret_cast<const float2 *>(g->partials + k));
        extrema_merge<ASYM>(e, Extrema{o.x, o.y});
    }
    extrema_group<256, ASYM>(e, threadIdx.x);
    if (threadIdx.x == 0) {
        const GroupParams p = group_of<ASYM>(e, n, bits);
        g->p = p;
        g->f = fast_of<ASYM>(e, bits, p.zp);
        scales[0] = p.scale;
        if (zps) zps[0] = p.zp;
    }
}

// U vectors per thread, requested before the wait for the first launch (which does not write them); a block covers
// 256 * U consecutive vectors.
template <typename T, bool ASYM, int U>
__global__ void __launch_bounds__(256)
quantize_tensor_kernel(const T *__restrict__ w, size_t n, TensorGroup *g, int8_t *__restrict__ q) {
    pdl_launch_dependents();
    constexpr int EPV = Vec16<T>::kElems;
    const bool aligned = ((reinterpret_cast<uintptr_t>(w) & 15) == 0) && ((reinterpret_cast<uintptr_t>(q) & (EPV - 1)) == 0);
    const size_t nvec = aligned ? n / EPV : 0;
    const size_t first = (size_t)(gridDim.x - 1 - blockIdx.x) * (256 * U) + threadIdx.x;
    const uint4 *w4 = reinterpret_cast<const uint4 *>(w);
    uint4 r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) r[u] = first + u * 256 < nvec ? __ldcs(w4 + first + u * 256) : make_uint4(0, 0, 0, 0);
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) g->arrived = 0;
    const FastGroup f = g->f;
    const uint32_t all = f.exact ? (1u << EPV) - 1u : 0u;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const size_t at = first + u * 256;
        if (at >= nvec) break;
        float x[EPV];
        uint32_t word[EPV / 4];
        unpack16(r[u], static_cast<const T *>(nullptr), x);
        const uint32_t redo = quant_words<ASYM, EPV>(x, f, word) | all;
        store_codes<EPV>(q, at, word);
#pragma unroll 1
        for (uint32_t left = redo; left != 0; left &= left - 1) {
            const size_t j = at * EPV + lowest_bit(left);
            q[j] = (int8_t)quant_ex(widen(w[j]), g->p);
        }
    }
    for (size_t j = nvec * EPV + (size_t)blockIdx.x * 256 + threadIdx.x; j < n; j += (size_t)gridDim.x * 256) {
        uint32_t m;
        const float d = quant_candidate<ASYM>(storage_to_f32(w[j]), f, m);
        q[j] = all || undecided<ASYM>(d) ? (int8_t)quant_ex(widen(w[j]), g->p) : (int8_t)m;
    }
}

struct TensorParams {
    RowParams p;
};

// (an empty tensor has amax 0, which gives the reference's scale 1.0 of an empty slice, quantize.rs:340-342)
__global__ void finalize_tensor_scale_kernel(const unsigned int *amax_bits, double *scales, TensorParams *out) {
    double scale;
    RowParams p;
    make_params(__uint_as_float(*amax_bits), &scale, &p);
    scales[0] = scale;
    out->p = p;
}

__global__ void __launch_bounds__(256)
quantize_flat_kernel(const float *__restrict__ w, size_t n, const TensorParams *__restrict__ tp,
                     int8_t *__restrict__ q) {
    const RowParams p = tp->p;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t nthreads = (size_t)gridDim.x * blockDim.x;
    const bool aligned =
        ((reinterpret_cast<uintptr_t>(w) & 15) == 0) && ((reinterpret_cast<uintptr_t>(q) & 3) == 0);
    const size_t nvec = aligned ? (n >> 2) : 0;
    const float4 *w4 = reinterpret_cast<const float4 *>(w);
    uint32_t *q4 = reinterpret_cast<uint32_t *>(q);
    for (size_t i = tid; i < nvec; i += nthreads) {
        const float4 v = __ldcs(w4 + i);
        __stcs(q4 + i, pack4(quant_one(v.x, p), quant_one(v.y, p), quant_one(v.z, p), quant_one(v.w, p)));
    }
    for (size_t i = (nvec << 2) + tid; i < n; i += nthreads) q[i] = (int8_t)quant_one(w[i], p);
}

// ---- dequantize -----------------------------------------------------------------------
// out = narrow((q as f64 - 0.0) * scale): one f64 multiply per element, then a single
// rounding to the output type (quantize.rs:262-266, :320-335, :219-224).
__device__ __forceinline__ float dq_f32(int q, double s) { return (float)(((double)q - 0.0) * s); }

// f64 -> bf16 with one rounding: narrow to f32 toward zero, make it sticky (round to odd),
// then round the f32 to bf16 to nearest even.
__device__ __forceinline__ uint16_t f64_to_bf16_rne(double v) {
    if (v != v) return 0x7FC0;
    float f = __double2float_rz(v);
    uint32_t b = __float_as_uint(f);
    if ((double)f != v && !isinf(f)) b |= 1u;  // inexact: keep a sticky bit below bf16's ulp
    if (isinf(v)) return (uint16_t)(b >> 16);
    uint32_t rounded = b + 0x7FFFu + ((b >> 16) & 1u);
    return (uint16_t)(rounded >> 16);
}

// A code as f64 without the conversion pipe: the byte goes into the mantissa of 2^52 (u = q + 128), one subtraction leaves q.
__device__ __forceinline__ double code_f64(uint32_t biased_byte) {
    return __longlong_as_double((long long)(0x4330000000000000ull | biased_byte)) - 4503599627370624.0;  // 2^52 + 128
}

// Four codes of one scale -> four bf16.  The f32 product is off by less than 2 ulp of f32 and decides the rounding unless its
// low half lies within 8 of the midpoint 0x8000; a word with such an element, and every word under a scale that is
// not an ordinary f32 number, takes the f64 products and the sticky rounding.  Two elements at a time: the test adds 8 to
// both low halves and looks for a half that became 0x800? (a carry out of the lower half moves the upper one by 1, well
// inside the margin).  About 40 instructions a word against 90 with the elements one by one.
__device__ __forceinline__ unsigned long long dq4_bf16(uint32_t biased, double s) {
    const float f = (float)s;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __uint_as_float(__byte_perm(biased, 0x4B000000u, 0x7440 + j));  // 2^23 + q + 128
    add_f32x2(v[0], v[1], -8388736.0f, -8388736.0f);
    add_f32x2(v[2], v[3], -8388736.0f, -8388736.0f);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] *= f;
    uint32_t near = 0;
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
        const uint32_t low = __byte_perm(__float_as_uint(v[j]), __float_as_uint(v[j + 1]), 0x5410);
        const uint32_t h = ((low + 0x00080008u) & 0xFFF0FFF0u) ^ 0x80008000u;  // a zero half: near
        near |= (h - 0x00010001u) & ~h & 0x80008000u;
    }
    uint32_t lo = pack_bf16x2_rn(v[1], v[0]), hi = pack_bf16x2_rn(v[3], v[2]);
    if (near != 0 || !(f > 1e-30f && f < 1e30f)) {
        uint32_t h[2] = {0, 0};
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
            const uint32_t x = (uint32_t)f64_to_bf16_rne(code_f64((biased >> (8 * j)) & 0xFFu) * s) << (16 * (j & 1));
            if (j < 2) h[0] |= x;
            else h[1] |= x;
        }
        lo = h[0];
        hi = h[1];
    }
    return (unsigned long long)lo | ((unsigned long long)hi << 32);
}

// vec_ok: q is 4-byte and out 16-byte (f32) or 8-byte aligned.  A block takes 256 * U consecutive words of four codes at a
// time, U per thread with their loads in flight together, in flat order whatever the row length (a word may straddle
// rows).  The row of a word comes from 32-bit divisions where the tensor allows (a 64-bit division per word was a third
// of the instructions).  Blocks of consecutive words, as many as there are, rather than a grid that strides over the
// tensor: the stores of a block then fill whole DRAM pages.
template <typename OutT>
struct DequantWords {
    static constexpr int kPerThread = sizeof(OutT) == 4 ? 4 : 8;
};
template <typename OutT>
__global__ void __launch_bounds__(256)
dequantize_kernel(const int8_t *__restrict__ q, const double *__restrict__ scales, size_t rows,
                  size_t cols, int per_channel, OutT *__restrict__ out, int vec_ok) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t n = rows * cols;
    size_t done = 0;
    if (vec_ok && (!per_channel || cols >= 4)) {
        constexpr int U = DequantWords<OutT>::kPerThread;
        const size_t nvec = n >> 2;
        done = nvec << 2;
        const uint32_t *q4 = reinterpret_cast<const uint32_t *>(q);
        const uint32_t width = per_channel ? (uint32_t)(cols < 0xFFFFFFFFull ? cols : 0xFFFFFFFFull) : 0xFFFFFFFFu;
        const uint32_t drow = 1024u / width, dcol = 1024u - drow * width;
        for (size_t first = (size_t)blockIdx.x * (256 * U) + threadIdx.x; first < nvec; first += (size_t)gridDim.x * (256 * U)) {
            uint32_t b[U];
#pragma unroll
            for (int u = 0; u < U; ++u) b[u] = first + u * 256 < nvec ? __ldcs(q4 + first + u * 256) ^ 0x80808080u : 0u;
            size_t row = 0, col = 0;
            if (per_channel) {
                const size_t e = first << 2;
                if (n <= 0xFFFFFFFFull) {
                    row = (uint32_t)e / width;
                    col = (uint32_t)e - (uint32_t)row * width;
                } else {
                    row = e / cols;
                    col = e - row * cols;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const size_t i = first + u * 256;
                if (i >= nvec) break;
                const double s0 = __ldg(scales + row);
                if (per_channel && cols - col < 4) {
                    // the elements of this word beyond the row's end belong to the next row
                    const int split = (int)(cols - col);
                    const double s1 = __ldg(scales + row + 1);
#pragma unroll 1
                    for (int j = 0; j < 4; ++j) {
                        const double v = code_f64((b[u] >> (8 * j)) & 0xFFu) * (split > j ? s0 : s1);
                        if constexpr (sizeof(OutT) == 4) out[4 * i + j] = (float)v;
                        else out[4 * i + j] = f64_to_bf16_rne(v);
                    }
                } else if constexpr (sizeof(OutT) == 4) {
                    __stcs(reinterpret_cast<float4 *>(out) + i,
                           make_float4((float)(code_f64(b[u] & 0xFFu) * s0), (float)(code_f64((b[u] >> 8) & 0xFFu) * s0),
                                       (float)(code_f64((b[u] >> 16) & 0xFFu) * s0), (float)(code_f64(b[u] >> 24) * s0)));
                } else {
                    __stcs(reinterpret_cast<unsigned long long *>(out) + i, dq4_bf16(b[u], s0));
                }
                if (per_channel) {
                    row += drow;
                    col += dcol;
                    if (col >= cols) {
                        col -= cols;
                        row += 1;
                    }
                }
            }
        }
    }
    for (size_t i = done + (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
        const double s = per_channel ? scales[i / cols] : scales[0];
        const int v = (int)q[i];
        if constexpr (sizeof(OutT) == 4)
            out[i] = dq_f32(v, s);
        else
            out[i] = f64_to_bf16_rne((double)v * s);
    }
}

// f64 scales -> f32 per-row scales used by the forward kernels (per-tensor is broadcast).
__global__ void scales_to_f32_kernel(const double *__restrict__ scales, int per_channel, size_t n,
                                     float *__restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)(per_channel ? scales[i] : scales[0]);
}

// x = hi + lo with hi = bf16(x), lo = bf16(x - hi): two bf16 matrices whose sum carries ~16
// significand bits of the f32 activations (relative error ~2^-17), so two tensor-core passes
// over exact bf16 x int8 products stay inside the 1e-4 tolerance of the f32 path.
__global__ void __launch_bounds__(256)
split_f32_kernel(const float *__restrict__ x, size_t n, __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float v = x[i];
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        hi[i] = h;
        lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
    }
}

}  // namespace
}  // namespace shrewq
