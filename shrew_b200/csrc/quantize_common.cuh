// What every quantizer shares (sm_100a): the reference's parameter and element arithmetic in f64, and the f32
// shortcut that gives the same codes.
//
// Reference semantics (crates/shrew/src/quantize.rs), all in f64 on a widened copy of the tensor:
//   qmax = 127 | 7;  qmin = -127 | -7 (symmetric), -128 | -8 (asymmetric)          (:124-139)
//   symmetric : scale = amax < 1e-30 ? 1 : amax / qmax,  zp = 0                     (:349-352)
//   asymmetric: range = max - min;  scale = range < 1e-30 ? 1 : range / (qmax - qmin);
//               zp = round(qmin - min / scale)                                      (:353-364)
//   inv  = |scale| < 1e-30 ? 0 : 1 / scale                                          (:236-240)
//   code = clamp(round_half_away(v * inv + zp), qmin, qmax) as i8   (NaN -> 0)      (:244-250)
//
// The shortcut.  f32, bf16 and f16 elements are exact in f32, and so are their extrema.  t = v * inv32 (+ zp) in f32 is
// off the f64 value by at most 127 * 2^-23 ~ 1.5e-5 (symmetric, |t| <= 127) or 1.3e-4 (asymmetric with |zp| <= 256:
// |v * inv| <= 512 and the sum is rounded once).  Adding 1.5 * 2^23 rounds t to the nearest integer and leaves it in
// the low mantissa bits as a two's complement byte; subtracting the constant again gives the rounded value r, and
// |t - r| <= 0.5 - window says that no rounding boundary lies within the window, so every way of rounding gives
// that integer (which also lies inside [qmin, qmax] then: a value past the end would have to be within the window of
// the boundary qmax + 0.5).  Elements inside the window, NaN (the comparison is false), and all elements of
// a group without an ordinary reciprocal (infinities, scales near 1e-30, large zero points) take the f64 operations one
// for one.  About eight instructions an element against about twenty with compares, truncations and conversions:
// 8192 x 8192 f32 was bound by instruction issue as much as by memory.
//
// Device code only (no launch syntax, no runtime calls): it also compiles as plain C++ against the CUDA stand-in of the
// CPU tests (tests/cpu_emu/).
#pragma once

#include "../../include/shrewq.h"
#ifndef SHREWQ_CPU_EMU
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#endif

namespace shrewq {
namespace {

struct GroupParams {
    double scale, zp, inv, qmin, qmax;
};

__device__ __forceinline__ double qmax_of(int bits) { return bits == 4 ? 7.0 : 127.0; }
__device__ __forceinline__ double qmin_of(int bits, int mode) {
    if (bits == 4) return mode == SHREWQ_ASYMMETRIC ? -8.0 : -7.0;
    return mode == SHREWQ_ASYMMETRIC ? -128.0 : -127.0;
}

__device__ __forceinline__ double round_half_away(double t) {
    if (t != t) return t;
    double r = trunc(t);
    if (fabs(t - r) >= 0.5) r += copysign(1.0, t);  // t - r is exact; false for +-Inf (NaN compare)
    return copysign(r, t);                          // round(-0.3) is -0.0, as f64::round
}

// Tensor element -> f64, exactly (Tensor::to_f64_vec, quantize.rs:198): f32, f64, bf16 or f16 storage.
__device__ __forceinline__ double widen(float v) { return (double)v; }
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double widen(__nv_bfloat16 v) { return (double)__bfloat162float(v); }
__device__ __forceinline__ double widen(__half v) { return (double)__half2float(v); }

// compute_scale_zp for a group of n elements whose extrema are lo / hi / amax (f64: exact for every
// storage type)
__device__ __forceinline__ GroupParams make_group(double lo, double hi, double amax, size_t n, int bits, int mode) {
    GroupParams p;
    p.qmin = qmin_of(bits, mode);
    p.qmax = qmax_of(bits);
    if (n == 0) {
        p.scale = 1.0;
        p.zp = 0.0;
    } else if (mode != SHREWQ_ASYMMETRIC) {
        p.scale = amax < 1e-30 ? 1.0 : amax / p.qmax;
        p.zp = 0.0;
    } else {
        const double range = hi - lo;
        p.scale = range < 1e-30 ? 1.0 : range / (p.qmax - p.qmin);
        p.zp = round_half_away(p.qmin - lo / p.scale);
    }
    p.inv = fabs(p.scale) < 1e-30 ? 0.0 : 1.0 / p.scale;
    return p;
}

__device__ __forceinline__ int quant_ex(double v, const GroupParams &p) {
    const double t = round_half_away(__dadd_rn(__dmul_rn(v, p.inv), p.zp));
    if (t != t) return 0;  // NaN as i8 == 0
    return (int)fmin(fmax(t, p.qmin), p.qmax);
}

// ---- the f32 shortcut --------------------------------------------------------------------------------------------
// The extrema of a group of f32 / bf16 / f16 elements: exact in f32.  Symmetric groups use hi for amax.
struct Extrema {
    float lo, hi;
};

struct FastGroup {
    float inv, zp;
    int exact;  // 1: no ordinary reciprocal, every element takes the f64 operations
};

constexpr float kRoundMagic = 12582912.0f;                  // 1.5 * 2^23
constexpr float kSafeSym = 0.5f - 1e-4f, kSafeAsym = 0.5f - 2.5e-4f;

__device__ __forceinline__ bool warp_any(bool v) {
#ifdef SHREWQ_CPU_EMU
    int a = v ? 1 : 0;
    for (int o = 16; o > 0; o >>= 1) a |= __shfl_xor_sync(0xFFFFFFFFu, a, o);
    return a != 0;
#else
    return __any_sync(0xFFFFFFFFu, v) != 0;
#endif
}

__device__ __forceinline__ int lowest_bit(uint32_t v) {
#ifdef SHREWQ_CPU_EMU
    return __builtin_ctz(v);
#else
    return __ffs((int)v) - 1;
#endif
}

template <bool ASYM>
__device__ __forceinline__ GroupParams group_of(const Extrema &e, size_t n, int bits) {
    return make_group((double)e.lo, (double)e.hi, (double)e.hi, n, bits, ASYM ? SHREWQ_ASYMMETRIC : SHREWQ_SYMMETRIC);
}

// inv to f32 precision from the extrema; zp_known: the f64 zero point (asymmetric)
template <bool ASYM>
__device__ __forceinline__ FastGroup fast_of(const Extrema &e, int bits, double zp_known) {
    FastGroup f;
    f.zp = 0.0f;
    const float top = bits == 4 ? 7.0f : 127.0f;
    if constexpr (ASYM) {
        const float range = e.hi - e.lo, steps = bits == 4 ? 15.0f : 255.0f;
        f.exact = !(range >= 1e-26f && range <= 3e38f && fabs(zp_known) <= 256.0);
        f.inv = steps / range;
        f.zp = (float)zp_known;
    } else {
        // amax < 1e-30 has scale 1 (and codes 0); from 1e-26 on scale and reciprocal are ordinary; in between the f64 code decides
        const bool tiny = e.hi < 1e-30f;
        f.exact = !(tiny || (e.hi >= 1e-26f && e.hi <= 3e38f));
        f.inv = tiny ? 1.0f : top / e.hi;
    }
    return f;
}

// One element's f32 candidate: m holds the code in its low byte; returns |t - r| (NaN for NaN).
template <bool ASYM>
__device__ __forceinline__ float quant_candidate(float v, const FastGroup &f, uint32_t &m) {
    const float t = ASYM ? fmaf(v, f.inv, f.zp) : v * f.inv;
    const float a = t + kRoundMagic;
    m = __float_as_uint(a);
    return fabsf(t - (a - kRoundMagic));
}
template <bool ASYM>
__device__ __forceinline__ bool undecided(float d) { return !(d <= (ASYM ? kSafeAsym : kSafeSym)); }

__device__ __forceinline__ uint32_t pack_low_bytes(const uint32_t *m) {
    return __byte_perm(__byte_perm(m[0], m[1], 0x0040), __byte_perm(m[2], m[3], 0x0040), 0x5410);
}

// Codes of N elements (a multiple of 4) as words; bit j of the result: element j is undecided.
template <bool ASYM, int N>
__device__ __forceinline__ uint32_t quant_words(const float *x, const FastGroup &f, uint32_t *word) {
    uint32_t redo = 0;
#pragma unroll
    for (int k = 0; k < N / 4; ++k) {
        uint32_t m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (undecided<ASYM>(quant_candidate<ASYM>(x[4 * k + j], f, m[j]))) redo |= 1u << (4 * k + j);
        word[k] = pack_low_bytes(m);
    }
    return redo;
}

// ---- 16-byte vectors of a storage type ---------------------------------------------------------------------------
template <typename T>
struct Vec16 {
    static constexpr int kElems = 16 / (int)sizeof(T);
};
__device__ __forceinline__ float storage_to_f32(float v) { return v; }
__device__ __forceinline__ float storage_to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float storage_to_f32(__half v) { return __half2float(v); }

__device__ __forceinline__ void unpack16(const uint4 &r, const float *, float *o) {
    o[0] = __uint_as_float(r.x);
    o[1] = __uint_as_float(r.y);
    o[2] = __uint_as_float(r.z);
    o[3] = __uint_as_float(r.w);
}
__device__ __forceinline__ void unpack16(const uint4 &r, const __nv_bfloat16 *, float *o) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o[2 * i] = __uint_as_float(w[i] << 16);
        o[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
}
__device__ __forceinline__ float f16_bits_to_f32(uint32_t b) {
    const uint16_t h = (uint16_t)b;
    __half v;
    memcpy(&v, &h, 2);
    return __half2float(v);
}
__device__ __forceinline__ void unpack16(const uint4 &r, const __half *, float *o) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o[2 * i] = f16_bits_to_f32(w[i] & 0xFFFFu);
        o[2 * i + 1] = f16_bits_to_f32(w[i] >> 16);
    }
}

template <bool ASYM>
__device__ __forceinline__ Extrema extrema_none() {
    Extrema e;
    e.lo = ASYM ? INFINITY : 0.0f;
    e.hi = ASYM ? -INFINITY : 0.0f;
    return e;
}
// (fminf / fmaxf drop a NaN operand, as f64::min / f64::max do in the reference's folds)
template <bool ASYM>
__device__ __forceinline__ void extrema_add(Extrema &e, float v) {
    if constexpr (ASYM) {
        e.lo = fminf(e.lo, v);
        e.hi = fmaxf(e.hi, v);
    } else {
        e.hi = fmaxf(e.hi, fabsf(v));
    }
}
template <typename T, bool ASYM>
__device__ __forceinline__ void extrema_add16(Extrema &e, const uint4 &r) {
    float x[Vec16<T>::kElems];
    unpack16(r, static_cast<const T *>(nullptr), x);
#pragma unroll
    for (int j = 0; j < Vec16<T>::kElems; ++j) extrema_add<ASYM>(e, x[j]);
}
#ifndef SHREWQ_CPU_EMU
// amax of the 16-bit types two elements at a time (the packed maximum drops a NaN operand too)
template <>
__device__ __forceinline__ void extrema_add16<__nv_bfloat16, false>(Extrema &e, const uint4 &r) {
    __nv_bfloat162 v[4];
    memcpy(v, &r, 16);
    const __nv_bfloat162 m = __hmax2(__hmax2(__habs2(v[0]), __habs2(v[1])), __hmax2(__habs2(v[2]), __habs2(v[3])));
    e.hi = fmaxf(e.hi, fmaxf(__low2float(m), __high2float(m)));
}
template <>
__device__ __forceinline__ void extrema_add16<__half, false>(Extrema &e, const uint4 &r) {
    __half2 v[4];
    memcpy(v, &r, 16);
    const __half2 m = __hmax2(__hmax2(__habs2(v[0]), __habs2(v[1])), __hmax2(__habs2(v[2]), __habs2(v[3])));
    e.hi = fmaxf(e.hi, fmaxf(__low2float(m), __high2float(m)));
}
#endif
template <bool ASYM>
__device__ __forceinline__ void extrema_merge(Extrema &e, const Extrema &o) {
    if constexpr (ASYM) e.lo = fminf(e.lo, o.lo);
    e.hi = fmaxf(e.hi, o.hi);
}
template <bool ASYM>
__device__ __forceinline__ void extrema_warp(Extrema &e) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if constexpr (ASYM) e.lo = fminf(e.lo, __shfl_xor_sync(0xFFFFFFFFu, e.lo, o));
        e.hi = fmaxf(e.hi, __shfl_xor_sync(0xFFFFFFFFu, e.hi, o));
    }
}

// codes of one 16-byte vector to dst[EPV * c ...]
template <int EPV>
__device__ __forceinline__ void store_codes(int8_t *dst, size_t c, const uint32_t *word) {
    if constexpr (EPV == 4)
        __stcs(reinterpret_cast<unsigned int *>(dst) + c, word[0]);
    else
        __stcs(reinterpret_cast<unsigned long long *>(dst) + c, (unsigned long long)word[0] | ((unsigned long long)word[1] << 32));
}

// R rows of one matrix by one warp, NV vectors per lane and row: read once, all loads in flight together, the
// reductions of the rows interleaved and their f64 parameters formed by R lanes side by side (a row costs two f64
// divisions, which for a short row is most of the arithmetic: 16384 x 128 took 8.1 us with a row per warp).
// Undecided elements are redone in f64 from memory, one at a time; half-way codes are rare in f32 weights and
// about one in 200 in bf16 ones, whose few significant bits meet the boundaries exactly.
template <int R, int NV, typename T, bool ASYM>
__device__ __forceinline__ void quantize_rows_by_warp(const T *src, size_t cols, int count, int bits, int8_t *dst, double *scales,
                                                      double *zps, int lane) {
    constexpr int EPV = Vec16<T>::kElems;
    const int nvec = (int)(cols / EPV);
    uint4 v[R][NV];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = lane + 32 * i;
            v[r][i] = r < count && c < nvec ? __ldcs(reinterpret_cast<const uint4 *>(src + r * cols) + c) : make_uint4(0, 0, 0, 0);
        }
    Extrema e[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        e[r] = extrema_none<ASYM>();
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (!ASYM || lane + 32 * i < nvec) extrema_add16<T, ASYM>(e[r], v[r][i]);  // (amax does not mind the zeros)
    }
#pragma unroll
    for (int r = 0; r < R; ++r) extrema_warp<ASYM>(e[r]);
    Extrema mine = e[0];
#pragma unroll
    for (int r = 1; r < R; ++r)
        if (lane == r) mine = e[r];
    const GroupParams p = group_of<ASYM>(mine, cols, bits);  // lane r: row r
    if (lane < count) {
        scales[lane] = p.scale;
        if (zps) zps[lane] = p.zp;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const double zp = ASYM ? __shfl_sync(0xFFFFFFFFu, p.zp, r) : 0.0;
        if (r >= count) break;
        const FastGroup f = fast_of<ASYM>(e[r], bits, zp);
        uint32_t redo[(NV * EPV + 31) / 32] = {0};
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = lane + 32 * i;
            if (c >= nvec) break;
            float x[EPV];
            uint32_t word[EPV / 4];
            unpack16(v[r][i], static_cast<const T *>(nullptr), x);
            redo[i * EPV / 32] |= quant_words<ASYM, EPV>(x, f, word) << (i * EPV % 32);
            store_codes<EPV>(dst + r * cols, c, word);
            if (f.exact) redo[i * EPV / 32] |= ((1u << EPV) - 1u) << (i * EPV % 32);
        }
        bool some = false;
#pragma unroll
        for (int h = 0; h < (NV * EPV + 31) / 32; ++h) some = some || redo[h] != 0;
        if (warp_any(some)) {
            GroupParams pr = p;
            pr.inv = __shfl_sync(0xFFFFFFFFu, p.inv, r);
            pr.zp = zp;
#pragma unroll
            for (int h = 0; h < (NV * EPV + 31) / 32; ++h) {
#pragma unroll 1
                for (uint32_t bitsleft = redo[h]; bitsleft != 0; bitsleft &= bitsleft - 1) {
                    const int k = h * 32 + lowest_bit(bitsleft);
                    const size_t at = r * cols + (size_t)(lane + 32 * (k / EPV)) * EPV + k % EPV;
                    dst[at] = (int8_t)quant_ex(widen(src[at]), pr);
                }
            }
        }
    }
}

}  // namespace
}  // namespace shrewq
