// CPU run of the persistent f32-activation forward (shrew_b200/csrc/gemm_tcgen05_f32_kernels.cuh), set up as launch_f32
// in shrew_b200/csrc/gemm_tcgen05_f32.cu does; the caller chooses the token tile and how many CTAs share the tiles.
// TEST INFRASTRUCTURE ONLY; see cuda_shim.h.
#include "cuda_shim.h"
#include "cuda_shim_tcgen05.h"
#include "../../shrew_b200/csrc/gemm_tcgen05_f32_kernels.cuh"

using namespace shrewq;

template <int TOK, int XKB>
static int run(const int8_t *q, const float *scales, const float *bias, const float *x, float *y, int M, int N, int K, size_t ldy,
               int epilogue, int ctas) {
    using C = F32Cfg<TOK, XKB>;
    const CUtensorMap tw{q, 1, (uint64_t)K, (uint64_t)N, (uint64_t)K, (uint32_t)kF32BlockK, 128, 64};
    const int n_tiles = (N + kF32Chan - 1) / kF32Chan, tiles = n_tiles * ((M + TOK - 1) / TOK);
    const int resident = K <= C::kXSlots * kF32BlockK;
    if (ctas > tiles) ctas = tiles;
    DeviceStatus st{0, 0, 0, 0};
    emu::g_failed = false;
    emu::launch3((unsigned)ctas, 1, 1, kF32Threads, C::kSmemBytes, [&] {
        linear_i8_tcgen05_f32_kernel<TOK, XKB>(tw, scales, bias, x, y, M, N, K, ldy, epilogue, n_tiles, tiles, resident, &st);
    });
    if (emu::g_failed) return -4;
    return st.timeout_flag ? -2 : 0;
}

// x: f32 [M,K]; y: f32 [M, ldy].  Returns 0; -2 when a bounded wait gave up; -4 when a rule of the model was violated.
extern "C" int emu_gemm_tcgen05_f32(const int8_t *q, const float *scales, const float *bias, const float *x, float *y, int M, int N,
                                    int K, size_t ldy, int epilogue, int tok, int ctas) {
    // shared memory for activations as launch_gemm_tcgen05_f32 chooses it
    if (tok == 128) return K <= 256 && ldy % 8 == 0 ? run<128, 128>(q, scales, bias, x, y, M, N, K, ldy, epilogue, ctas) : run<128, 192>(q, scales, bias, x, y, M, N, K, ldy, epilogue, ctas);
    return K <= 512 ? run<64, 128>(q, scales, bias, x, y, M, N, K, ldy, epilogue, ctas) : run<64, 192>(q, scales, bias, x, y, M, N, K, ldy, epilogue, ctas);
}

extern "C" void emu_drop_tma(int n) {
    emu::g_drop_tma = n;
    emu::g_tma_count = 0;
}
extern "C" void emu_tma_async(unsigned seed, unsigned one_in) {
    emu::g_tma_async_seed = seed;
    emu::g_tma_one_in = one_in ? one_in : 8;
}
extern "C" const char *emu_fail_message() { return emu::g_failed ? emu::g_fail_msg : ""; }
