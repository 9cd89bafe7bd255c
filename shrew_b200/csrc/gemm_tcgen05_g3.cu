// The tcgen05 forward with 3 converter groups.
#include "gemm_tcgen05_launch.cuh"

namespace shrewq {

#ifdef SHREWQ_TRACE
extern "C" __attribute__((visibility("default"))) int shrewq_debug_set_trace(long long *dev_buf) {
    return (int)cudaMemcpyToSymbol(g_trace, &dev_buf, sizeof(dev_buf));
}
#endif

int launch_tcgen05_groups3(shrewq_ctx *ctx, const ForwardArgs &a, int tok, const CUtensorMap &tw, const CUtensorMap &tw2, void *fs, size_t fsb) {
    return launch_groups<3>(ctx, a, tok, tw, tw2, fs, fsb);
}

}  // namespace shrewq
