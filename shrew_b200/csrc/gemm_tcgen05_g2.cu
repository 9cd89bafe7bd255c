// The tcgen05 forward with 2 converter groups.
#include "gemm_tcgen05_launch.cuh"

namespace shrewq {

int launch_tcgen05_groups2(shrewq_ctx *ctx, const ForwardArgs &a, int tok, const CUtensorMap &tw, const CUtensorMap &tw2, void *fs, size_t fsb) {
    return launch_groups<2>(ctx, a, tok, tw, tw2, fs, fsb);
}

}  // namespace shrewq
