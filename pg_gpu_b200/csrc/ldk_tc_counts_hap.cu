// Haplotype populations of more than kSpinMaxN: statistics from counts, the wider tile.
#include "ldk_tc_kernel.cuh"

namespace ldk {
cudaError_t launch_tc_counts_hap(const ldk_parse_t* d, const ldk_parse_out_t* o, const Scratch& w, const ParseShape& sh,
                                 int max_items, int variant, cudaStream_t s) {
    if (variant != 0) return cudaErrorInvalidConfiguration;
    return dispatch_tc<false, 0, true>(d, o, w, sh, max_items, s);
}
}  // namespace ldk
