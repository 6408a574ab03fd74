// Chain-kernel instantiations with 128 threads per chain.
#include "achr_chain_kernel.cuh"

namespace achr {

cudaError_t launch_chain_cfg_mid(int bd, int ept, const ChainArgs &a, cudaStream_t s, int max_ctas, ChainFit *fit) {
    switch (bd * 100 + ept) {
        case 128 * 100 + 4: return launch_cfg<128, 4>(a, s, max_ctas, fit);
        case 128 * 100 + 8: return launch_cfg<128, 8>(a, s, max_ctas, fit);
        case 128 * 100 + 12: return launch_cfg<128, 12>(a, s, max_ctas, fit);
        case 128 * 100 + 16: return launch_cfg<128, 16>(a, s, max_ctas, fit);
        case 128 * 100 + 20: return launch_cfg<128, 20>(a, s, max_ctas, fit);
        case 128 * 100 + 24: return launch_cfg<128, 24>(a, s, max_ctas, fit);
        case 128 * 100 + 32: return launch_cfg<128, 32>(a, s, max_ctas, fit);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_chain_queue_mid(int bd, int ept, const ChainQueue &q, cudaStream_t s, int grid, int *per_sm) {
    switch (bd * 100 + ept) {
        case 128 * 100 + 4: return launch_queue_cfg<128, 4>(q, s, grid, per_sm);
        case 128 * 100 + 8: return launch_queue_cfg<128, 8>(q, s, grid, per_sm);
        case 128 * 100 + 12: return launch_queue_cfg<128, 12>(q, s, grid, per_sm);
        case 128 * 100 + 16: return launch_queue_cfg<128, 16>(q, s, grid, per_sm);
        case 128 * 100 + 20: return launch_queue_cfg<128, 20>(q, s, grid, per_sm);
        case 128 * 100 + 24: return launch_queue_cfg<128, 24>(q, s, grid, per_sm);
        case 128 * 100 + 32: return launch_queue_cfg<128, 32>(q, s, grid, per_sm);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace achr
