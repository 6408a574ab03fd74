// Chain-kernel instantiations with 32 and 64 threads per chain.
#include "achr_chain_kernel.cuh"

namespace achr {

cudaError_t launch_chain_cfg_small(int bd, int ept, const ChainArgs &a, cudaStream_t s, int max_ctas, ChainFit *fit) {
    switch (bd * 100 + ept) {
        case 32 * 100 + 4: return launch_cfg<32, 4>(a, s, max_ctas, fit);
        case 32 * 100 + 8: return launch_cfg<32, 8>(a, s, max_ctas, fit);
        case 64 * 100 + 4: return launch_cfg<64, 4>(a, s, max_ctas, fit);
        case 64 * 100 + 6: return launch_cfg<64, 6>(a, s, max_ctas, fit);
        case 64 * 100 + 8: return launch_cfg<64, 8>(a, s, max_ctas, fit);
        case 64 * 100 + 12: return launch_cfg<64, 12>(a, s, max_ctas, fit);
        case 64 * 100 + 16: return launch_cfg<64, 16>(a, s, max_ctas, fit);
        case 64 * 100 + 20: return launch_cfg<64, 20>(a, s, max_ctas, fit);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_chain_queue_small(int bd, int ept, const ChainQueue &q, cudaStream_t s, int grid, int *per_sm) {
    switch (bd * 100 + ept) {
        case 32 * 100 + 4: return launch_queue_cfg<32, 4>(q, s, grid, per_sm);
        case 32 * 100 + 8: return launch_queue_cfg<32, 8>(q, s, grid, per_sm);
        case 64 * 100 + 4: return launch_queue_cfg<64, 4>(q, s, grid, per_sm);
        case 64 * 100 + 6: return launch_queue_cfg<64, 6>(q, s, grid, per_sm);
        case 64 * 100 + 8: return launch_queue_cfg<64, 8>(q, s, grid, per_sm);
        case 64 * 100 + 12: return launch_queue_cfg<64, 12>(q, s, grid, per_sm);
        case 64 * 100 + 16: return launch_queue_cfg<64, 16>(q, s, grid, per_sm);
        case 64 * 100 + 20: return launch_queue_cfg<64, 20>(q, s, grid, per_sm);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace achr
