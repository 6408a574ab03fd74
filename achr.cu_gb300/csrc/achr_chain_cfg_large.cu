// Chain-kernel instantiations with 256 to 512 threads per chain.
#include "achr_chain_kernel.cuh"

namespace achr {

cudaError_t launch_chain_cfg_large(int bd, int ept, const ChainArgs &a, cudaStream_t s, int max_ctas, ChainFit *fit) {
    switch (bd * 100 + ept) {
        case 256 * 100 + 4: return launch_cfg<256, 4>(a, s, max_ctas, fit);
        case 256 * 100 + 8: return launch_cfg<256, 8>(a, s, max_ctas, fit);
        case 256 * 100 + 16: return launch_cfg<256, 16>(a, s, max_ctas, fit);
        case 256 * 100 + 18: return launch_cfg<256, 18>(a, s, max_ctas, fit);
        case 256 * 100 + 20: return launch_cfg<256, 20>(a, s, max_ctas, fit);
        case 256 * 100 + 24: return launch_cfg<256, 24>(a, s, max_ctas, fit);
        case 256 * 100 + 26: return launch_cfg<256, 26>(a, s, max_ctas, fit);
        case 256 * 100 + 30: return launch_cfg<256, 30>(a, s, max_ctas, fit);
        case 320 * 100 + 12: return launch_cfg<320, 12>(a, s, max_ctas, fit);
        case 384 * 100 + 10: return launch_cfg<384, 10>(a, s, max_ctas, fit);
        case 384 * 100 + 20: return launch_cfg<384, 20>(a, s, max_ctas, fit);
        case 512 * 100 + 4: return launch_cfg<512, 4>(a, s, max_ctas, fit);
        case 512 * 100 + 8: return launch_cfg<512, 8>(a, s, max_ctas, fit);
        case 512 * 100 + 12: return launch_cfg<512, 12>(a, s, max_ctas, fit);
        case 512 * 100 + 16: return launch_cfg<512, 16>(a, s, max_ctas, fit);
        case 512 * 100 + 32: return launch_cfg<512, 32>(a, s, max_ctas, fit);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_chain_queue_large(int bd, int ept, const ChainQueue &q, cudaStream_t s, int grid, int *per_sm) {
    switch (bd * 100 + ept) {
        case 256 * 100 + 4: return launch_queue_cfg<256, 4>(q, s, grid, per_sm);
        case 256 * 100 + 8: return launch_queue_cfg<256, 8>(q, s, grid, per_sm);
        case 256 * 100 + 16: return launch_queue_cfg<256, 16>(q, s, grid, per_sm);
        case 256 * 100 + 18: return launch_queue_cfg<256, 18>(q, s, grid, per_sm);
        case 256 * 100 + 20: return launch_queue_cfg<256, 20>(q, s, grid, per_sm);
        case 256 * 100 + 24: return launch_queue_cfg<256, 24>(q, s, grid, per_sm);
        case 256 * 100 + 26: return launch_queue_cfg<256, 26>(q, s, grid, per_sm);
        case 256 * 100 + 30: return launch_queue_cfg<256, 30>(q, s, grid, per_sm);
        case 320 * 100 + 12: return launch_queue_cfg<320, 12>(q, s, grid, per_sm);
        case 384 * 100 + 10: return launch_queue_cfg<384, 10>(q, s, grid, per_sm);
        case 384 * 100 + 20: return launch_queue_cfg<384, 20>(q, s, grid, per_sm);
        case 512 * 100 + 4: return launch_queue_cfg<512, 4>(q, s, grid, per_sm);
        case 512 * 100 + 8: return launch_queue_cfg<512, 8>(q, s, grid, per_sm);
        case 512 * 100 + 12: return launch_queue_cfg<512, 12>(q, s, grid, per_sm);
        case 512 * 100 + 16: return launch_queue_cfg<512, 16>(q, s, grid, per_sm);
        case 512 * 100 + 32: return launch_queue_cfg<512, 32>(q, s, grid, per_sm);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace achr
