// Dispatcher of the chain kernel's configurations (the ladder and its rules: achr_chain_rule.h).
#include "achr_internal.h"

namespace achr {

cudaError_t launch_chain_cfg_small(int bd, int ept, const ChainArgs &a, cudaStream_t s, int max_ctas, ChainFit *fit);
cudaError_t launch_chain_cfg_large(int bd, int ept, const ChainArgs &a, cudaStream_t s, int max_ctas, ChainFit *fit);
cudaError_t launch_chain_cfg_mid(int bd, int ept, const ChainArgs &a, cudaStream_t s, int max_ctas, ChainFit *fit);
cudaError_t launch_chain_queue_small(int bd, int ept, const ChainQueue &q, cudaStream_t s, int grid, int *per_sm);
cudaError_t launch_chain_queue_mid(int bd, int ept, const ChainQueue &q, cudaStream_t s, int grid, int *per_sm);
cudaError_t launch_chain_queue_large(int bd, int ept, const ChainQueue &q, cudaStream_t s, int grid, int *per_sm);

namespace {

cudaError_t launch_cfg_of(const ChainCfg &c, const ChainArgs &a, cudaStream_t stream, int max_ctas, ChainFit *fit) {
    if (c.bd <= 64) return launch_chain_cfg_small(c.bd, c.ept, a, stream, max_ctas, fit);
    if (c.bd <= 128) return launch_chain_cfg_mid(c.bd, c.ept, a, stream, max_ctas, fit);
    return launch_chain_cfg_large(c.bd, c.ept, a, stream, max_ctas, fit);
}

// The default for a model that reprojects through the residual in the kernel:
// the first configuration, from its length's default on, in which z has room.
// Reprojecting as N (N^T x) instead costs 4 n d FP64 operations, 11 ms of an SM
// at 5063 x 7440 against a step's 23 K clocks.  The form and its turns (*turn; 0:
// no configuration has room) do not depend on the number of chains.
cudaError_t find_cfg_residual(const ChainArgs &a, const ChainCfg **out, int *turn) {
    const int scratch = a.m > a.d ? a.m : a.d;
    const ChainCfg *dflt = *out = find_cfg(a.n, 0, scratch);
    *turn = 0;
    if (!dflt) return cudaSuccess;
    ChainArgs q = a;
    q.P = 0;  // (asks for the residency only)
    for (const ChainCfg *c = dflt; c != kLadder + sizeof(kLadder) / sizeof(kLadder[0]); ++c) {
        if (c->bd * c->ept > a.np) continue;
        if (!cfg_holds(*c, scratch)) continue;
        ChainFit fit;
        const cudaError_t e = launch_cfg_of(*c, q, nullptr, 0, &fit);
        if (e != cudaSuccess) return e;
        if (fit.turn > 0) {
            *out = c;
            *turn = fit.turn;
            break;
        }
    }
    return cudaSuccess;
}

// Whether the kernel may reproject through the residual at its checks.
bool residual_form(const ChainArgs &a) { return a.pinv32 && a.check_period != 0x7fffffff && !a.seg; }

}  // namespace

int chain_block_size(int n, int threads_per_chain) {
    const ChainCfg *c = find_cfg(n, threads_per_chain);
    return c ? c->bd : 0;
}

int chain_candidates(int n, int max_np, int scratch, int *bds, int cap) {
    const int np0 = chain_padded_length(n, 0);
    int k = 0;
    for (const ChainCfg &c : kLadder) {
        const int np = c.bd * c.ept;
        if (np < n || np > max_np || np > 2 * np0) continue;
        if (!cfg_holds(c, scratch)) continue;
        bool dup = false;
        for (int j = 0; j < k; ++j) dup |= bds[j] == c.bd;
        if (dup || chain_padded_length(n, c.bd) != np) continue;
        if (k < cap) bds[k++] = c.bd;
    }
    return k;
}

bool chain_takes_threads(int n, int threads_per_chain) {
    const int most = threads_per_chain == 32    ? 256
                     : threads_per_chain == 64  ? 512
                     : threads_per_chain == 320 ? 3840
                     : threads_per_chain == 384 ? 3840
                     : threads_per_chain <= 256 ? 4096
                                                : 16384;
    return threads_per_chain == 0 || n <= most;
}

bool chain_config(const ChainArgs &a, int threads_per_chain, int chains_per_sm, int *bd, int *ept) {
    const int scratch = a.m > a.d ? a.m : a.d;
    const ChainCfg *c = find_cfg(a.n, threads_per_chain, scratch);
    int turn = 0;
    if (c && threads_per_chain == 0) {
        if (!residual_form(a)) c = few_chains_cfg(c, a.n, a.np, a.m, scratch, 0, chains_per_sm);
        else if (find_cfg_residual(a, &c, &turn) != cudaSuccess) return false;
    }
    if (!c) return false;
    *bd = c->bd;
    *ept = c->ept;
    return true;
}

cudaError_t launch_chain_queue(int bd, int ept, const ChainQueue &q, cudaStream_t stream, int grid, int *per_sm) {
    if (bd <= 64) return launch_chain_queue_small(bd, ept, q, stream, grid, per_sm);
    if (bd <= 128) return launch_chain_queue_mid(bd, ept, q, stream, grid, per_sm);
    return launch_chain_queue_large(bd, ept, q, stream, grid, per_sm);
}

cudaError_t launch_chains(const ChainArgs &a_in, int threads_per_chain, cudaStream_t stream, int max_ctas,
                          ChainFit *fit) {
    ChainArgs a = a_in;
    a.z_rows = 0;
    const int scratch = a.m > a.d ? a.m : a.d;
    const ChainCfg *c = find_cfg(a.n, threads_per_chain, scratch);
    if (threads_per_chain == 0) {
        int turn = 0;
        if (residual_form(a)) {
            const cudaError_t e = find_cfg_residual(a, &c, &turn);
            if (e != cudaSuccess) return e;
        }
        if (a.P > 0 && (turn > 0 || !residual_form(a))) {
            int dev = 0, sms = 0;
            cudaError_t e = cudaGetDevice(&dev);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return e;
            const ChainCfg *dflt = c;
            c = few_chains_cfg(dflt, a.n, a.np, a.m, scratch, turn, (a.P + sms - 1) / sms);
            if (c != dflt) a.z_rows = turn;
        }
    }
    if (!c || c->bd * c->ept > a.np) return cudaErrorInvalidValue;
    if (a.P <= 0 && !fit) return cudaSuccess;
    return launch_cfg_of(*c, a, stream, max_ctas, fit);
}

}  // namespace achr
