// Configuration ladder of the chain kernel and its dispatcher.
//
// A configuration is (threads per chain BD, elements per thread EPT); its
// padded length BD * EPT must hold the model's n reactions.  For each padded
// length there is a default configuration (used when threads_per_chain = 0)
// and alternatives: for launches of few chains, and for the autotuner.
#include "achr_internal.h"

namespace achr {

cudaError_t launch_chain_cfg_small(int bd, int ept, const ChainArgs &a, cudaStream_t s, int max_ctas, int *per_sm);
cudaError_t launch_chain_cfg_large(int bd, int ept, const ChainArgs &a, cudaStream_t s, int max_ctas, int *per_sm);
cudaError_t launch_chain_cfg_mid(int bd, int ept, const ChainArgs &a, cudaStream_t s, int max_ctas, int *per_sm);
cudaError_t launch_chain_queue_small(int bd, int ept, const ChainQueue &q, cudaStream_t s, int grid, int *per_sm);
cudaError_t launch_chain_queue_mid(int bd, int ept, const ChainQueue &q, cudaStream_t s, int grid, int *per_sm);
cudaError_t launch_chain_queue_large(int bd, int ept, const ChainQueue &q, cudaStream_t s, int grid, int *per_sm);

namespace {

struct Cfg {
    int bd, ept;
    bool dflt;
};

// Ordered by padded length; the default for each length comes first.  The
// kernel is bound by the FP64 pipe once enough chains share an SM to fill each
// other's latency, so a default has few warps per chain (each repeats the
// reductions) where shared memory still holds four chains or more, and more
// warps where it holds two.  Measured, SM clocks per chain-step at full
// residency (the previous kernel's in brackets): n = 95, 32 x 4: 400 [689];
// n = 1060, 64 x 20: 3550 [7760], 256 x 8: 4920; n = 2500, 128 x 20: 6790,
// 320 x 12: 8680; n = 3000, 128 x 24: 8690, 320 x 12: 9080; n = 3742, 320 x 12:
// 10190 [13960 with 384 x 10], 384 x 10: 10350, 256 x 16: 10940; n = 7440, 256 x
// 30: 23090, 384 x 20: 26500 [31020 with 512 x 15], 512 x 16: 26600.  The others serve an explicit
// threads_per_chain and the autotuner.
const Cfg kLadder[] = {
    {32, 4, true},    {64, 4, false},   {32, 8, true},    {64, 6, true},    {128, 4, false},  {64, 8, true},
    {64, 12, true},   {64, 16, true},   {128, 8, false},  {256, 4, false},  {64, 20, true},   {128, 12, true},
    {128, 16, true},  {256, 8, false},  {512, 4, false},  {128, 20, true},  {128, 24, true},  {320, 12, true},
    {384, 10, false}, {256, 16, true},  {512, 8, false},  {128, 32, false}, {256, 18, true},  {256, 20, true},
    {256, 24, true},  {512, 12, false}, {256, 26, true},  {256, 30, true},  {384, 20, true},  {512, 16, true},  {512, 32, true},
};

// 256 x 30 keeps 6 x 256 of the accumulator's doubles in registers, and the rest
// is too little scratch for a reprojection onto more than 6144 coordinates.
constexpr int kScratch256x30 = 256 * (30 - 6);

constexpr int kFewWarps = 16;  // warps per SM up to which a launch counts as one of few chains

const Cfg *find_cfg(int n, int threads_per_chain, int scratch = 0) {
    for (const Cfg &c : kLadder) {
        if (c.bd * c.ept < n) continue;
        if (c.bd == 256 && c.ept == 30 && scratch > kScratch256x30) continue;
        if (threads_per_chain == 0 ? c.dflt : c.bd == threads_per_chain) return &c;
    }
    return nullptr;
}

// The default for P chains on `sms` SMs.  A launch of few chains per SM is bound
// by a chain's own latency, which more warps shorten, up to about 16 warps on an
// SM; after that the FP64 pipe is the bound, where more warps only repeat the
// reductions.  The results do not depend on it.  Measured, SM clocks per
// chain-step, default and the one taken, at 1, 2, 4 and 8 chains per SM: n = 95
// (32 -> 64 threads) 5358 4607, 2707 2321, 1362 1246, 736 739; n = 250 (32 ->
// 128, from 8 per SM 64) 7839 5367, 3930 2847, 1980 1650, 1107 1060; n = 500 (64
// -> 256, 256, 128) 8425 5712, 4255 3400, 2378 2094; n = 1060 (64 -> 256, 256,
// 128) 16027 8972, 8004 5664, 4649 3895.
const Cfg *find_cfg_for(const ChainArgs &a, int sms) {
    const int scratch = a.m > a.d ? a.m : a.d;
    const Cfg *best = find_cfg(a.n, 0, scratch);
    if (!best) return nullptr;
    const int per_sm = (a.P + sms - 1) / sms, np0 = best->bd * best->ept;
    for (int bd : {64, 128, 256, 512}) {
        const Cfg *c = find_cfg(a.n, bd, scratch);
        const int np = c ? c->bd * c->ept : 0;
        if (c && bd > best->bd && np <= a.np && np <= 2 * np0 && (long long)per_sm * (bd / 32) <= kFewWarps) best = c;
    }
    return best;
}

cudaError_t launch_cfg_of(const Cfg &c, const ChainArgs &a, cudaStream_t stream, int max_ctas, int *per_sm) {
    if (c.bd <= 64) return launch_chain_cfg_small(c.bd, c.ept, a, stream, max_ctas, per_sm);
    if (c.bd <= 128) return launch_chain_cfg_mid(c.bd, c.ept, a, stream, max_ctas, per_sm);
    return launch_chain_cfg_large(c.bd, c.ept, a, stream, max_ctas, per_sm);
}

// The default for a model that reprojects through the residual in the kernel:
// the first configuration, from its length's default on, in which z has room.
// Reprojecting as N (N^T x) instead costs 4 n d FP64 operations, 11 ms of an SM
// at 5063 x 7440 against a step's 23 K clocks.  The choice, and with it the form
// and its turns, does not depend on the number of chains.
cudaError_t find_cfg_residual(const ChainArgs &a, const Cfg **out) {
    const int scratch = a.m > a.d ? a.m : a.d;
    const Cfg *dflt = *out = find_cfg(a.n, 0, scratch);
    if (!dflt) return cudaSuccess;
    ChainArgs q = a;
    q.P = 0;  // (asks for the residency only)
    for (const Cfg *c = dflt; c != kLadder + sizeof(kLadder) / sizeof(kLadder[0]); ++c) {
        if (c->bd * c->ept > a.np) continue;
        if (c->bd == 256 && c->ept == 30 && scratch > kScratch256x30) continue;
        int per_sm = 0;
        const cudaError_t e = launch_cfg_of(*c, q, nullptr, 0, &per_sm);
        if (e != cudaSuccess) return e;
        if (per_sm > 0) {
            *out = c;
            break;
        }
    }
    return cudaSuccess;
}

// Whether the kernel may reproject through the residual at its checks.
bool residual_form(const ChainArgs &a) { return a.pinv32 && a.check_period != 0x7fffffff && !a.seg; }

}  // namespace

int chain_padded_length(int n, int threads_per_chain) {
    const Cfg *c = find_cfg(n, threads_per_chain);
    return c ? c->bd * c->ept : 0;
}

int chain_block_size(int n, int threads_per_chain) {
    const Cfg *c = find_cfg(n, threads_per_chain);
    return c ? c->bd : 0;
}

int chain_alloc_length(int n) {
    const int np = chain_padded_length(n, 0);
    if (np == 0) return 0;
    return np * 2 > 16384 ? np : np * 2;
}

int chain_candidates(int n, int max_np, int scratch, int *bds, int cap) {
    const int np0 = chain_padded_length(n, 0);
    int k = 0;
    for (const Cfg &c : kLadder) {
        const int np = c.bd * c.ept;
        if (np < n || np > max_np || np > 2 * np0) continue;
        if (c.bd == 256 && c.ept == 30 && scratch > kScratch256x30) continue;
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

int chain_scratch_doubles(int bd, int ept) {
    return bd == 256 && ept == 30 ? kScratch256x30 : bd * ept;
}

bool chain_config(const ChainArgs &a, int threads_per_chain, int *bd, int *ept) {
    const Cfg *c = find_cfg(a.n, threads_per_chain, a.m > a.d ? a.m : a.d);
    if (c && threads_per_chain == 0 && residual_form(a) && find_cfg_residual(a, &c) != cudaSuccess) return false;
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

cudaError_t launch_chains(const ChainArgs &a, int threads_per_chain, cudaStream_t stream, int max_ctas,
                          int *per_sm) {
    const Cfg *c = find_cfg(a.n, threads_per_chain, a.m > a.d ? a.m : a.d);
    if (threads_per_chain == 0 && residual_form(a)) {
        const cudaError_t e = find_cfg_residual(a, &c);
        if (e != cudaSuccess) return e;
    } else if (threads_per_chain == 0 && a.P > 0) {
        int dev = 0, sms = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        c = find_cfg_for(a, sms);
    }
    if (!c || c->bd * c->ept > a.np) return cudaErrorInvalidValue;
    if (a.P <= 0 && !per_sm) return cudaSuccess;
    return launch_cfg_of(*c, a, stream, max_ctas, per_sm);
}

}  // namespace achr
