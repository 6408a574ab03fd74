// Configuration ladder of the chain kernel and the rules that choose from it (host code, no CUDA types).
//
// A configuration is (threads per chain, elements per thread); its padded
// length, their product, must hold the model's n reactions.  For each padded
// length there is a default configuration (used when threads_per_chain = 0)
// and alternatives: for launches of few chains, and for the autotuner.
#pragma once

#include <initializer_list>

namespace achr {

struct ChainCfg {
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
constexpr ChainCfg kLadder[] = {
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

// Doubles of a configuration's accumulator in shared memory, the reprojection's scratch, and whether
// max(m, d) = `scratch` of them suffice (elsewhere d <= n does, and the residual form asks for m <= n).
inline int cfg_scratch(const ChainCfg &c) { return c.bd == 256 && c.ept == 30 ? kScratch256x30 : c.bd * c.ept; }
inline bool cfg_holds(const ChainCfg &c, int scratch) { return !(c.bd == 256 && c.ept == 30 && scratch > kScratch256x30); }

inline const ChainCfg *find_cfg(int n, int threads_per_chain, int scratch = 0) {
    for (const ChainCfg &c : kLadder) {
        if (c.bd * c.ept < n) continue;
        if (!cfg_holds(c, scratch)) continue;
        if (threads_per_chain == 0 ? c.dflt : c.bd == threads_per_chain) return &c;
    }
    return nullptr;
}

// Rows of z = (S S^T)^+ r that fit beside r (m float pairs) in `scratch` doubles; 0
// where that would take more than eight turns.
inline int residual_z_rows(int m, int scratch) {
    const int rows = 2 * (scratch - m);
    return rows <= 0 || (long long)rows * 8 < m ? 0 : rows < m ? rows : m;
}

// The configuration for `per_sm` chains per SM where `best` is the one for many.
// A launch of few chains per SM is bound by a chain's own latency, which more
// warps shorten, up to about 16 warps on an SM; after that the FP64 pipe is the
// bound, where more warps only repeat the reductions.  The results do not depend
// on it.  Measured, SM clocks per chain-step, default and the one taken, at 1, 2, 4 and 8 chains per SM: n = 95
// (32 -> 64 threads) 5358 4607, 2707 2321, 1362 1246, 736 739; n = 250 (32 ->
// 128, from 8 per SM 64) 7839 5367, 3930 2847, 1980 1650, 1107 1060; n = 500 (64
// -> 256, 256, 128) 8425 5712, 4255 3400, 2378 2094; n = 1060 (64 -> 256, 256,
// 128) 16027 8972, 8004 5664, 4649 3895.
// max_np: the length the per-reaction arrays were padded to.  turn > 0: the launch reprojects through the
// residual in turns of that many rows of z; a configuration that takes the same turns (all m at once
// always has room) gives the same points.  Two warps form z = (S S^T)^+ r slowly, so such launches gain
// most: reprojecting at every check, 20 steps of one chain, the default and the one taken, microseconds:
// n = 250 327, 135; 1060 1239, 263; 2500 2050, 662; 7440 11226, 5875; without reprojections, 100
// chains of n = 7440: 411, 285.
inline const ChainCfg *few_chains_cfg(const ChainCfg *best, int n, int max_np, int m, int scratch, int turn, int per_sm) {
    if (!best) return nullptr;
    const int np0 = best->bd * best->ept;
    const int least = best->bd;
    for (int bd : {64, 128, 256, 512}) {
        const ChainCfg *c = find_cfg(n, bd, scratch);
        if (!c || bd <= least || c->bd * c->ept > max_np || c->bd * c->ept > 2 * np0) continue;
        if (turn > 0 && turn < m && 2 * (cfg_scratch(*c) - m) < turn) continue;
        if ((long long)per_sm * (bd / 32) <= kFewWarps) best = c;
    }
    return best;
}

inline int chain_padded_length(int n, int threads_per_chain) {
    const ChainCfg *c = find_cfg(n, threads_per_chain);
    return c ? c->bd * c->ept : 0;
}

// Length to pad per-reaction arrays to, at most `most`: twice the default padded length (so every
// configuration for few chains and every autotuning candidate fits).
inline int chain_alloc_length(int n, int most = 16384) {
    const int np = chain_padded_length(n, 0);
    if (np == 0 || np > most) return 0;
    return np * 2 < most ? np * 2 : most;
}

}  // namespace achr
