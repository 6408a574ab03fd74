// Which runs defer their reprojections to the batched passes (host only).
#pragma once

namespace achr {

// Reprojecting P chains in the chain kernel takes P 4 n d FP64 operations at every
// check, deferring it about 0.1 ms of launches and passes, so the line lies at a
// work of P n d.  Measured per 50 steps (five checks), in the kernel / deferred:
//   n = 95, d = 20:    P = 1000 0.23 / 0.64 ms, 5000 0.75 / 1.18
//   n = 200, d = 43:   P = 1000 0.49 / 0.82,    5000 1.85 / 1.58   (P n d = 8.6e6, 4.3e7)
//   n = 400, d = 84:   P = 1000 1.08 / 0.87,    5000 5.19 / 2.23   (3.4e7, 1.7e8)
//   n = 1060, d = 159: P = 1000 3.92 / 1.61,    5000 19.9 / 5.62
// Models of n d >= 2.5e5 are always deferred.
// Neither side of the line is the less exact one by being deferred: against a projection refined in
// 128-bit floating point a deferred point's rms error is 2e-14 to 4e-14 for 95 to 1060 reactions,
// N (N^T x) in the kernel 6e-14 to 6e-13.
constexpr double kDeferWork = 2.0e7, kDeferModel = 2.5e5;

enum class DeferUse {
    kKernel,   // reprojections in the chain kernel
    kMay,      // deferred if nothing stands in the way
    kAlways,   // deferred, or the call fails
};

// selected: the model, its warmup points and the options allow it (defer_selected).
inline DeferUse defer_use(bool selected, bool asked, double chains, double nd) {
    if (!selected) return DeferUse::kKernel;
    if (asked || nd >= kDeferModel) return DeferUse::kAlways;
    return chains * nd >= kDeferWork ? DeferUse::kMay : DeferUse::kKernel;
}

enum class DeferBuffers { kReady, kNoMemory, kFailed };

struct DeferChoice {
    bool deferred, failed;
};

// Whether a run of `chains` chains is deferred.  A captured run that need not be stays in the kernel,
// whether or not buffers exist: its graph then holds no buffer that the context may replace, and what a
// capture gives does not depend on the calls before it.  Where there is no memory for the buffers
// (prepare) a run that need not be deferred stays in the kernel too, and so does every later run of the
// context of that size or more (short_from, 0 at first): a run continued in segments keeps its form, and
// memory is not asked for at every call.  Any other failure is the call's.
template <class Prepare>
DeferChoice defer_choose(DeferUse use, bool capturing, int chains, int &short_from, Prepare prepare) {
    if (use == DeferUse::kAlways) return {true, false};
    if (use == DeferUse::kKernel || capturing || (short_from > 0 && chains >= short_from)) return {false, false};
    switch (prepare()) {
        case DeferBuffers::kReady: return {true, false};
        case DeferBuffers::kNoMemory: short_from = chains; return {false, false};
        default: return {false, true};
    }
}

}  // namespace achr
