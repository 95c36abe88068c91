// pairs_lean_weighted.cu -- the branch-free pair kernel for exact integer weights.
#include "pairs_lean.cuh"

template <int KIND, bool C, int FB>
static cudaError_t launch(const PairArgs &A, int nc, cudaStream_t st, int sm_count, int device) {
    if (KIND == K_ANI || nc == 32) return launch_lean<KIND, true, C, FB, 32>(A, st, sm_count, device);
    // (an anisotropic launch has no columns)
    if (nc == 16) return launch_lean<KIND, true, C, FB, KIND == K_ANI ? 32 : 16>(A, st, sm_count, device);
    return launch_lean<KIND, true, C, FB, KIND == K_ANI ? 32 : 8>(A, st, sm_count, device);
}

template <bool C>
static cudaError_t launch_kind(const PairArgs &A, const PairLaunch &pl, int nc, cudaStream_t st, int sm_count,
                               int device) {
    // an anisotropic copy of limbs has room for 110 bins at most: 16 fraction bits
    static_assert(kLeanWideBins >= 110, "readout of the weighted anisotropic counts");
    if (pl.both) return launch<K_BOTH, C, 16>(A, nc, st, sm_count, device);
    if (pl.ani) return launch<K_ANI, C, 16>(A, nc, st, sm_count, device);
    return pl.rule.bins <= kLeanWideBins ? launch<K_ISO, C, 16>(A, nc, st, sm_count, device)
                                         : launch<K_ISO, C, 15>(A, nc, st, sm_count, device);
}

cudaError_t launch_lean_weighted(const PairArgs &A, const PairLaunch &pl, int nc, cudaStream_t st, int sm_count,
                                 int device) {
    if (pl.ani && pl.rule.bins > kLeanWideBins) return cudaErrorInvalidConfiguration;  // lean_columns is 0 there
    return pl.count ? launch_kind<true>(A, pl, nc, st, sm_count, device)
                    : launch_kind<false>(A, pl, nc, st, sm_count, device);
}
