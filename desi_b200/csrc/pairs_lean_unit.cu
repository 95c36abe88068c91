// pairs_lean_unit.cu -- the branch-free pair kernel for unit weights.
#include "pairs_lean.cuh"

template <int FB>
static cudaError_t launch(const PairArgs &A, const PairLaunch &pl, cudaStream_t st, int sm_count, int device) {
    if (pl.both) return launch_lean<K_BOTH, false, false, FB, 32>(A, st, sm_count, device);
    if (pl.ani) return launch_lean<K_ANI, false, false, FB, 32>(A, st, sm_count, device);
    return launch_lean<K_ISO, false, false, FB, 32>(A, st, sm_count, device);
}

cudaError_t launch_lean_unit(const PairArgs &A, const PairLaunch &pl, cudaStream_t st, int sm_count, int device) {
    return pl.rule.bins <= kLeanWideBins ? launch<16>(A, pl, st, sm_count, device)
                                         : launch<15>(A, pl, st, sm_count, device);
}
