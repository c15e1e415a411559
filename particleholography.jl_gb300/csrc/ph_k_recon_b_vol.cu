// Reconstruction pass B with the EPI_VOL epilogue (one translation unit per
// epilogue so the build compiles them in parallel).
#include "ph_two_b.cuh"

namespace ph {

cudaError_t launch_recon_b(int n, const ReconB<EPI_VOL> &b, cudaStream_t s) {
    const int groups = (b.nbatch + b.group - 1) / b.group;
    switch (n) {
#define PH_TWO_CASE(N) case N: return two::launch_b<N>(b, groups, 1, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return launch_engine_len<false>(n, b, b.rows, groups, s);
}

}  // namespace ph
