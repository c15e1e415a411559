// Reconstruction pass B with the EPI_SUB epilogue (sub-volumes around boxes).
#include "ph_two_b.cuh"

namespace ph {

cudaError_t launch_recon_b(int n, const ReconB<EPI_SUB> &b, cudaStream_t s) {
    const int groups = (b.nbatch + b.group - 1) / b.group;
    switch (n) {
        case 256: return two::launch_b<256>(b, groups, 1, s);
        case 512: return two::launch_b<512>(b, groups, 1, s);
        case 1024: return two::launch_b<1024>(b, groups, 1, s);
        case 2048: return two::launch_b<2048>(b, groups, 1, s);
        case 4096: return two::launch_b<4096>(b, groups, 1, s);
    }
    return launch_engine_len<false>(n, b, b.rows, groups, s);
}

}  // namespace ph
