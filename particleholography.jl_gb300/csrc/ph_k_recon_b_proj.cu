// Reconstruction pass B with the EPI_PROJ epilogue (one translation unit per
// epilogue so the build compiles them in parallel).
#include "ph_two_b.cuh"

namespace ph {

int recon_b_ctas(int n, int rows) {
    switch (n) {
#define PH_CTAS_B(N) case N: return (rows + two::PassB<N, EPI_PROJ, false>::ROWS - 1) / two::PassB<N, EPI_PROJ, false>::ROWS;
        PH_CTAS_B(256) PH_CTAS_B(512) PH_CTAS_B(1024) PH_CTAS_B(2048) PH_CTAS_B(4096)
#undef PH_CTAS_B
    }
    return 0;
}

int recon_b_ctas_per_sm(int n) {
    switch (n) {
#define PH_PER_SM_B(N) case N: return two::PassB<N, EPI_PROJ, false>::CTAS;
        PH_PER_SM_B(256) PH_PER_SM_B(512) PH_PER_SM_B(1024) PH_PER_SM_B(2048) PH_PER_SM_B(4096)
#undef PH_PER_SM_B
    }
    return 0;
}

cudaError_t launch_recon_b(int n, const ReconB<EPI_PROJ> &b, cudaStream_t s) {
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
