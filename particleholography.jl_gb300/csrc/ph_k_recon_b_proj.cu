// Reconstruction pass B with the EPI_PROJ epilogue (one translation unit per
// epilogue so the build compiles them in parallel).
#include "ph_two_b.cuh"

namespace ph {

int recon_b_ctas(int n, int rows) {
    switch (n) {
#define PH_CTAS_B(N) case N: return (rows + two::PassB<N, EPI_PROJ, false>::ROWS - 1) / two::PassB<N, EPI_PROJ, false>::ROWS;
        PH_FOR_EACH_N_TWO(PH_CTAS_B)
#undef PH_CTAS_B
    }
    return 0;
}

int recon_b_ctas_per_sm(int n) {
    switch (n) {
#define PH_PER_SM_B(N) case N: return two::PassB<N, EPI_PROJ, false>::CTAS;
        PH_FOR_EACH_N_TWO(PH_PER_SM_B)
#undef PH_PER_SM_B
    }
    return 0;
}

cudaError_t launch_recon_b(int n, const ReconB<EPI_PROJ> &b, cudaStream_t s) {
    const int groups = (b.nbatch + b.group - 1) / b.group;
    switch (n) {
#define PH_TWO_CASE(N) case N: return two::launch_b<N>(b, groups, 1, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return launch_engine_len<false>(n, b, b.rows, groups, s);
}

}  // namespace ph
