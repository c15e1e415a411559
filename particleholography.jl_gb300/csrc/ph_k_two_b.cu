// Reconstruction pass B on the two-stage transform.
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

template <int EPI>
static cudaError_t pass_b(int n, const ReconB<EPI> &b, cudaStream_t s) {
    const int groups = (b.nbatch + b.group - 1) / b.group;
    switch (n) {
#define PH_TWO_CASE(N) case N: return two::launch_b<N>(b, groups, 1, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return cudaErrorInvalidValue;
}
cudaError_t launch_recon_b_two(int n, const ReconB<EPI_PROJ> &b, cudaStream_t s) { return pass_b(n, b, s); }
cudaError_t launch_recon_b_two(int n, const ReconB<EPI_VOL> &b, cudaStream_t s) { return pass_b(n, b, s); }
cudaError_t launch_recon_b_two(int n, const ReconB<EPI_CVOL> &b, cudaStream_t s) { return pass_b(n, b, s); }

cudaError_t launch_recon_b_group_two(int n, const ReconB<EPI_PROJ, true> &b, cudaStream_t s) {
    int gy = 1;
    for (int i = 0; i < b.nitems; ++i) gy = std::max(gy, (b.item_nb(i) + b.item_group(i) - 1) / b.item_group(i));
    switch (n) {
#define PH_TWO_CASE(N) case N: return two::launch_b<N>(b, gy, b.nitems, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return cudaErrorInvalidValue;
}

}  // namespace ph
