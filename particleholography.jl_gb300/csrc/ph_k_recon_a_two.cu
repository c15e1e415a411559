// Reconstruction pass A on the two-stage transform (lengths 128 .. 4096).
#include "ph_two_a.cuh"

namespace ph {

bool recon_a_two(int n) { return two::supported(n); }

int recon_a_two_box(int n) {
    switch (n) {
#define PH_BOX_A(N) case N: return two::PassA<N>::RB;
        PH_FOR_EACH_N_TWO(PH_BOX_A)
#undef PH_BOX_A
    }
    return 0;
}

int recon_a_two_box_y(int n) { return two::box_y(n); }

int recon_a_two_ctas_per_sm(int n) {
    switch (n) {
#define PH_PER_SM_A(N) case N: return two::PassA<N>::CTAS;
        PH_FOR_EACH_N_TWO(PH_PER_SM_A)
#undef PH_PER_SM_A
    }
    return 0;
}

cudaError_t launch_recon_a_two(int n, const ReconA &b, const CUtensorMap &tm, int nbatch, cudaStream_t s) {
    const int gy = (nbatch + b.group - 1) / b.group;
    switch (n) {
#define PH_TWO_CASE(N) case N: return two::launch_a<N>(b, tm, gy, 1, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_recon_a_group_two(int n, const ReconAGrouped &b, const CUtensorMap &tm, cudaStream_t s) {
    int gy = 1;
    for (int i = 0; i < b.nitems; ++i) gy = std::max(gy, (b.item_nb(i) + b.item_group(i) - 1) / b.item_group(i));
    switch (n) {
#define PH_TWO_CASE(N) case N: return two::launch_a<N>(b, tm, gy, b.nitems, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return cudaErrorInvalidValue;
}

}  // namespace ph
