// Reconstruction pass A on the two-stage transform (lengths 256 .. 4096).
#include "ph_two_a.cuh"

namespace ph {

bool recon_a_two(int n, int y0, int ny_out) {
    return two::supported(n) && y0 % kTwoBoxY == 0 && ny_out % kTwoBoxY == 0;
}

int recon_a_two_box(int n) {
    switch (n) {
#define PH_BOX_A(N) case N: return two::PassA<N>::RB;
        PH_BOX_A(256) PH_BOX_A(512) PH_BOX_A(1024) PH_BOX_A(2048) PH_BOX_A(4096)
#undef PH_BOX_A
    }
    return 0;
}

int recon_a_two_ctas_per_sm(int n) {
    switch (n) {
#define PH_PER_SM_A(N) case N: return two::PassA<N>::CTAS;
        PH_PER_SM_A(256) PH_PER_SM_A(512) PH_PER_SM_A(1024) PH_PER_SM_A(2048) PH_PER_SM_A(4096)
#undef PH_PER_SM_A
    }
    return 0;
}

cudaError_t launch_recon_a_two(int n, const ReconA &b, const CUtensorMap &tm, int nbatch, cudaStream_t s) {
    const int gy = (nbatch + b.group - 1) / b.group;
    switch (n) {
        case 256: return two::launch_a<256>(b, tm, gy, 1, s);
        case 512: return two::launch_a<512>(b, tm, gy, 1, s);
        case 1024: return two::launch_a<1024>(b, tm, gy, 1, s);
        case 2048: return two::launch_a<2048>(b, tm, gy, 1, s);
        case 4096: return two::launch_a<4096>(b, tm, gy, 1, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_recon_a_group_two(int n, const ReconAGrouped &b, const CUtensorMap &tm, cudaStream_t s) {
    int gy = 1;
    for (int i = 0; i < b.nitems; ++i) gy = std::max(gy, (b.item_nb(i) + b.item_group(i) - 1) / b.item_group(i));
    switch (n) {
        case 256: return two::launch_a<256>(b, tm, gy, b.nitems, s);
        case 512: return two::launch_a<512>(b, tm, gy, b.nitems, s);
        case 1024: return two::launch_a<1024>(b, tm, gy, b.nitems, s);
        case 2048: return two::launch_a<2048>(b, tm, gy, b.nitems, s);
        case 4096: return two::launch_a<4096>(b, tm, gy, b.nitems, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace ph
