// Gerchberg-Saxton and propagation passes on the two-stage transform.
#include "ph_two_gs.cuh"

namespace ph {

bool gs_two(int n) { return two::supported(n); }

template <int MODE, bool RESID>
static cudaError_t gs(int n, const two::GsParams &p, cudaStream_t s) {
    switch (n) {
#define PH_TWO_CASE(N) case N: return two::launch_gs<N, MODE, RESID>(p, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_gs_two_col(int n, const two::GsParams &p, cudaStream_t s) { return gs<two::GS_COL, false>(n, p, s); }
cudaError_t launch_gs_two_row(int n, const two::GsParams &p, cudaStream_t s) {
    return p.resid != nullptr ? gs<two::GS_ROW, true>(n, p, s) : gs<two::GS_ROW, false>(n, p, s);
}
cudaError_t launch_gs_two_final(int n, const two::GsParams &p, cudaStream_t s) {
    return gs<two::GS_ROW_FINAL, false>(n, p, s);
}
cudaError_t launch_gs_two_inv(int n, const two::GsParams &p, cudaStream_t s) { return gs<two::GS_ROW_INV, false>(n, p, s); }

}  // namespace ph
