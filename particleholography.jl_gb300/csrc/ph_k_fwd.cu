// Forward row passes (transposed store).
#include "ph_two_f.cuh"

namespace ph {

template <int MODE>
static cudaError_t fwd(int n, const FwdRowsT<MODE> &b, cudaStream_t s) {
    switch (n) {
#define PH_TWO_CASE(N) \
    case N: return two::launch_f<N, false>(two::k_two_fwd<N, MODE>, two::PassF<N>::SMEM, b, b.nrows, b.nitems, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return launch_engine_len<true>(n, b, b.nrows, 1, s, b.nitems);
}

cudaError_t launch_fwd_rows(int n, const FwdRowsT<FWD_COMPLEX> &b, cudaStream_t s) { return fwd(n, b, s); }
cudaError_t launch_fwd_rows(int n, const FwdRowsT<FWD_SQRT_REAL> &b, cudaStream_t s) { return fwd(n, b, s); }
cudaError_t launch_fwd_rows(int n, const FwdRowsT<FWD_PADDED> &b, cudaStream_t s) { return fwd(n, b, s); }

}  // namespace ph
