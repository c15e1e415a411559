// Forward rows and spectrum on the two-stage transform.
#include "ph_two_f.cuh"

namespace ph {

bool recon_two(int n) { return two::supported(n); }

template <int MODE>
static cudaError_t fwd(int n, const FwdRowsT<MODE> &b, cudaStream_t s) {
    switch (n) {
#define PH_TWO_CASE(N) case N: return two::launch_f<N, false>(two::k_two_fwd<N, MODE>, two::PassF<N>::SMEM, b, b.nrows, b.nitems, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return cudaErrorInvalidValue;
}
cudaError_t launch_fwd_rows_two(int n, const FwdRowsT<FWD_COMPLEX> &b, cudaStream_t s) { return fwd(n, b, s); }
cudaError_t launch_fwd_rows_two(int n, const FwdRowsT<FWD_SQRT_REAL> &b, cudaStream_t s) { return fwd(n, b, s); }

// state[kx][ky] = (a1[kx][ky] hf scale (lpf), turns(hdz), log2 |hdz|), the transfers
// centred [ny][nx]: 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256) k_state(const SpectrumCols p) {
    __shared__ float4 tile[32][33];
    grid_dependents_launch();
    const int z = blockIdx.z, tx = threadIdx.x % 32, ty = threadIdx.x / 32;
    const float2 *hf = p.nitems > 1 ? p.hf_items[z] : p.hf;
    const float2 *hdz = p.nitems > 1 ? p.hdz_items[z] : p.hdz;
    const int kx0 = blockIdx.x * 32, ky0 = blockIdx.y * 32;
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
        const int ky = ky0 + ty + i, kx = kx0 + tx;
        if (ky < p.ny && kx < p.nx) {
            const size_t at = (size_t)shift_idx(ky, p.ny) * p.nx + shift_idx(kx, p.nx);
            const float2 d = hdz[at], h = cscale(hf[at], p.lpf != nullptr ? p.scale * p.lpf[at] : p.scale);
            tile[ty + i][tx] = make_float4(h.x, h.y, __uint_as_float(phase_turns_u32(d, p.ptab)), log2_modulus(d));
        }
    }
    __syncthreads();
    grid_dependency_wait();   // the transfers above are the caller's; a1 and the state are not
    const float2 *a1 = p.a1 + (size_t)z * p.a1_stride;
    float4 *state = p.state + (size_t)z * p.state_stride;
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
        const int kx = kx0 + ty + i, ky = ky0 + tx;
        if (kx < p.nx && ky < p.ny) {
            const float4 t = tile[tx][ty + i];
            const float2 x0 = cmul(a1[(size_t)kx * p.ny + ky], make_float2(t.x, t.y));
            state[(size_t)kx * p.ny + ky] = make_float4(x0.x, x0.y, t.z, t.w);
        }
    }
}

static cudaError_t cols(int n, const SpectrumCols &b, cudaStream_t s) {
    switch (n) {
#define PH_TWO_CASE(N) case N: return two::launch_f<N, true>(two::k_two_cols<N>, two::PassF<N>::RB * two::PassF<N>::XB, b, b.nx, b.nitems, s);
        PH_FOR_EACH_N_TWO(PH_TWO_CASE)
#undef PH_TWO_CASE
    }
    return cudaErrorInvalidValue;
}
cudaError_t launch_spectrum_two(int n, const SpectrumCols &b, cudaStream_t s) {
    const cudaError_t e = cols(n, b, s);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_state, dim3((b.nx + 31) / 32, (b.ny + 31) / 32, b.nitems), 256, 0, s, b);
}

}  // namespace ph
