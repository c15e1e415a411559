"""The two-stage row transform of passes A and B (lengths 192 .. 4096) against the
oracle at its edges: a CTA with fewer rows than it holds, a warp of two rows with
one, threads without a transform of their own (3 * 2^a), a box of kx that ends
outside the frame, one slice, slice counts that leave the last group short and
cross the lengths of the product chain."""
import numpy as np
import pytest
import torch

from oracle import ref_semantics as ref
from phtest import rel_l2, to_dev, to_np

pytestmark = pytest.mark.gpu
LAM, DX = 0.6328, 10.0
# An FP32 FFT of 2^22 points is good to ~ eps log2(n) / sqrt(2) ~ 1e-6 in relative L2, on
# either side; pass A's product chain adds eps / 2 per slice.
TOL = 5e-6


@pytest.mark.parametrize("nx,ny,slices", [(256, 1, 1), (256, 3, 5), (256, 24, 33), (512, 1, 2), (512, 6, 65),
                                          (512, 96, 7), (1024, 3, 3), (1024, 6, 34), (2048, 1, 5), (2048, 3, 3),
                                          (2048, 12, 17), (4096, 1, 2), (4096, 3, 9), (192, 1, 2), (192, 6, 33),
                                          (384, 3, 5), (768, 1, 3), (768, 6, 34), (1536, 3, 17), (3072, 1, 2),
                                          (3072, 3, 9),
                                          (4, 192, 3), (24, 192, 18), (4, 256, 1), (12, 256, 35), (12, 384, 9),
                                          (12, 512, 17), (24, 768, 18), (4, 1024, 9), (12, 1024, 33), (8, 1536, 34),
                                          (12, 2048, 17), (4, 3072, 18), (4, 4096, 17)])
def test_rows_and_slices_at_the_edges(ph, cuda, nx, ny, slices):
    rng = np.random.default_rng(nx + ny)
    holo = rng.uniform(0.1, 1.0, (ny, nx)).astype(np.float32)
    d = ref.transfer_sqrt_arr(nx, LAM, DX, n_slow=ny)
    hf, hdz = ref.transfer(-1000.0, nx, LAM, d), ref.transfer(-200.0, nx, LAM, d)
    args = (ph.cu_gabor_wavefront(to_dev(holo, cuda)), ph.CuTransfer(to_dev(hf, cuda)), ph.CuTransfer(to_dev(hdz, cuda)),
            slices)
    wave = ref.gabor_wavefront(holo)
    field = ref.reconst_complex_vol(wave, hf, hdz, slices)
    assert rel_l2(to_np(ph.cu_get_reconst_complex_vol(*args)), field) < TOL
    proj, arg = ph.cu_get_reconst_xyprojection(*args, return_argmin=True)
    p_ref, a_ref = ref.reconst_xyprojection(wave, hf, hdz, slices, with_argmin=True)
    assert rel_l2(to_np(proj), p_ref) < TOL
    assert np.mean(to_np(arg) == a_ref) >= 0.999
    assert torch.equal(ph.cu_get_reconst_xyprojection(*args), proj)     # merged without the slices: the same minima
    vol, vproj = ph.cu_get_reconst_vol_and_xyprojection(*args, torch.float32)
    want = np.clip(np.abs(field.astype(np.complex128)) ** 2, 0.0, 1.0)
    assert rel_l2(to_np(vol), want) < TOL
    assert torch.equal(vproj, vol.amin(0))


@pytest.mark.parametrize("n", [128, 192, 256, 384, 512, 768, 1536])
@pytest.mark.parametrize("iters", [1, 3])
def test_phase_retrieval(ph, cuda, n, iters):
    rng = np.random.default_rng(n)
    h1, h2 = (rng.uniform(0.1, 1.0, (n, n)).astype(np.float32) for _ in range(2))
    d = ref.transfer_sqrt_arr(n, LAM, DX)
    tf, tfi = ref.transfer(700.0, n, LAM, d), ref.transfer(-700.0, n, LAM, d)
    got, res = ph.cu_phase_retrieval_holo(to_dev(h1, cuda), to_dev(h2, cuda), ph.CuTransfer(to_dev(tf, cuda)),
                                          ph.CuTransfer(to_dev(tfi, cuda)), iters, n, return_residual=True)
    want = ref.phase_retrieval_holo(h1, h2, tf, tfi, iters, n)
    # the replacement divides by |u|: rounding of the transforms grows where the field is small
    assert rel_l2(to_np(got.data), want) < 4 * iters * TOL
    assert 0.0 < float(res) < 1.0


@pytest.mark.parametrize("n", [128, 192, 384, 512, 768, 1024, 1536, 2048])
def test_propagation(ph, cuda, n):
    rng = np.random.default_rng(n)
    u = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))).astype(np.complex64)
    d = ref.transfer_sqrt_arr(n, LAM, DX)
    out = ph.CuWavefront(torch.empty((n, n), dtype=torch.complex64, device=cuda))
    ph.cu_asm_prop_(out, ph.CuWavefront(to_dev(u, cuda)), ph.CuTransferSqrtPart(to_dev(d, cuda)), 4321.0, n, LAM)
    assert rel_l2(to_np(out.data), ref.asm_prop(u, d, 4321.0, n, LAM)) < TOL
