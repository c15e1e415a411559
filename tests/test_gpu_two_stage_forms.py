"""The two-stage passes in the forms that single Float32 calls do not take: grouped
launches, Float64 volumes, several slice batches, and the largest propagations."""
import numpy as np
import pytest
import torch

from oracle import ref_semantics as ref
from phtest import rel_l2, to_dev, to_np

pytestmark = pytest.mark.gpu
LAM, DX = 0.6328, 10.0
TOL = 5e-6   # relative L2 of a Float32 transform chain (eps log2(n), a few of them)


def _frame(ph, cuda, nx, ny, seed):
    rng = np.random.default_rng(seed)
    holo = rng.uniform(0.1, 1.0, (ny, nx)).astype(np.float32)
    d = ref.transfer_sqrt_arr(nx, LAM, DX, n_slow=ny)
    return holo, ref.transfer(-1000.0, nx, LAM, d), ref.transfer(-200.0 - seed, nx, LAM, d)


@pytest.mark.parametrize("nx,ny", [(192, 128), (12, 192), (384, 64), (24, 768), (1536, 6), (8, 3072), (3072, 8), (12, 4096),
                                   (4096, 6)])
def test_grouped_items_match_single_calls(ph, cuda, nx, ny):
    """Items of one shape and different slice counts, launched together: a single call's words."""
    counts = [1, 9, 34, 17, 5]
    items, want = [], []
    for i, slices in enumerate(counts):
        holo, hf, hdz = _frame(ph, cuda, nx, ny, i)
        a = (to_dev(holo, cuda), ph.CuTransfer(to_dev(hf, cuda)), ph.CuTransfer(to_dev(hdz, cuda)))
        items.append({"hologram": a[0], "transfer_front": a[1], "transfer_dz": a[2], "slices": slices})
        want.append((ph.cu_get_reconst_xyprojection(ph.cu_gabor_wavefront(a[0]), a[1], a[2], slices, return_argmin=True),
                     ref.reconst_xyprojection(ref.gabor_wavefront(holo), hf, hdz, slices)))
    batch = ph.ReconBatch(items, lanes=1)
    projs, args = batch.run()
    for p, a, ((p1, a1), oracle) in zip(projs, args, want):
        assert torch.equal(p, p1) and torch.equal(a, a1)
        assert rel_l2(to_np(p), oracle) < TOL
    batch.close()


@pytest.mark.parametrize("n", [128, 192, 1024])
def test_float64_volume_widens_the_float32_one(ph, cuda, n):
    holo, hf, hdz = _frame(ph, cuda, n, 128, 3)
    args = (ph.cu_gabor_wavefront(to_dev(holo, cuda)), ph.CuTransfer(to_dev(hf, cuda)), ph.CuTransfer(to_dev(hdz, cuda)), 7)
    wide, proj = ph.cu_get_reconst_vol_and_xyprojection(*args, torch.float64)
    narrow = ph.cu_get_reconst_vol(*args, torch.float32)
    assert wide.dtype == torch.float64 and torch.equal(wide, narrow.double())
    assert torch.equal(proj, narrow.amin(0))


@pytest.mark.parametrize("nx,ny", [(192, 384), (768, 24), (12, 1536), (3072, 4), (128, 2048)])
@pytest.mark.parametrize("batch", [1, 5, 16])
def test_slice_batches_give_the_same_words(ph, cuda, nx, ny, batch):
    from ph_gb300 import _lib
    holo, hf, hdz = _frame(ph, cuda, nx, ny, 1)
    args = (ph.cu_gabor_wavefront(to_dev(holo, cuda)), ph.CuTransfer(to_dev(hf, cuda)), ph.CuTransfer(to_dev(hdz, cuda)), 37)
    want = ph.cu_get_reconst_xyprojection(*args, return_argmin=True)
    ctx = _lib.default_context(0)
    try:
        ctx.set_option(_lib.PH_OPT_SLICE_BATCH, batch)
        got = ph.cu_get_reconst_xyprojection(*args, return_argmin=True)
    finally:
        ctx.set_option(_lib.PH_OPT_SLICE_BATCH, 0)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("n", [3072, 4096])
def test_largest_propagations(ph, cuda, n):
    """Against torch in 64 bits (the oracle's field takes minutes at these lengths)."""
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    u = torch.randn((n, n), dtype=torch.complex64, generator=g, device=cuda)
    d = ph.cu_transfer_sqrt_arr(n, LAM, DX)
    out = ph.CuWavefront(torch.empty_like(u))
    ph.cu_asm_prop_(out, ph.CuWavefront(u), d, 4321.0, n, LAM)
    h = torch.fft.ifftshift(ph.cu_transfer(4321.0, n, LAM, d).data.to(torch.complex128))
    want = torch.fft.ifft2(torch.fft.fft2(u.to(torch.complex128)) * h)
    assert float((out.data - want).abs().square().sum().sqrt() / want.abs().square().sum().sqrt()) < TOL


def test_retrieval_at_3072(ph, cuda):
    n, iters = 3072, 1
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    h1, h2 = (0.1 + torch.rand((n, n), generator=g, device=cuda) for _ in range(2))
    d = ph.cu_transfer_sqrt_arr(n, LAM, DX)
    tf, tfi = ph.cu_transfer(700.0, n, LAM, d), ph.cu_transfer(-700.0, n, LAM, d)
    got = ph.cu_phase_retrieval_holo(h1, h2, tf, tfi, iters, n).data
    there, back = (torch.fft.ifftshift(t.data.to(torch.complex128)) for t in (tf, tfi))
    u = torch.sqrt(h1).to(torch.complex128)
    u = torch.fft.ifft2(torch.fft.fft2(u) * there)
    u = torch.polar(torch.sqrt(h2).double(), torch.angle(u))
    u = torch.fft.ifft2(torch.fft.fft2(u) * back)
    want = torch.polar(torch.sqrt(h1).double(), torch.angle(u))
    assert float((got - want).abs().square().sum().sqrt() / want.abs().square().sum().sqrt()) < 4 * iters * TOL
