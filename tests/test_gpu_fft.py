"""The imager's own complex-to-real transform (power-of-two grids from 256 to 16384) and the cuFFT path beside it
(other sizes): images against a double-precision transform of the same grid, with crops whose half is odd, the
beam, both output types, and the sizes of every split of the columns axis."""
import numpy as np
import pytest

from fastimaging_b200 import capi
from oracle import stp_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = capi.Context(0)
    yield c
    c.close()


def _reference(ctx, N, size, uv, vis, wts, corr):
    """Image and beam (column-major memory order) from the gridder's own double grid."""
    import torch

    grid, beam, total = ctx.convolve_to_grid(capi.GaussianSinc, 3.0, 3, N, uv, vis, wts, kernel_exact=False,
                                             oversampling=8)
    keep = torch.cat([torch.arange(size // 2), N - size // 2 + torch.arange(size // 2)]).cuda()
    gcf = torch.ones(size, dtype=torch.float64, device="cuda")
    if corr:
        gcf = torch.from_numpy(np.fft.ifftshift(orc.img_dom_kernel(capi.GaussianSinc, 3.0, N, False))).cuda()[keep]
    out = []
    for g in (grid, beam):
        x = torch.from_numpy(np.ascontiguousarray(g.T)).cuda()
        y = torch.fft.irfft2(x, s=(N, N), norm="forward")
        out.append((y[keep][:, keep] / total / gcf[:, None] / gcf[None, :]).cpu().numpy())
        del x, y
    return out[0], out[1], (gcf[:, None] * gcf[None, :]).cpu().numpy()


@pytest.mark.parametrize("N,size,corr", [(256, 256, True), (256, 90, True), (512, 512, False), (512, 300, True),
                                         (1024, 1024, True), (2048, 2046, True), (4096, 4096, True), (8192, 1000, True),
                                         (16384, 500, False), (600, 500, True), (128, 128, True)])
def test_images_match_the_transform_of_the_grid(ctx, N, size, corr):
    rng = np.random.default_rng(N + size)
    n = 400
    uv = rng.uniform(-0.45 * N, 0.45 * N, size=(n, 2))
    uv[::4, 1] *= 0.01
    vis = rng.normal(size=n) + 1j * rng.normal(size=n)
    wts = rng.uniform(0.5, 1.5, n)
    ref, rbeam, g2 = _reference(ctx, N, size, uv, vis, wts, corr)
    cell = 1.0
    uvw = np.column_stack([uv / (N * (cell / 3600.0) * (np.pi / 180.0)), np.zeros(n)])
    kw = dict(kernel_func=capi.GaussianSinc, kernel_support=3, kernel_exact=False, oversampling=8,
              gridding_correction=corr, padded_image_size=N)
    # uv scaled by another route: positions differ by 1e-16 of the grid, kernel offsets rarely by a step
    for precision, dtype, tol in ((capi.FP64, capi.F64, 1e-12), (capi.FP64, capi.F32, 2e-7), (capi.FP32C, capi.F32, 2e-6),
                                  (capi.FP32, capi.F64, 2e-6)):
        img, beam, _ = ctx.image_visibilities(vis, wts, uvw, size, cell, precision=precision, out_dtype=dtype,
                                              generate_beam=True, **kw)
        # Before the correction (g2 = gcf_i gcf_j): a single-precision transform leaves an error of about
        # 2^-24 sqrt(2 log2 N) of the rms, alike at every pixel, which the correction multiplies by up to 890;
        # 2e-6 of the peak is five sigma of it and of the rounded grid.
        for a, b in ((img.T, ref), (beam.T, rbeam)):
            assert (np.abs(a - b) * g2).max() <= tol * (np.abs(b) * g2).max(), (precision, dtype)
