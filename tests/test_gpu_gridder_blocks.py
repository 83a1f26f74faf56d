"""The block gridder at the sizes where it can go wrong: grids that are not a multiple of the 8 x 8 blocks or
smaller than a footprint, footprints across the grid's edges, mirrored copies, supports on both sides of a
block's width, blocks with more entries than one warp takes, and entries that are not finite."""
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


def _points(seed, n, N, spread):
    """uv in pixels: over the whole grid, at its edges and near v = 0."""
    rng = np.random.default_rng(seed)
    uv = rng.uniform(-0.5 * N, 0.5 * N, size=(n, 2)) * spread
    uv[::5, 1] *= 0.02
    uv[1::7, 0] *= 0.02
    vis = rng.normal(size=n) + 1j * rng.normal(size=n)
    return uv, vis, rng.uniform(0.5, 1.5, n)


def _compare(ctx, kf, S, N, uv, vis, wts, exact, os, half, **kw):
    g = ctx.convolve_to_grid(kf, float(S), S, N, uv, vis, wts, kernel_exact=exact, oversampling=os, halfplane=half,
                             shift_uv=True, generate_beam=True, **kw)
    r = orc.convolve_to_grid(kf, S, N, uv, vis, wts, exact, os, True, half, True)
    # double-precision sums of at most n terms in another order
    tol = 1e-12 * max(1.0, float(np.abs(r.vis_grid).max()))
    assert np.abs(g[0] - r.vis_grid).max() <= tol
    assert np.abs(g[1] - r.sampling_grid).max() <= 1e-12 * max(1.0, float(np.abs(r.sampling_grid).max()))
    assert abs(g[2] - r.sample_grid_total) <= 1e-12 * abs(r.sample_grid_total)


@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("N,S", [(10, 1), (18, 4), (30, 3), (64, 4), (66, 5), (102, 8), (130, 9), (256, 3)])
def test_blocks_match_oracle(ctx, N, S, exact, half):
    uv, vis, wts = _points(N + S, 700, N, 1.05)
    _compare(ctx, capi.PSWF if S > 1 else capi.Triangle, S, N, uv, vis, wts, exact, 4, half)


@pytest.mark.parametrize("n", [4000, 20000])
def test_dense_blocks_match_oracle(ctx, n):
    """A few blocks hold every entry: the eight warps of a CTA share them."""
    uv, vis, wts = _points(n, n, 64, 0.15)
    _compare(ctx, capi.GaussianSinc, 3, 64, uv, vis, wts, False, 8, True)


def _uneven(seed, n, N):
    """A grid with few entries a block on average: a quarter of them in the blocks around the origin (more than one
    warp takes alone), a quarter at a few dozen entries a block (more than a CTA stages at once), the rest anywhere."""
    uv, vis, wts = _points(seed, n, N, 1.02)
    rng = np.random.default_rng(seed + 1)
    uv[::4] = rng.normal(scale=4.0, size=uv[::4].shape)
    uv[1::4] = rng.uniform(20.0, 100.0, size=uv[1::4].shape)
    return uv, vis, wts


@pytest.mark.parametrize("exact,S", [(False, 3), (True, 3), (False, 5), (True, 6)])
def test_uneven_blocks_match_oracle(ctx, exact, S):
    uv, vis, wts = _uneven(S, 16000, 512)
    _compare(ctx, capi.PSWF, S, 512, uv, vis, wts, exact, 8, True)


def _sparse(seed, n, N):
    """Few entries a block on average, so that a CTA takes eight columns of blocks: half of them anywhere (a warp's few
    entries), the rest in a handful of blocks around the origin (more than one warp takes alone) and in a square of
    some dozen entries a block (staged by the CTA)."""
    uv, vis, wts = _points(seed, n, N, 1.02)
    rng = np.random.default_rng(seed + 1)
    uv[::4] = rng.normal(scale=5.0, size=uv[::4].shape)
    uv[1::4] = rng.uniform(300.0, 340.0, size=uv[1::4].shape)
    return uv, vis, wts


@pytest.mark.parametrize("exact,S,os", [(False, 3, 8), (True, 3, 8), (False, 7, 64), (False, 20, 4), (True, 18, 4)])
def test_sparse_grids_match_oracle(ctx, exact, S, os):
    N = 2308  # 289 columns of blocks: the last CTA's group has one
    uv, vis, wts = _sparse(S, 6000, N)
    _compare(ctx, capi.PSWF, S, N, uv, vis, wts, exact, os, True)


@pytest.mark.parametrize("smax,trunc", [(4, 0.0), (12, 1.0), (20, 0.0)])
def test_sparse_w_grids_match_oracle(ctx, smax, trunc):
    N, cell = 2308, 5.0
    uv, vis, wts = _sparse(smax, 6000, N)
    w = np.random.default_rng(smax).uniform(-3000.0, 3000.0, len(vis))
    kw = dict(num_wplanes=4, max_wpconv_support=smax, kernel_trunc_perc=trunc, w=w, cell_size=cell, analytic_gcf=False)
    r = orc.convolve_to_grid(capi.GaussianSinc, 3, N, uv, vis, wts, False, 4, True, True, True,
                             wproj=orc.WProj(4, smax, 1, trunc), w=w, cell_size=cell, analytic_gcf=False)
    g = ctx.convolve_to_grid(capi.GaussianSinc, 3.0, 3, N, uv, vis, wts, kernel_exact=False, oversampling=4, **kw)
    assert np.abs(g[0] - r.vis_grid).max() <= 1e-11 * np.abs(r.vis_grid).max()
    assert np.abs(g[1] - r.sampling_grid).max() <= 1e-11 * np.abs(r.sampling_grid).max()
    # without the beam, in double and in single precision (tolerance as in test_w_kernels_match_oracle)
    uvw = np.column_stack([uv / (N * np.deg2rad(cell / 3600.0)), w])
    kwi = dict(kernel_func=capi.GaussianSinc, kernel_support=3, kernel_exact=False, oversampling=4, padded_image_size=N,
               gridding_correction=False, num_wplanes=4, max_wpconv_support=smax, kernel_trunc_perc=trunc)
    ref = ctx.image_visibilities(vis, wts, uvw, 300, cell, generate_beam=True, **kwi)[0]
    for precision, tol in ((capi.FP64, 1e-12), (capi.FP32C, 5e-6), (capi.FP32, 5e-6)):
        img = ctx.image_visibilities(vis, wts, uvw, 300, cell, precision=precision, **kwi)[0]
        assert np.abs(img - ref).max() <= tol * np.abs(ref).max(), precision


@pytest.mark.parametrize("smax", [3, 8, 12])
def test_uneven_w_blocks_match_oracle(ctx, smax):
    N, cell = 512, 20.0
    uv, vis, wts = _uneven(smax, 16000, N)
    w = np.random.default_rng(smax).uniform(-3000.0, 3000.0, len(vis))
    kw = dict(num_wplanes=4, max_wpconv_support=smax, kernel_trunc_perc=1.0, w=w, cell_size=cell, analytic_gcf=False)
    r = orc.convolve_to_grid(capi.GaussianSinc, 3, N, uv, vis, wts, False, 4, True, True, True,
                             wproj=orc.WProj(4, smax, 1, 1.0), w=w, cell_size=cell, analytic_gcf=False)
    g = ctx.convolve_to_grid(capi.GaussianSinc, 3.0, 3, N, uv, vis, wts, kernel_exact=False, oversampling=4, **kw)
    assert np.abs(g[0] - r.vis_grid).max() <= 1e-11 * np.abs(r.vis_grid).max()
    assert np.abs(g[1] - r.sampling_grid).max() <= 1e-11 * np.abs(r.sampling_grid).max()


@pytest.mark.parametrize("N", [64, 2308])  # (the second takes the form of sparse grids)
@pytest.mark.parametrize("exact", [True, False])
def test_entries_that_are_not_finite_stay_in_their_footprint(ctx, exact, N):
    S = 3
    uv, vis, wts = _points(3, 200, N, 0.8)
    vis[17] = np.nan
    wts[40] = np.inf
    uv[17] = (10.3, 12.2)
    uv[40] = (-11.4, 20.9)
    with np.errstate(all="ignore"):
        r = orc.convolve_to_grid(capi.PSWF, S, N, uv, vis, wts, exact, 4, True, True, True)
    g = ctx.convolve_to_grid(capi.PSWF, float(S), S, N, uv, vis, wts, kernel_exact=exact, oversampling=4)
    for a, b in ((g[0], r.vis_grid), (g[1], r.sampling_grid)):
        fine = np.isfinite(b.real) & np.isfinite(b.imag)
        assert 0 < (~fine).sum() <= 2 * (2 * S + 1) ** 2
        assert np.array_equal(fine, np.isfinite(a.real) & np.isfinite(a.imag))
        assert np.abs(a[fine] - b[fine]).max() <= 1e-12 * np.abs(b[fine]).max()


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("N,P,smax,trunc", [(28, 2, 3, 0.0), (66, 4, 8, 0.0), (102, 8, 12, 2.0), (130, 5, 16, 0.0),
                                            (256, 3, 40, 0.0)])
def test_w_kernels_match_oracle(ctx, N, P, smax, trunc, precision):
    """Supports below, at and beyond a block's width, planes of different supports, both signs of w, dense blocks."""
    uv, vis, wts = _points(N + smax, 900, N, 1.05)
    uv[::3] *= 0.1  # several hundred entries in the blocks around the origin
    w = np.random.default_rng(N).uniform(-3000.0, 3000.0, len(vis))
    cell = 20.0
    kw = dict(num_wplanes=P, max_wpconv_support=smax, kernel_trunc_perc=trunc, w=w, cell_size=cell, analytic_gcf=False)
    r = orc.convolve_to_grid(capi.GaussianSinc, 3, N, uv, vis, wts, False, 4, True, True, True,
                             wproj=orc.WProj(P, smax, 1, trunc), w=w, cell_size=cell, analytic_gcf=False)
    if precision == "fp64":
        g = ctx.convolve_to_grid(capi.GaussianSinc, 3.0, 3, N, uv, vis, wts, kernel_exact=False, oversampling=4, **kw)
        assert np.abs(g[0] - r.vis_grid).max() <= 1e-11 * np.abs(r.vis_grid).max()
        assert np.abs(g[1] - r.sampling_grid).max() <= 1e-11 * np.abs(r.sampling_grid).max()
        return
    # single-precision kernel values and weighted visibilities (relative error 2^-23 in all, or 1.2e-7 per tap):
    # the image before correction is within that of the peak of the sum of all taps' magnitudes
    inv = N * np.deg2rad(cell / 3600.0)
    uvw = np.column_stack([uv / inv, w])
    kwi = dict(kernel_func=capi.GaussianSinc, kernel_support=3, kernel_exact=False, oversampling=4,
               gridding_correction=False, num_wplanes=P, max_wpconv_support=smax, kernel_trunc_perc=trunc)
    img = ctx.image_visibilities(vis, wts, uvw, N, cell, precision=capi.FP32C, **kwi)[0]
    ref = ctx.image_visibilities(vis, wts, uvw, N, cell, precision=capi.FP64, **kwi)[0]
    assert np.abs(img - ref).max() <= 5e-6 * np.abs(ref).max()


@pytest.mark.parametrize("smax,under,os,P", [(12, 0, 4, 3), (8, 0, 8, 40), (70, 1, 8, 2), (70, 1, 4, 2), (5, 3, 8, 2)])
def test_w_kernel_generation_beyond_shared_memory(ctx, smax, under, os, P):
    """Workareas whose quadrant (16 half^2 bytes), and with support 70 and oversampling 8 its row transforms too, do
    not fit into shared memory, with one and with several CTAs a plane."""
    N, cell = 256, 20.0
    uv, vis, wts = _points(smax + os, 300, N, 0.7)
    uv[:, :] *= 0.6 if smax > 40 else 1.0
    w = np.random.default_rng(smax).uniform(-2000.0, 2000.0, len(vis))
    r = orc.convolve_to_grid(capi.GaussianSinc, 3, N, uv, vis, wts, False, os, True, True, True,
                             wproj=orc.WProj(P, smax, under, 0.0), w=w, cell_size=cell, analytic_gcf=False)
    g = ctx.convolve_to_grid(capi.GaussianSinc, 3.0, 3, N, uv, vis, wts, kernel_exact=False, oversampling=os,
                             num_wplanes=P, max_wpconv_support=smax, undersampling_opt=under, w=w, cell_size=cell,
                             analytic_gcf=False)
    assert np.abs(r.vis_grid).max() > 0
    # double-precision cosine sums over up to 128^2 values in place of an FFT
    assert np.abs(g[0] - r.vis_grid).max() <= 1e-11 * np.abs(r.vis_grid).max()
    assert np.abs(g[1] - r.sampling_grid).max() <= 1e-11 * np.abs(r.sampling_grid).max()


def test_w_kernel_entries_that_are_not_finite_stay_in_their_footprint(ctx):
    N, smax = 64, 4
    uv, vis, wts = _points(5, 200, N, 0.8)
    vis[17] = np.nan
    uv[17] = (10.3, 12.2)
    w = np.linspace(-500.0, 500.0, 200)
    with np.errstate(all="ignore"):
        r = orc.convolve_to_grid(capi.GaussianSinc, 3, N, uv, vis, wts, False, 4, True, True, True,
                                 wproj=orc.WProj(2, smax, 1, 0.0), w=w, cell_size=5.0, analytic_gcf=False)
    g = ctx.convolve_to_grid(capi.GaussianSinc, 3.0, 3, N, uv, vis, wts, kernel_exact=False, oversampling=4,
                             num_wplanes=2, max_wpconv_support=smax, w=w, cell_size=5.0, analytic_gcf=False)
    fine = np.isfinite(r.vis_grid.real) & np.isfinite(r.vis_grid.imag)
    assert (~fine).sum() == (2 * smax + 1) ** 2
    assert np.array_equal(fine, np.isfinite(g[0].real) & np.isfinite(g[0].imag))
    assert np.abs(g[0][fine] - r.vis_grid[fine]).max() <= 1e-11 * np.abs(r.vis_grid[fine]).max()
