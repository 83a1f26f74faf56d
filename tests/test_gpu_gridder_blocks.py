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


@pytest.mark.parametrize("exact", [True, False])
def test_entries_that_are_not_finite_stay_in_their_footprint(ctx, exact):
    N, S = 64, 3
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
