"""Staging of the back-projection kernels at the edges of rows and chunks.

The production kernels convert only the range bins a tile reads, without bounds
tests where a window lies inside its row; with 16-pulse chunks of 32 x 64 tiles
two extra warps do it beside the pixel loop.  The checked kernels convert every
window whole, bin by bin with bounds tests, and report any read outside it.
Both run the same pixel arithmetic, so their images have to be the same bits,
here for rows shorter than the scene (windows inside the row, across either end
and outside it), ragged grids and pulse counts around the chunk size, in every
chunk, tile height and phase form the planner can pick."""
import numpy as np
import pytest

from sar_cambrianaccelerationcard_gb300 import sarbp, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with sarbp.Context(0) as c:
        yield c


def rows(n_p, nbins, storage, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n_p, nbins, 2)).astype(np.float32)
    if storage == sarbp.STORE_C64:
        return x.view(np.complex64)[..., 0].copy(), None
    return x.astype(np.float16), np.exp2(rng.integers(-3, 4, n_p)).astype(np.float32)


@pytest.mark.parametrize("storage", [sarbp.STORE_C64, sarbp.STORE_C32H])
@pytest.mark.parametrize("n_p", [1, 15, 16, 17, 50])
@pytest.mark.parametrize("spacing,chunk,linear", [(0.25, 0, 0), (0.25, 0, 1), (0.25, 8, 0), (0.75, 0, 0), (1.3, 4, 0),
                                                  (2.2, 0, 0)])
def test_rows_shorter_than_the_scene(ctx, storage, n_p, spacing, chunk, linear):
    radar = scenes.Radar()
    mode = sarbp.MODE_SPLIT if storage == sarbp.STORE_C64 else sarbp.MODE_FP16STORE
    grid = scenes.centred_grid(radar, 301, 67, spacing)
    if spacing > 1.0:  # 45 degrees to the track: the wide windows and short tiles
        s = spacing / np.sqrt(2.0)
        grid.ux, grid.uy = np.array([s, s, 0.0]), np.array([s, -s, 0.0])
        grid.origin = np.array([0.0, radar.r0, 0.0]) - 150 * grid.ux - 33 * grid.uy
    bins_per_m = 2.0 / radar.c * radar.upsample * radar.fs
    span = 301 * spacing * (1.0 if spacing < 1.0 else 0.7)
    nbins = 4 * int(0.5 * span * bins_per_m / 4)  # rows over the middle half of the scene's ranges
    t0 = (radar.r0 - 0.25 * span) * 2.0 / radar.c
    apc = scenes.straight_track(radar, n_p)
    data, scale = rows(n_p, nbins, storage, n_p)
    r, g = sarbp.radar_struct(radar, t0), sarbp.grid_struct(grid)
    args = (r, data, apc, g, mode, t0, radar.upsample * radar.fs)
    try:
        ctx.debug_set(sarbp.DEBUG_BP_CHUNK, chunk)
        ctx.debug_set(sarbp.DEBUG_BP_LINEAR_PHASE, linear)
        image = ctx.backproject(*args, scale=scale)
        ctx.debug_set(sarbp.DEBUG_BP_CHECKED, 1)
        checked = ctx.backproject(*args, scale=scale)
    finally:
        ctx.debug_set(sarbp.DEBUG_BP_CHECKED, 0)
        ctx.debug_set(sarbp.DEBUG_BP_LINEAR_PHASE, 0)
        ctx.debug_set(sarbp.DEBUG_BP_CHUNK, 0)
    assert np.array_equal(image, checked)
    mag = np.abs(image)
    assert mag.max() > 0 and (mag == 0).any()  # part of the scene lies outside the rows
