"""The device reduction of the planning extremes, whose FP32 pass rules points
out before the FP64 evaluation, against every point evaluated in FP64: the same
bits for geometries where the pass is tight or useless (coordinates far larger
than the distances, satellite ranges, many equal points, an axis across every
line of sight, one pulse, more pulses than a block), and a non-finite antenna
position still found anywhere."""
import numpy as np
import pytest

from sar_cambrianaccelerationcard_gb300 import sarbp, scenes
from test_gpu_plan import brute_extremes, view

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with sarbp.Context(0) as c:
        yield c


def scene(name):
    s = scenes.config1(np_=777, n_img=129)
    rng = np.random.default_rng(3)
    if name == "one_pulse":
        s = scenes.config1(np_=1, n_img=129)
    elif name == "many_pulses":
        s = scenes.config1(np_=20011, n_img=2001, spacing=0.3)
    elif name == "earth_centred":
        off = np.array([4.1e6, -2.3e6, 4.2e6])
        s.apc, s.grid.origin = s.apc + off, s.grid.origin + off
    elif name == "satellite":
        s.apc = s.apc * 50.0 + np.array([0.0, -2.5e5, 7.9e5])
    elif name == "jitter":
        s.apc = s.apc + rng.normal(0, 30.0, s.apc.shape)
    elif name == "same_position":
        s.apc = np.repeat(s.apc[:1], len(s.apc), axis=0)
    elif name == "axis_across":  # the grid's y axis is perpendicular to every line of sight
        s.grid.uy = np.array([0.0, 0.0, 0.5])
        s.grid.ny = 1
        s.apc = s.apc * 1.0
        s.apc[:, 2] = 0.0
    return s


@pytest.mark.parametrize("name", ["plain", "one_pulse", "many_pulses", "earth_centred", "satellite", "jitter",
                                  "same_position", "axis_across"])
def test_device_extremes_equal_every_point(ctx, name):
    s = scene(name)
    apc = np.ascontiguousarray(s.apc)
    r, g, _ = sarbp.scene_args(s)
    want = brute_extremes(apc, g)
    for _ in range(2):  # the reduction's state is ready for the next call
        info = ctx.bp_plan(r, view(s), apc, g, sarbp.MODE_FP64)
        assert (info.rmin, info.rmax, info.cos_x, info.cos_y) == want


@pytest.mark.parametrize("pulse", [0, 400, 776])
def test_nonfinite_position_is_found_and_forgotten(ctx, pulse):
    s = scene("plain")
    r, g, _ = sarbp.scene_args(s)
    bad = s.apc.copy()
    bad[pulse, pulse % 3] = np.nan
    with pytest.raises(sarbp.SarbpError, match="finite"):
        ctx.bp_plan(r, view(s), bad, g, sarbp.MODE_FP64)
    info = ctx.bp_plan(r, view(s), np.ascontiguousarray(s.apc), g, sarbp.MODE_FP64)
    assert (info.rmin, info.rmax, info.cos_x, info.cos_y) == brute_extremes(s.apc, g)
