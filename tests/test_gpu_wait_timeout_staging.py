"""The bounded staging waits in the scheme of the usual 32 x 64 tiles with 16-pulse
chunks: two helper warps stage chunk c + 1 beside the pixel warps' chunk c, so the
wait that runs out is inside the helpers and the vote at the end of the
iteration; the first chunk's is ahead of the loop.  As in the other wait tests the
fault is 16 bytes that the drain delivers, the limit 200 us, and nothing hangs:
the call returns SARBP_ERR_TIMEOUT with its copies landed, and the context then
gives the bits of one that never faulted.  A limit without a fault gives the
production bits."""
import numpy as np
import pytest

from sar_cambrianaccelerationcard_gb300 import sarbp, scenes

pytestmark = pytest.mark.gpu

WAIT_TIMEOUT_BIT = 1
DRAIN_TIMEOUT_BIT = 16
PULSES = 200  # 13 chunks, the last of 8 pulses


@pytest.fixture(scope="module")
def case():
    s = scenes.config1(np_=PULSES, ns=1024, n_img=150, spacing=0.25)
    r, g, lay = sarbp.scene_args(s)
    with sarbp.Context(0) as ctx:
        echo = sarbp.synthesize(ctx, s)
        rc = ctx.range_compress(r, echo)
        h, scale = ctx.range_compress(r, echo, storage=sarbp.STORE_C32H)
        v = sarbp.RcView()
        v.storage, v.np, v.nbins, v.t0_bins, v.bin_rate = sarbp.STORE_C64, PULSES, lay.nbins, lay.t0_bins, lay.bin_rate
        info = ctx.bp_plan(r, v, s.apc, g, sarbp.MODE_SPLIT)
        assert (info.pulse_chunk, info.tile_y, info.linear_phase) == (16, 64, 0)
    w = (np.random.default_rng(3).standard_normal((g.ny, g.nx)) + 0j).astype(np.complex64)

    def call(ctx, kind):
        rows, sc = (h, scale) if kind.endswith("fp16") else (rc, None)
        mode = sarbp.MODE_FP16STORE if kind.endswith("fp16") else sarbp.MODE_SPLIT
        if kind.startswith("project"):
            return ctx.project_weighted(r, rows, s.apc, g, mode, lay.t0_bins, lay.bin_rate, w, scale=sc)
        return ctx.backproject(r, rows, s.apc, g, mode, lay.t0_bins, lay.bin_rate, scale=sc)
    return call


@pytest.mark.parametrize("kind", ["image", "image_fp16", "project", "project_fp16"])
@pytest.mark.parametrize("chunk", [0, 1, 2, 3, 6, 11, 12])
def test_helper_wait_runs_out_then_drains_and_recovers(case, kind, chunk):
    with sarbp.Context(0) as ctx:
        ctx.debug_set(sarbp.DEBUG_BP_SEGMENTS, 1)
        ref = case(ctx, kind)
        ctx.debug_set(sarbp.DEBUG_WAIT_LIMIT_NS, 200_000)
        ctx.debug_set(sarbp.DEBUG_WAIT_FAULT_CHUNK, chunk)
        with pytest.raises(sarbp.SarbpError) as e:
            case(ctx, kind)
        assert e.value.status == sarbp.ERR_TIMEOUT, str(e.value)
        flags = ctx.debug_get(sarbp.DEBUG_DEVICE_FLAGS)
        assert flags & WAIT_TIMEOUT_BIT, hex(flags)
        assert not flags & DRAIN_TIMEOUT_BIT, f"a copy was still in flight after the drain ({flags:#x})"
        ctx.debug_set(sarbp.DEBUG_WAIT_FAULT_CHUNK, -1)
        ctx.debug_set(sarbp.DEBUG_WAIT_LIMIT_NS, 0)
        assert np.array_equal(case(ctx, kind), ref)


@pytest.mark.parametrize("kind", ["image", "image_fp16", "project", "project_fp16"])
def test_limit_without_a_fault(case, kind):
    with sarbp.Context(0) as ctx:
        ref = case(ctx, kind)
        ctx.debug_set(sarbp.DEBUG_WAIT_LIMIT_NS, 500_000_000)
        assert np.array_equal(case(ctx, kind), ref)
