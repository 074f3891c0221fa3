"""Range compression where its CTAs are laid out differently: one or two
upsampling phases per CTA (4096 and 8192 points, by storage and by whether the
phases divide evenly), 32768-point spectra folded into two 16384-point
transforms at every upsampling factor up to 16, and rows that end anywhere in a
phase's outputs.  Against the FP64 oracle; tolerances of the size sweep
(tests/test_gpu_rc_sizes.py): FP32 transforms -110 dB, FP16 rows -60 dB."""
import numpy as np
import pytest

from sar_cambrianaccelerationcard_gb300 import metrics, sarbp, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with sarbp.Context(0) as c:
        yield c


@pytest.mark.parametrize("ns,L", [(2501, 1), (2897, 2), (1100, 16), (4097, 1), (5003, 2), (6993, 8), (3100, 16),
                                  (8209, 4), (16000, 1), (15187, 2), (17000, 8), (31001, 4), (15500, 16)])
def test_layouts(ctx, orc, ns, L):
    radar = scenes.Radar(upsample=L)
    s = scenes.config1(np_=3, ns=ns, n_img=8)
    s.radar = radar
    s.t_rec0 = scenes.centred_record_start(radar, ns)
    rng = np.random.default_rng(ns + L)
    echo = (rng.standard_normal((3, ns)) + 1j * rng.standard_normal((3, ns))).astype(np.complex64)
    echo[1] *= 1e-3  # another storage scale
    ref = orc.range_compress(s, echo.astype(np.complex128))
    r, _, lay = sarbp.scene_args(s)
    rc = ctx.range_compress(r, echo)
    h, scale = ctx.range_compress(r, echo, storage=sarbp.STORE_C32H)
    rc16 = (h[..., 0].astype(np.float64) + 1j * h[..., 1].astype(np.float64)) * scale[:, None]
    assert rc.shape == (3, lay.nbins) == rc16.shape
    for p in range(3):
        assert metrics.rel_l2_db(rc[p], ref[p]) <= -110.0
        assert metrics.rel_l2_db(rc16[p], ref[p]) <= -60.0
