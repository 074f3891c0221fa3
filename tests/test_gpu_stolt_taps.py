"""The Stolt stage at tap counts compiled in (4, 6, 8) and general ones, on rows
short enough that most outputs clip at the ends and on long ones, against the
FP64 restatement.  Tolerance as for the omega-K image: FP32 weights and phases,
-80 dB."""
import dataclasses

import numpy as np
import pytest

from oracle import wk
from sar_cambrianaccelerationcard_gb300 import metrics, sarbp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with sarbp.Context(0) as c:
        yield c


@pytest.mark.parametrize("taps", [1, 3, 4, 5, 6, 7, 8, 12])
@pytest.mark.parametrize("shape", [(64, 7), (37, 130), (16, 1001)])
def test_taps(ctx, shape, taps):
    p = dataclasses.replace(wk.radarsat1(), taps=taps)
    rng = np.random.default_rng(taps + shape[1])
    spec = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    ref = wk.rfm_stolt(spec.astype(np.complex128), p)
    got = ctx.wk_focus(p, spec)
    assert np.isfinite(got.view(np.float32)).all()
    assert metrics.rel_l2_db(got, ref) <= -80.0
