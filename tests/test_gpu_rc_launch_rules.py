"""Range compression on both sides of the rules that choose a launch's layout,
against the FP64 oracle: short transforms at 16x upsampling, whose phase table goes
through shared memory at 128 and 256 points, and lengths whose upsampling phases
run one or two per CTA depending on the launch.  Tolerances of the size sweep
(tests/test_gpu_rc_sizes.py): complex64 rows -110 dB, FP16 rows -60 dB."""
import numpy as np
import pytest

from sar_cambrianaccelerationcard_gb300 import metrics, sarbp, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with sarbp.Context(0) as c:
        yield c


def against_oracle(ctx, orc, tp, ns, L, n_p):
    s = scenes.config1(np_=n_p, ns=ns, n_img=8)
    s.radar = scenes.Radar(tp=tp, upsample=L)
    s.t_rec0 = scenes.centred_record_start(s.radar, ns)
    rng = np.random.default_rng(ns + L)
    echo = (rng.standard_normal((n_p, ns)) + 1j * rng.standard_normal((n_p, ns))).astype(np.complex64)
    ref = orc.range_compress(s, echo.astype(np.complex128))
    r, _, _ = sarbp.scene_args(s)
    rc = ctx.range_compress(r, echo)
    h, scale = ctx.range_compress(r, echo, storage=sarbp.STORE_C32H)
    rc16 = (h[..., 0].astype(np.float64) + 1j * h[..., 1].astype(np.float64)) * scale[:, None]
    assert metrics.rel_l2_db(rc, ref) <= -110.0
    assert metrics.rel_l2_db(rc16, ref) <= -60.0


@pytest.mark.parametrize("nfft", [64, 128, 256, 512])
@pytest.mark.parametrize("L", [8, 16])
def test_short_transforms(ctx, orc, nfft, L):
    tp = 0.05e-6  # 6 samples
    against_oracle(ctx, orc, tp, nfft - 6, L, 5)
    against_oracle(ctx, orc, tp, nfft // 2 - 3, L, 5)  # the shortest rows of the size


@pytest.mark.parametrize("ns,L", [(2897, 2), (1501, 4), (2501, 8), (1100, 16), (6993, 2), (5003, 4), (4001, 8), (6001, 16)])
def test_single_and_paired_phases(ctx, orc, ns, L):
    """A pulse's row has the same bits in launches of any number of pulses, on
    either side of every bound of the rule, and matches the oracle in the smallest."""
    torch = pytest.importorskip("torch")
    against_oracle(ctx, orc, 10e-6, ns, L, 2)
    n = 700
    r = sarbp.radar_struct(scenes.Radar(upsample=L), 3e-5)
    g = torch.Generator("cuda").manual_seed(ns)
    echo = torch.view_as_complex(torch.randn(n, ns, 2, device="cuda", generator=g))
    full = torch.empty(n, L * ns, dtype=torch.complex64, device="cuda")
    half = torch.empty(n, L * ns, 2, dtype=torch.float16, device="cuda")
    scale = torch.empty(n, device="cuda")
    torch.cuda.synchronize()
    ctx.range_compress(r, echo, out=full)
    ctx.range_compress(r, echo, sarbp.STORE_C32H, out=half, scale=scale)
    ctx.synchronize()
    for m in (1, 152 // L, 152 // L + 1, 304 // L + 1, 456 // L, 456 // L + 1, 608 // L + 1, 350):
        m = max(1, m)
        a = torch.empty(m, L * ns, dtype=torch.complex64, device="cuda")
        h = torch.empty(m, L * ns, 2, dtype=torch.float16, device="cuda")
        c = torch.empty(m, device="cuda")
        ctx.range_compress(r, echo[:m], out=a)
        ctx.range_compress(r, echo[:m], sarbp.STORE_C32H, out=h, scale=c)
        ctx.synchronize()
        assert torch.equal(torch.view_as_real(a), torch.view_as_real(full[:m])), m
        assert torch.equal(h, half[:m]) and torch.equal(c, scale[:m]), m
