"""Back-projection and projection calls of one context on several streams, queued
back to back without a wait: the context's scratch (pulse references, partial
images, projection sums) must not be overwritten by a later call while an
earlier one still reads it.  Every result has the bits of the same call alone."""
import numpy as np
import pytest

from sar_cambrianaccelerationcard_gb300 import sarbp, scenes

pytestmark = pytest.mark.gpu


def test_calls_on_different_streams():
    torch = pytest.importorskip("torch")
    with sarbp.Context(0) as ctx:
        s = scenes.config1(np_=1500, ns=1024, n_img=700)
        r, g, lay = sarbp.scene_args(s)
        rc = torch.from_numpy(ctx.range_compress(r, sarbp.synthesize(ctx, s))).cuda()
        rng = np.random.default_rng(1)
        tracks = [torch.from_numpy(s.apc + rng.normal(0, 0.2, s.apc.shape)).cuda() for _ in range(4)]
        weight = torch.from_numpy((rng.standard_normal((700, 700)) + 0j).astype(np.complex64)).cuda()
        images = [torch.zeros(700, 700, dtype=torch.complex64, device="cuda") for _ in tracks]
        sums = [torch.zeros(1500, dtype=torch.complex128, device="cuda") for _ in tracks]
        streams = [torch.cuda.Stream() for _ in tracks]

        def call(k, stream):
            ctx.backproject(r, rc, tracks[k], g, sarbp.MODE_SPLIT, lay.t0_bins, lay.bin_rate, image=images[k],
                            stream=stream)
            ctx.project_weighted(r, rc, tracks[k], g, sarbp.MODE_SPLIT, lay.t0_bins, lay.bin_rate, weight, out=sums[k],
                                 stream=stream)

        alone = []
        for k in range(4):
            torch.cuda.synchronize()
            call(k, streams[0].cuda_stream)
            torch.cuda.synchronize()
            alone.append((images[k].clone(), sums[k].clone()))
        for _ in range(3):
            for k in range(4):
                images[k].zero_()
                sums[k].zero_()
            torch.cuda.synchronize()
            for k in range(4):
                call(k, streams[k].cuda_stream)
            ctx.synchronize()
            for k in range(4):
                assert torch.equal(torch.view_as_real(images[k]), torch.view_as_real(alone[k][0])), k
                assert torch.equal(torch.view_as_real(sums[k]), torch.view_as_real(alone[k][1])), k
