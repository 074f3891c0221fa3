"""Calls of one context queued back to back without a wait, on streams of their
own: none may touch the context's scratch, or replace its tables, while an
earlier call still uses them.  Every result has the bits of the same call alone."""
import numpy as np
import pytest

from sar_cambrianaccelerationcard_gb300 import sarbp, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return pytest.importorskip("torch")


def bits(torch, x):
    return (torch.view_as_real(x) if x.is_complex() else x).view(torch.int16)


def check(torch, ctx, calls, one_stream=False):
    """calls: (queue(stream), outputs) pairs; each alone, then all in flight at once, three times."""
    alone = []
    for queue, outs in calls:
        torch.cuda.synchronize()
        queue(torch.cuda.Stream().cuda_stream)
        torch.cuda.synchronize()
        alone.append([o.clone() for o in outs])
    streams = [torch.cuda.Stream() for _ in range(1 if one_stream else len(calls))] * (len(calls) if one_stream else 1)
    for _ in range(3):
        for _, outs in calls:
            for o in outs:
                o.zero_()
        torch.cuda.synchronize()
        for (queue, _), s in zip(calls, streams):
            queue(s.cuda_stream)
        ctx.synchronize()
        for k, (_, outs) in enumerate(calls):
            for o, ref in zip(outs, alone[k]):
                assert torch.equal(bits(torch, o), bits(torch, ref)), k


def noise(torch, k, *shape):
    g = torch.Generator("cuda").manual_seed(k)
    return torch.view_as_complex(torch.randn(*shape, 2, device="cuda", generator=g)) * 10.0 ** -k


@pytest.mark.parametrize("ns", [2500, 20000])  # one transform per CTA, and the folded 32768-point layout
def test_range_compression(torch, ns):
    n_p = 4_000_000 // ns
    with sarbp.Context(0) as ctx:
        r = sarbp.radar_struct(scenes.Radar(upsample=4), 3e-5)
        calls = []
        for k in range(4):
            echo = noise(torch, k, n_p, ns)
            if k % 2:
                out = torch.zeros(n_p, 4 * ns, 2, dtype=torch.float16, device="cuda")
                scale = torch.zeros(n_p, device="cuda")
                calls.append((lambda s, e=echo, o=out, c=scale: ctx.range_compress(r, e, sarbp.STORE_C32H, out=o, scale=c,
                                                                                  stream=s), [out, scale]))
            else:
                out = torch.zeros(n_p, 4 * ns, dtype=torch.complex64, device="cuda")
                calls.append((lambda s, e=echo, o=out: ctx.range_compress(r, e, out=o, stream=s), [out]))
        check(torch, ctx, calls)


def test_images(torch):
    s = scenes.config1(np_=700, ns=2000, n_img=300)
    r, g, _ = sarbp.scene_args(s)
    apc = torch.from_numpy(s.apc).cuda()
    with sarbp.Context(0) as ctx:
        calls = []
        for k in range(4):
            echo = noise(torch, k, 700, 2000)
            img = torch.zeros(300, 300, dtype=torch.complex64, device="cuda")
            mode = sarbp.MODE_FP16STORE if k % 2 else sarbp.MODE_SPLIT
            calls.append((lambda st, e=echo, i=img, m=mode: ctx.image(r, e, apc, g, m, image=i, stream=st), [img]))
        check(torch, ctx, calls)


def test_transposed_transforms(torch):
    with sarbp.Context(0) as ctx:
        calls = []
        for k in range(4):
            x = noise(torch, k, 700, 300)  # 700 points down the columns: through transposes
            out = torch.zeros_like(x)

            def dft(st, x=x, out=out):
                with torch.cuda.stream(torch.cuda.ExternalStream(st)):
                    out.copy_(x)
                ctx.dft2d(out, stream=st)
            calls.append((dft, [out]))
        check(torch, ctx, calls)


@pytest.mark.parametrize("one_stream", [True, False])
def test_parameters_change_between_queued_calls(torch, one_stream):
    with sarbp.Context(0) as ctx:
        calls = []
        for k in range(4):  # one layout, other chirps: the same tables' memory
            radar = scenes.Radar(bandwidth=100e6 if k % 2 else 90e6)
            r = sarbp.radar_struct(radar, 3e-5)
            echo = noise(torch, k, 1500, 2500)
            out = torch.zeros(1500, 8 * 2500, dtype=torch.complex64, device="cuda")
            calls.append((lambda s, r=r, e=echo, o=out: ctx.range_compress(r, e, out=o, stream=s), [out]))
        check(torch, ctx, calls, one_stream)
        assert not torch.equal(calls[0][1][0], calls[1][1][0])


@pytest.mark.parametrize("one_stream", [True, False])
def test_more_dft_lengths_than_kept_tables(torch, one_stream):
    with sarbp.Context(0) as ctx:
        calls = []
        for k, n in enumerate((1000, 1024, 1500, 2048, 3000, 999)):
            x = noise(torch, k, 4000, n)
            out = torch.zeros_like(x)

            def dft(st, x=x, out=out):
                with torch.cuda.stream(torch.cuda.ExternalStream(st)):
                    out.copy_(x)
                ctx.dft(out, stream=st)
            calls.append((dft, [out]))
        check(torch, ctx, calls, one_stream)


def test_captured_range_compression_replays(torch):
    """A device-buffer call is captured into a graph after a first one (which uploads the
    tables and sizes the scratch) and replays on new data."""
    with sarbp.Context(0) as ctx:
        r = sarbp.radar_struct(scenes.Radar(upsample=4), 3e-5)
        a, b = noise(torch, 0, 300, 2500), noise(torch, 1, 300, 2500)
        echo, out = a.clone(), torch.zeros(300, 4 * 2500, dtype=torch.complex64, device="cuda")
        torch.cuda.synchronize()
        ctx.range_compress(r, b, out=out)
        ctx.synchronize()
        ref = out.clone()
        graph = torch.cuda.CUDAGraph()
        stream = torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=stream):
            ctx.range_compress(r, echo, out=out, stream=stream.cuda_stream)
        echo.copy_(b)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(torch.view_as_real(out), torch.view_as_real(ref))
        ctx.range_compress(r, a, out=out)  # the context goes on as before
        ctx.synchronize()
        assert not torch.equal(torch.view_as_real(out), torch.view_as_real(ref))
