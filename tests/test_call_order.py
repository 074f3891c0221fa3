"""What orders the memory accesses of a context's calls, checked on the CPU.

tests/shim/call_order.cpp links the library's host code with a CUDA runtime of
its own, which runs nothing and follows what each stream, event and host wait
orders: two accesses to the same bytes, one of them a write, that nothing orders
are reported, whatever the timing would have been on a device.  Device-pointer
calls are asynchronous on the caller's stream, so whatever they share in the
context has to be ordered by the calls themselves."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sar_cambrianaccelerationcard_gb300", "csrc")

CALLS = ["autofocus", "bp", "bp_fp16", "bp_host", "ceos", "ceos_host", "dft", "dft2d", "dft_host", "image", "image_fp16",
         "image_host", "plan", "project", "project_host", "rc", "rc_32768", "rc_fp16", "rc_host", "synth", "synth_host",
         "wk", "wk_focus", "wk_preprocess"]


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    cuda = next((d for d in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda")
                 if d and os.path.exists(os.path.join(d, "include", "cuda_runtime.h"))), None)
    if not (shutil.which("g++") and cuda):
        pytest.skip("needs g++ and the CUDA headers")
    exe = tmp_path_factory.mktemp("order") / "call_order"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    "-I", os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "shim", "call_order.cpp"),
                    os.path.join(CSRC, "api.cpp"), os.path.join(CSRC, "plan.cpp"), "-o", str(exe)], check=True)

    def call(*args):
        r = subprocess.run([str(exe), *args], capture_output=True, text=True)
        return r.returncode, r.stdout
    return call


def test_detector_and_call_list(run):
    assert run("detector")[0] == 0
    assert run("list")[1].split() == CALLS


@pytest.mark.parametrize("name", CALLS)
def test_first_call_of_a_context(run, name):
    """Tables and state uploaded for the first call are on the device before its launches read them."""
    rc, out = run("first", name)
    assert rc == 0, out


@pytest.mark.parametrize("name", CALLS)
def test_calls_on_streams_of_their_own(run, name):
    """A call, each other call and the first again, on three streams, without a wait between them."""
    rc, out = run("streams", name)
    assert rc == 0, out


def test_call_behind_a_failed_one(run):
    """What a failing call had queued is ordered before the next call too."""
    rc, out = run("failed")
    assert rc == 0, out


@pytest.mark.parametrize("name", ["rc", "rc_fp16", "rc_32768", "rc_host", "image", "image_fp16", "image_host", "dft", "dft2d",
                                  "wk", "wk_focus", "ceos", "ceos_host"])
def test_tables_are_not_replaced_under_queued_launches(run, name):
    """Two sets of parameters in turn, queued without a wait on one stream and on two."""
    rc, out = run("tables", name)
    assert rc == 0, out


def test_more_dft_lengths_than_kept_tables(run):
    rc, out = run("lengths")
    assert rc == 0, out


@pytest.mark.parametrize("n_p,ns,L", [(20, 900, 8), (300, 2000, 8), (1111, 4000, 8), (3000, 14000, 2), (3001, 900, 1),
                                      (8000, 2000, 4), (8000, 6000, 8), (5000, 14000, 1)])
def test_upload_chunks(run, n_p, ns, L):
    """A host echo goes up in chunks of 256 pulses and then half as many again, up to
    an eighth of the pulses, or 1024 where compression takes as long as the copy, or
    without a bound where it takes twice that; the last chunk, whose compression nothing
    hides, is no larger than a quarter above the bound."""
    rc, out = run("uploads", str(n_p), str(ns), str(L))
    assert rc == 0, out
    chunks = [int(x) for x in out.splitlines()[0].split()]
    nfft = 1 << (ns + 1200 - 2).bit_length()
    load = (1 + L) * nfft // ns
    bound = n_p if load >= 18 else max(1024 if load >= 9 else 256, -(-n_p // 8))
    assert sum(chunks) == n_p and chunks[0] == min(n_p, 256 if n_p >= 320 else n_p)
    assert max(chunks) <= bound + bound // 4
    for a, b in zip(chunks, chunks[1:-1]):
        assert a <= b <= a + a // 2


@pytest.mark.parametrize("n_p,ns,L", [(3000, 900, 8), (8000, 2000, 8), (3000, 14000, 2)])
def test_first_host_echo_frees_nothing(run, n_p, ns, L):
    """A context's first host call sizes its scratch once: growing it between chunks would
    free, and so wait for the copies and launches in flight."""
    rc, out = run("uploads", str(n_p), str(ns), str(L))
    assert rc == 0 and out.splitlines()[1] == "0 buffers freed", out
