"""Pulse segments of small images, checked on the CPU through the library's own rules:
where the wave rule splits the pulses but leaves SMs without a CTA, more segments,
down to a chunk of 16 pulses each, whether or not the pulses are a whole number of
chunks."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sar_cambrianaccelerationcard_gb300")
LIB = os.path.join(PKG, "libsarbp.so")
SMS, CHUNK = 152, 16

HARNESS = r"""
#include <cstdio>
#include "sarbp_internal.h"
int main() {
    int tiles, npl;
    while (scanf("%d %d", &tiles, &npl) == 2) {
        const int a = sarbp::bp_choose_segments(tiles, npl, 2048LL * tiles, 152);
        printf("%d %d\n", a, sarbp::bp_fill_segments(tiles, npl, 152, a));
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def segments(tmp_path_factory):
    cuda = next((d for d in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda")
                 if d and os.path.exists(os.path.join(d, "include", "cuda_runtime.h"))), None)
    if not (shutil.which("g++") and cuda and os.path.exists(LIB)):
        pytest.skip("needs g++, the CUDA headers and the built library")
    d = tmp_path_factory.mktemp("fill")
    src, exe = d / "harness.cpp", d / "harness"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(cuda, "include"), str(src), "-o", str(exe), LIB, f"-Wl,-rpath,{PKG}"], check=True)

    def run(cases):
        out = subprocess.run([str(exe)], input="".join(f"{t} {n}\n" for t, n in cases), capture_output=True, text=True,
                             check=True).stdout.split()
        return list(zip(map(int, out[0::2]), map(int, out[1::2])))
    return run


def pulses_per_segment(npl, s):
    return -(-(-(-npl // s)) // CHUNK) * CHUNK


def test_small_images_fill_the_chip(segments):
    cases = [(t, n) for t in (1, 2, 3, 8, 16, 28, 40, 75, 76, 151, 152, 500)
             for n in [*range(1, 700, 7), 128, 250, 256, 512, 1000, 1024, 4000, 4096, 20000]]
    refined = set()
    for (tiles, npl), (wave, s) in zip(cases, segments(cases)):
        assert wave <= s <= 64
        if s == wave:
            refined.add(False)
        else:
            refined.add(True)
            assert wave >= 2 and tiles * wave < SMS
            assert (s - 1) * pulses_per_segment(npl, s) < npl  # no empty segment
        if wave >= 2 and 4 * tiles * s < 3 * SMS and s < 64:
            # a quarter of the SMs idle: only because no larger count has pulses for every
            # segment, whole chunks of them where some SMs would get a second CTA
            assert not any((k - 1) * pulses_per_segment(npl, k) < npl and (tiles * k <= SMS or npl // k >= CHUNK)
                           for k in range(s + 1, 65)), (tiles, npl, s)
    assert refined == {False, True}


def test_pulse_counts_near_each_other_are_split_alike(segments):
    (_, a), (_, b) = segments([(8, 250), (8, 256)])
    assert a == b == 16
