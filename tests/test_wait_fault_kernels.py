"""The kernels that test the bounded waits (shortened limit, injected fault) run
the staging schemes of production: for every series-form back-projection and
projection kernel of 32 x 64 tiles that production launches, one with the same
mode, storage, terms and pulse chunk is built with the test switches.  Checked on the
CPU from the library's symbol names."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "sar_cambrianaccelerationcard_gb300", "libsarbp.so")


def test_wait_fault_kernels_cover_the_production_schemes():
    if not (shutil.which("nm") and os.path.exists(LIB)):
        pytest.skip("needs nm and the built library")
    names = subprocess.run(["nm", "-C", LIB], capture_output=True, text=True, check=True).stdout
    # <mode, storage, terms, checked, pixels, projection, chunk, test switches, linear>
    kernels = {tuple(m.split(", ")) for m in re.findall(r"bp_kernel<([^>]*)>\(", names)}
    assert kernels and all(len(k) == 9 for k in kernels)
    production = {k for k in kernels if k[3:5] == ("false", "8") and k[7:] == ("false", "false")}
    assert {k[6] for k in production} == {"0", "16"}
    missing = {k for k in production if k[:7] + ("true", "false") not in kernels}
    assert not missing, sorted(missing)
