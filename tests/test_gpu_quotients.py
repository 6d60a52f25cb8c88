"""The FP64 step's short quotient forms on the device: against plain division over the operands
that their range checks admit and refuse, and within the update, which must not depend on the form
taken (native/quotient_check.cu, compiled as the FP64 kernels are)."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
CSRC = os.path.join(REPO, "clip_b200", "csrc")

pytestmark = pytest.mark.gpu


def test_short_quotients_are_the_quotients(tmp_path):
    sys.path.insert(0, os.path.join(REPO, "clip_b200"))
    import build

    exe = str(tmp_path / "quotient_check")
    subprocess.run([build.nvcc(), "-std=c++17", "-O3", "-I", CSRC, *build.ARCH, *build.UNITS["kernels_fp64.cu"],
                    os.path.join(HERE, "native", "quotient_check.cu"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stdout + res.stderr
    lines = dict(l.split(": ", 1) for l in res.stdout.strip().splitlines())
    assert list(lines) == ["by constants", "by density", "ranges", "2D update", "3D update"]
    for dim in ("2D", "3D"):  # both forms are met
        assert 10000 < int(lines[dim + " update"].split("short form ")[1].split()[0]) < 65000
