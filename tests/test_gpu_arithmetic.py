"""The shortened divisions and square roots of the gather, the field and the Volkov passes (csrc/quotient.cuh,
csrc/phasor.cuh) against CUDA's division and 64-bit arithmetic, special values included; the bounds stand beside each
check in arith_check.cu."""
import pathlib
import subprocess

import pytest

from mtd_transmission_gb300 import build

HERE = pathlib.Path(__file__).resolve().parent
pytestmark = pytest.mark.gpu


def test_shortened_arithmetic(tmp_path):
    exe = tmp_path / "arith_check"
    subprocess.run([build._nvcc(), build.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", f"-I{build.CSRC}",
                    str(HERE / "arith_check.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    rows = [line.split() for line in out.stdout.splitlines()]
    assert len(rows) == 9
    for name, worst, bad, seen in rows:
        assert int(seen) > 0 and int(bad) == 0, out.stdout
