"""The cap gather's form for every accepted band and angle count fits a CTA's shared memory, static bytes included
(mtd_transmission_gb300/csrc/gather_smem.cuh, host arithmetic, no GPU)."""
import pathlib
import subprocess

from mtd_transmission_gb300 import build

HERE = pathlib.Path(__file__).resolve().parent


def test_chosen_form_fits(tmp_path):
    exe = tmp_path / "gather_smem_check"
    subprocess.run([build._nvcc(), build.ARCH, "-O2", "-std=c++17", f"-I{build.CSRC}",
                    str(HERE / "gather_smem_check.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
