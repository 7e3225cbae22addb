"""The quotient beta = rrn / rro that the on-chip CG loops form from the reciprocal of rro
(csrc/tl_fp64emu.cuh), built for the host, against the division: the same bits over all exponents, the
range where the remainder is not exact among them (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_quotient_from_a_reciprocal_is_the_division(tmp_path):
    exe = str(tmp_path / "quotient_host")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "tealeaf_ref_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "quotient_host.cpp"), "-o", exe], check=True)
    for seed in (1, 2):
        r = subprocess.run([exe, "8000000", str(seed)], capture_output=True, text=True)
        assert r.returncode == 0 and "mismatch 0" in r.stdout, r.stdout + r.stderr
