"""The contact distance of the mixed path, (float)sqrt(x) from an FP32 root and an exact remainder
(pg_sqrt_float.cuh), gives the bits of the FP64 root rounded: host build of the same code, with the
quotient's estimate exact and off by 2^-20, eight units in the last place where the GPU's is off by at
most two. CPU only."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "perigrain_gb300", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("scale", ["1.0f", "1.000000953674316f", "0.999999046325684f"])
def test_root_rounded_to_float(scale):
    d = tempfile.mkdtemp(prefix="sqrtf_")
    exe = os.path.join(d, "sqrt_float_check")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", f"-DPG_SQRT_FLOAT_EST_SCALE={scale}", "-I", CSRC, "-x", "c++",
                    os.path.join(HERE, "native", "sqrt_float_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "20000", "7"], capture_output=True, text=True, timeout=300).stdout
    assert out.strip().endswith("bad 0"), out
