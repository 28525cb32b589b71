"""The FP32 StVK-Hencky coefficients lose nothing to reciprocals: each is as
close to FP64 as its quotient divided in FP32 (host build of the device code)."""
import os
import subprocess

from ziran2019_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_fp32_coefficients_round_as_divisions(tmp_path):
    exe = str(tmp_path / "hencky")
    subprocess.run([build.NVCC, *build.FLAGS, "-o", exe, os.path.join(HERE, "cpp", "hencky_rounding.cu")], check=True)
    rows = [line.split() for line in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert len(rows) == 36
    for amp, k, mine, plain in rows:
        # 200,000 samples: the two estimates of one error differ by less than 1%
        assert float(mine) <= 1.01 * float(plain), (amp, k, mine, plain)
