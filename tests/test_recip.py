"""The projection's quotients (csrc/ts_common.cuh, recip and quot1, run on the host) carry the one
rounding of a division: half a unit in the last place, where a product with the rounded reciprocal
has up to one and a half; and they are 0 where K^2 is 0 or infinite."""
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
NVCC = Path(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))


def test_quotients_round_as_a_division(tmp_path):
    if not NVCC.exists():
        pytest.skip("no nvcc")
    exe = tmp_path / "recip"
    subprocess.run([str(NVCC), "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    str(ROOT / "tarang_b200" / "csrc"), str(ROOT / "tests" / "cpp" / "recip_main.cu"), "-o", str(exe)], check=True)
    f32, f64, zero, inf = map(float, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert 0.49 < f32 < 0.5001 and 0.49 < f64 < 0.501  # 0.501: the long double quotient has 11 bits more
    assert zero == 0 and inf == 0
