"""The sphere limit of the energy flux (csrc/ts_radius.h): |K| <= R exactly where K^2 <= k2_limit(R),
for every radius that ts_flux takes (all but NaN)."""
import math
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
RADII = [0.0, -0.0, 1.0, math.sqrt(2.0), math.sqrt(3.0), math.sqrt(14.0), 7.3, 443.4050067376326, 1e9, 1e-170, 5e-324,
         1e154, 1e200, 1.7976931348623157e308, math.inf, -1.0, -1e-300, -1e200, -math.inf]


@pytest.fixture(scope="module")
def limits(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = tmp_path_factory.mktemp("radius") / "radius"
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", str(ROOT / "tarang_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "radius_main.cpp"), "-o", str(exe)], check=True)
    return lambda R: float(subprocess.run([str(exe), repr(R)], check=True, capture_output=True, text=True, timeout=10).stdout)


@pytest.mark.parametrize("R", RADII)
def test_limit_separates_inside_from_outside(limits, R):
    x = limits(R)
    if R < 0:
        assert x < 0  # K^2 >= 0: no mode is inside
        return
    assert math.sqrt(x) <= R
    up = math.nextafter(x, math.inf)
    assert up == x == math.inf or math.sqrt(up) > R
