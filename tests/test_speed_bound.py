"""The FP32 bound of a face point's wave speed (rkdg3d_gb300/csrc/rkdg_speed_bound.h)
lies above the FP64 speed, checked on the CPU by tests/speed_bound_check.cpp over
the elements' face rows, gases, Mach numbers, jumps and normals."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "rkdg3d_gb300", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("speedbound") / "check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "speed_bound_check.cpp"),
                    os.path.join(CSRC, "rkdg_refelem.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("geom,order", [(2, 1), (2, 2), (3, 1), (3, 2), (3, 3), (5, 1), (5, 2)])
def test_bound_holds(checker, geom, order):
    out = subprocess.run([checker, str(geom), str(order), "100000"], capture_output=True, text=True, check=True)
    lebesgue, points, bounded, below, negative, smooth, tight = (float(v) for v in out.stdout.split())
    # the roundings of a trace (the cut, then table, products and sums of one sum, or
    # of a hexahedron's three) stay below kTraceErr
    terms = 3 * (order + 2) if geom == 5 else 7
    assert lebesgue * (2.0 ** -23 + terms * 2.0 ** -24) < 6e-6
    assert below == 0 and negative == 0
    assert bounded > 0.8 * points  # it is of use
    assert smooth > 1000 and tight > 0.95 * smooth
