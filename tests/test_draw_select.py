"""The selection that avoids the division (lcg_select) equals the comparison with the
quotient, on the host build of vlt_math.cuh."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_draw_select_equals_division(tmp_path):
    exe = str(tmp_path / "draw_select_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "native", "draw_select_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe, "200000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
