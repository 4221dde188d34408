"""The scene tracer's march, which evaluates no sample whose sign is certain, finds what
the march over every sample finds, on the host build of scene_gen.cuh."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_march_equals_every_sample(tmp_path):
    exe = str(tmp_path / "scene_march_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "native", "scene_march_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe, "200000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
