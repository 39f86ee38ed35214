"""The limits of the lane-per-group fill, asked before a pair is prepared, are the
ones that its preparation applies (tests/cpp/lane_limits_demo.cu; CPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_lane_limits():
    from locarna_gb300.build import GENCODE, NVCC, OUT, _run, build_engine
    build_engine()
    exe = os.path.join(OUT, "lane_limits_demo")
    _run([NVCC, GENCODE, "-std=c++17", "-O2", os.path.join(ROOT, "tests", "cpp", "lane_limits_demo.cu"), "-o", exe,
          "-L", OUT, "-llocarna_gb300", "-Xlinker", "-rpath=" + OUT])
    r = subprocess.run([exe], capture_output=True, text=True, check=True)
    assert r.stdout == "ok\n", r.stdout
