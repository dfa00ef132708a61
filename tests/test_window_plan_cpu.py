"""Which 2D steps go out in windows (fdtd_b200/csrc/window_plan.h): the plans of
all kinds of grids and stretches are ones that the windows can take, and for
measured calls they choose the faster form (tests/cpp/window_plan_check.cu)."""
import os
import subprocess

from fdtd_b200.build_lib import NVCC

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_window_plans(tmp_path):
    exe = str(tmp_path / "window_plan_check")
    subprocess.run([NVCC, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "window_plan_check.cu")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "plans checked" in out.stdout
