"""CPU check: how many tiles the experts' rows of a prompt are taken to fill, and the cut of the columns that follows from it
(wayruntime_b200/csrc/gemm_plan.h, plain C++), against drawn routers."""
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_tiles_of_experts_and_the_cut_for_them():
    exe = os.path.join(tempfile.mkdtemp(prefix="wr_gpc_"), "gemm_plan_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "wayruntime_b200", "csrc"),
                    os.path.join(ROOT, "tests", "gemm_plan_check.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert res.returncode == 0, res.stdout
