"""How the kernels deal their work (csrc/splits.h), compiled with g++ alone and checked over whole ranges of sizes."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_work_split_cases(tmp_path):
    exe = str(tmp_path / "work_splits_test")
    cc = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-fsanitize=undefined", "-fno-sanitize-recover",
                         "-I", os.path.join(ROOT, "crucible_strix_halo_b200", "csrc"), os.path.join(ROOT, "tests", "work_splits_test.cpp"), "-o", exe],
                        capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout + run.stderr
