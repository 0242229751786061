"""The team kernels' pivot search and dense elimination on matrices with NaN (of either
sign) and infinite entries, the kernels' own source run on the CPU (tests/warp_emu): a row
that was a pivot row is never found again, so the elimination's second half has its eight
rows and nothing is stored outside the matrix."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "finite_root_generation_gb300", "csrc")


def test_nonfinite_pivots_stay_in_bounds(tmp_path):
    emu = os.path.join(HERE, "warp_emu")
    exe = str(tmp_path / "team_lu")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", f"-I{emu}", f"-I{CSRC}", os.path.join(emu, "team_lu.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
