"""The library's code depends on its source and flags alone.

nvcc's -split-compile cuts a module into parts whose number, and with it register allocation, instruction order and
rounding, follows the cores that the building machine has: two machines would build libraries that differ in bits
and by several percent in time.  So neither nvcc nor the steps it runs (its dry run lists them) may be given it.
"""
import subprocess

from ding_nsch_core_solver_b200 import build


def test_no_build_step_splits_by_the_number_of_cores():
    cmd = [build.NVCC, "--dryrun"] + build.FLAGS + ["-c", "dn_capi.cu", "-o", "dn_capi.o"]
    steps = subprocess.run(cmd, capture_output=True, text=True, check=True)
    text = steps.stdout + steps.stderr
    assert "ptxas" in text and "cicc" in text
    assert "split-compile" not in text
