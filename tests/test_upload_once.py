"""Tables uploaded on first use (csrc/cmd_internal.h), over a fake CUDA runtime: a failed copy is not taken for done."""
import subprocess
from pathlib import Path

from classical_mcmc_spin_b200 import build
from shim_build import PKG, ROOT


def test_a_table_whose_copy_failed_is_uploaded_again(tmp_path):
    exe = tmp_path / "prog"
    cuda = Path(build.nvcc()).resolve().parents[1] / "include"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(cuda), "-I", str(ROOT / "include"), "-I", str(PKG / "csrc"),
                        str(ROOT / "tests" / "cpp" / "upload_once.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
