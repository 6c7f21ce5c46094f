"""The bounded waits of the flow kernels, host side: csrc/flow_wait.h compiled by g++ and run for every CTA size."""
import subprocess

from shim_build import PKG, ROOT


def _program(tmp_path, source):
    exe = tmp_path / "prog"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-I", str(PKG / "csrc"),
                        str(ROOT / "tests" / "cpp" / source), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


def test_wait_words_are_written_whatever_the_ctas_size(tmp_path):
    """A 4-atom lattice of up to 32 cells runs 32 threads: the word that ends a run must be cleared there too (it was
    cleared by thread 32).  And a row's wait has room for every wait of the steps before it, for any save interval."""
    r = subprocess.run([str(_program(tmp_path, "flow_wait_words.cpp"))], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
