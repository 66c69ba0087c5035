"""Look-back words of the digit passes: compiles and runs tests/cpp/sort_words.cu
on the host."""
import subprocess
from pathlib import Path

from gpma_bfs_gb300.build import ARCH, CSRC, INCLUDE, _nvcc

ROOT = Path(__file__).resolve().parent.parent


def test_counts_of_the_largest_launches(tmp_path):
    exe = tmp_path / "sort_words"
    subprocess.run([_nvcc(), *ARCH, "-std=c++17", "-O2", "--expt-relaxed-constexpr", f"-I{CSRC}", f"-I{INCLUDE}",
                    str(ROOT / "tests/cpp/sort_words.cu"), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
