"""The grid barrier where its counter starts over (long searches), on the
host: compiles and runs tests/cpp/barrier_wrap.cu."""
import subprocess
from pathlib import Path

from gpma_bfs_gb300.build import ARCH, CSRC, INCLUDE, _nvcc

ROOT = Path(__file__).resolve().parent.parent


def test_barrier_rounds_across_the_wrap(tmp_path):
    exe = tmp_path / "barrier_wrap"
    subprocess.run([_nvcc(), *ARCH, "-std=c++17", "-O2", "--expt-relaxed-constexpr", f"-I{CSRC}", f"-I{INCLUDE}",
                    str(ROOT / "tests/cpp/barrier_wrap.cu"), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
