"""Memory of another GPU is copied, not accessed by kernels (the predicate alone:
compiles and runs tests/cpp/memory_place.cu on the host)."""
import subprocess
from pathlib import Path

from gpma_bfs_gb300.build import ARCH, CSRC, INCLUDE, _nvcc

ROOT = Path(__file__).resolve().parent.parent


def test_only_this_device_is_used_in_place(tmp_path):
    exe = tmp_path / "memory_place"
    subprocess.run([_nvcc(), *ARCH, "-std=c++17", "-O2", "--expt-relaxed-constexpr", f"-I{CSRC}", f"-I{INCLUDE}",
                    str(ROOT / "tests/cpp/memory_place.cu"), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
