"""The four-phonon kernels' shared-memory sizes on the host: no class count, however
large, comes back as a size that fits."""
import os
import subprocess

from fourphonon_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_size_wraps(tmp_path):
    exe = str(tmp_path / "layout_check")
    lib = build.build()
    subprocess.run([build.NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-ccbin", "/usr/bin/g++", os.path.join(HERE, "cuda", "layout_check.cu"), lib, "-Xlinker",
                    "-rpath," + os.path.dirname(lib), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
