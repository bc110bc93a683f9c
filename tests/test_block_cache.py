"""The cache of small device buffers when the host is out of memory (tests/cpp/block_cache.cu),
on the CPU."""
import os
import subprocess

from conftest import ROOT
from femgpu import build


def test_a_buffer_is_given_back_without_host_memory(tmp_path):
    exe = tmp_path / "block_cache"
    cmd = [build.nvcc_path()] + build.ARCH + ["-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, "-I",
                                              build.INCLUDE, "-o", str(exe)]
    cmd += [os.path.join(ROOT, "tests", "cpp", f) for f in ("block_cache.cu", "block_cache_new.cpp")]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stderr)
