"""The kernel launcher reports a refused launch itself (tests/cpp/launch_status.cu):
a status that is only read at the end of a call could be lost to a query in
between.  Needs no GPU: the launch is refused either way, on the host."""
import os
import subprocess

from conftest import ROOT
from open_quadtree_mapping_b200 import build_ext


def test_refused_launch_throws(tmp_path):
    build_ext.build()
    exe = str(tmp_path / "launch_status")
    subprocess.run([build_ext.nvcc(), *build_ext.ARCH, "-std=c++17", "-I", build_ext.CSRC,
                    "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "launch_status.cu"),
                    "-L", build_ext.OUT_DIR, "-lqm_b200",
                    "-Xlinker", "-rpath=" + build_ext.OUT_DIR, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 3, r.stdout + r.stderr
    assert "kernel launch" in r.stdout
