"""How a trace's rays are laid out over warps, on the host: the tuned number of
sub-rays per lane is the most a lane carries, and never keeps a trace whose
items are large enough from sharing one walk of the tree."""
import os
import subprocess

from dvsrender4deepspace_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_tuned_rays_keep_shared_walks(tmp_path):
    lib = build.build()
    exe = str(tmp_path / "trace_shapes_selftest")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-I", build.CSRC, "-I",
                    os.path.join(build.ROOT, "include"), "-I", os.path.join(cuda, "include"),
                    os.path.join(HERE, "trace_shapes_selftest.cpp"), lib, "-Wl,-rpath," + os.path.dirname(lib), "-o", exe],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = dict(line.split() for line in out.splitlines())
    assert int(rows["broken"]) == 0
    assert int(rows["beams"]) > 1000 and int(rows["traces"]) > 8 * int(rows["beams"])
