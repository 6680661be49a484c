"""Which way a caller's pointer goes (own device, another device, managed, pinned,
pageable memory), decided on faked pointer attributes: a kernel must not be given
another GPU's memory, and that can only be seen without one."""
import os
import subprocess

from conftest import ROOT


def test_routes(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = tmp_path / "routes"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "openpfc_b200", "csrc"), "-I",
                    os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "cpp", "test_user_buffer.cpp"), "-o",
                    str(exe), "-L", os.path.join(cuda, "lib64"), "-lcudart_static", "-ldl", "-lpthread", "-lrt"],
                   check=True, capture_output=True, text=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, p.stdout
