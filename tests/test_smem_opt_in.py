"""Dynamic shared memory beyond 48 KB is opted in to per device: a process that
uses a second device must get it there too. The library's host code runs on two
devices of a fake CUDA runtime (tests/native/smem_opt_in_check.cpp), which
checks every launch."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_opt_in_on_every_device(tmp_path):
    from tdsez_gb300 import build
    build.build()
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    cuda_inc = None
    for cand in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda"):
        if cand and os.path.isfile(os.path.join(cand, "include", "cuda_runtime.h")):
            cuda_inc = os.path.join(cand, "include")
    if cuda_inc is None:
        pytest.skip("CUDA headers not found")
    cuda_lib = os.path.join(os.path.dirname(cuda_inc), "lib64")
    exe, pkg = str(tmp_path / "smem_opt_in_check"), os.path.join(ROOT, "tdsez_gb300")
    # -rdynamic: the program's runtime functions take the place of the library's
    subprocess.run([cxx, "-O1", "-std=c++17", "-rdynamic", "-I", os.path.join(ROOT, "include"), "-I", cuda_inc,
                    os.path.join(HERE, "native", "smem_opt_in_check.cpp"), "-o", exe, "-L", pkg, "-ltdz",
                    "-Wl,-rpath," + pkg, "-L", cuda_lib, "-lcudart", "-Wl,-rpath," + cuda_lib], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout[-2000:] + out.stderr[-500:]
    words = out.stdout.split()
    large, refused = int(words[words.index("large") + 1]), int(words[words.index("refused") + 1])
    assert large > 500 and refused == 0, out.stdout[-2000:]
