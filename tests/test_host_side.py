"""CPU tests of the C calls' host side, with a CUDA runtime and a world of the tests' own."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("name", ["dropin_errors", "batch_priorities"])
def test_host_side(tmp_path, name):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-fopenmp", "-I" + os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "cpp", "test_%s.cpp" % name), "-o", exe,
                    # the library's other parts are not called
                    "-no-pie", "-Wl,--unresolved-symbols=ignore-all"], check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
