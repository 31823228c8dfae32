"""CPU test of the sort scratch's size, through an allocator of the test's own."""
import os
import subprocess

import ae_mpm as M

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_scratch_holds_what_the_radix_sort_uses(tmp_path):
    lib = os.path.dirname(M.LIB_PATH)
    exe = str(tmp_path / "sort_scratch")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),
                    os.path.join(ROOT, "tests", "cpp", "test_sort_scratch.cpp"), "-o", exe, "-L" + lib, "-lae_mpm",
                    "-Wl,-rpath," + lib], check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
