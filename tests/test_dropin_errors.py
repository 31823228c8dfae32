"""CPU test of the drop-in calls' error returns, with a CUDA runtime and a world of the test's own."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_failed_calls_leave_nothing_in_flight(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / "dropin_errors")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-fopenmp", "-I" + os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "cpp", "test_dropin_errors.cpp"), "-o", exe,
                    # the library's other parts are not called
                    "-no-pie", "-Wl,--unresolved-symbols=ignore-all"], check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
