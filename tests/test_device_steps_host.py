"""Steps of the device code that also compile for the host, run on the CPU
(tests/cpp/test_device_steps.cu): what a step may read once it has handed
memory on, and what it reads for inputs that break an order it relies on."""
import glob
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "test_device_steps.cu")
BIN = os.path.join(ROOT, "tests", "cpp", "_build", "test_device_steps")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def build_program() -> str:
    deps = [SRC] + glob.glob(os.path.join(ROOT, "include", "b2p_device", "*.cuh"))
    if os.path.exists(BIN) and os.path.getmtime(BIN) >= max(os.path.getmtime(p) for p in deps):
        return BIN
    os.makedirs(os.path.dirname(BIN), exist_ok=True)
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                        "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "include"), "-o", BIN, SRC],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return BIN


def test_device_steps():
    r = subprocess.run([build_program()], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ALL PASSED" in r.stdout, r.stdout + r.stderr
