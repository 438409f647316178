"""Kernels that need more shared memory than the default are opted in on every
device that a process uses, not only on its first."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hobakv1_gb300", "csrc")


def test_set_up_runs_once_on_each_device(tmp_path):
    exe = str(tmp_path / "once_per_device")
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, os.path.join(ROOT, "tests", "cpp", "once_per_device.cpp"),
                    "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout == "ok\n"


def test_every_opt_in_is_per_device():
    """CUDA keeps a function's attributes per device: where they are set, that is
    behind OncePerDevice and not behind a flag of the process."""
    n = 0
    for f in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, f)) as fh:
            text = fh.read()
        if "cudaFuncSetAttribute" in text:
            n += 1
            assert "OncePerDevice" in text, f
            assert not re.search(r"static std::atomic<\w+> done", text), f
    assert n == 3
