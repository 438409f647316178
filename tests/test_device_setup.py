"""Kernels that need more shared memory than the default are opted in on every
device that a process uses, not only on its first."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hobakv1_gb300", "csrc")


def runs(name, tmp_path):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, os.path.join(ROOT, "tests", "cpp", name + ".cpp"), "-o", exe],
                   check=True)
    return subprocess.run([exe], capture_output=True, text=True).stdout


def test_set_up_runs_once_on_each_device(tmp_path):
    assert runs("once_per_device", tmp_path) == "ok\n"


def test_kept_scratch_makes_room_for_a_batch(tmp_path):
    """The evaluation calls' pool keeps memory between calls; no allocation of a
    batch (precision, contact, rest Hessian, autotuner, inspection) fails for it."""
    assert runs("alloc_retry", tmp_path) == "ok\n"
    with open(os.path.join(CSRC, "api.cu")) as fh:
        text = fh.read()
    assert len(re.findall(r"[^a-z_]cudaMalloc\(", text)) == 1  # in batch_malloc


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
