"""The tcgen05 GEMM's waits, host builds of the header that the kernel uses (ewf_umma.h):
  * umma_warp_wait.cpp: a bounded wait has one answer for all lanes of a warp;
  * umma_ring_sim.cpp: the ring of stages and the accumulators between the producers, the MMA issuer and the epilogue's
    warps under random interleavings -- no deadlock, nothing refilled, overwritten or read too early."""
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "elanfmt_gb300", "csrc")


def _run(tmp_path, name):
    exe = str(tmp_path / name)
    subprocess.run([shutil.which("g++") or "c++", "-O2", "-std=c++20", "-pthread", "-I", CSRC, os.path.join(HERE, name + ".cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr


def test_a_wait_has_one_answer_per_warp(tmp_path):
    _run(tmp_path, "umma_warp_wait")


def test_ring_protocol(tmp_path):
    _run(tmp_path, "umma_ring_sim")
