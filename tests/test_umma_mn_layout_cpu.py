"""The transposed operand stages of the tcgen05 GEMM: layout and descriptors (host build of the header)."""
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_transposed_operand_layout(tmp_path):
    exe = str(tmp_path / "mn")
    inc = os.path.join(os.path.dirname(HERE), "elanfmt_gb300", "csrc")
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-O1", "-I", inc, os.path.join(HERE, "umma_mn_check.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout.strip() == "ok"
