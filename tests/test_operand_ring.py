"""The schedule of the split GEMM's operand ring (sd3.c_b200/csrc/operand_ring.h), model-checked on the host:
operand_ring_model.cpp walks every interleaving of loads, their landing, MMA issue and completion."""
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sd3.c_b200", "csrc")


def test_operand_ring_schedule(tmp_path):
    exe = str(tmp_path / "model")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(HERE, "operand_ring_model.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_split_gemm_uses_a_checked_ring():
    """The kernel's barriers and phases come from OperandRing, with a stage count that the model covers."""
    src = open(os.path.join(CSRC, "gemm_split.cu")).read()
    stages = int(re.search(r"constexpr int STAGES = (\d+);", src).group(1))
    assert re.search(r"using Ring = OperandRing<STAGES, 2>;", src)
    assert "OperandRing<%d, 2>" % stages in open(os.path.join(HERE, "operand_ring_model.cpp")).read()
    assert "s < Ring::FULL_BARS; ++s) mbar_init(&full_bar[s], 1)" in src
    assert "mbar_wait(&full_bar[ring.full], ring.full_parity," in src
