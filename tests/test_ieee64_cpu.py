"""The branch-free quotients and square roots of the FP64 stage kernels
(csrc/ieee64.h) against the host's IEEE `/` and sqrt: equal on every operand
of tests/ieee64_check.cpp."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotients_and_roots_are_correctly_rounded(tmp_path):
    exe = str(tmp_path / "ieee64_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "tsuner_b200", "csrc"),
                    os.path.join(ROOT, "tests", "ieee64_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "400000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
