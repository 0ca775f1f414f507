"""The solver's FP32 evaluations of the reference's double expressions
(flip3d_gb300/csrc/refmath.h stencil_ref, ghost_ref, scale2_ref) against the
expressions themselves, bit for bit, on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_solver_expressions(tmp_path):
    exe = tmp_path / "refmath_solver_check"
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-o", str(exe),
                           os.path.join(ROOT, "tests", "native", "refmath_solver_check.cpp")])
    out = subprocess.check_output([str(exe), "400000"], text=True).split()
    assert out[1] == out[3] == out[5] == "0", out
