"""Every plan of the tcgen05 convolution (lines per unit, pipeline stages)
against a plain convolution, bit for bit on integer values whose sums FP32
holds exactly (tests/native/conv_lines_check.cu).

The sizes are the ones where eight tiles a unit are taken: levels of 112 and
120 cells, whose tiles run across line ends, and 128-cell segments, one and two
a line; and levels of 64, 56 and 24 cells, which take at most five. 48 output
channels leave no room for eight in tensor memory."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path_factory.mktemp("conv") / "conv_lines_check")
    csrc = os.path.join(ROOT, "flip3d_gb300", "csrc")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17",
                           "--expt-relaxed-constexpr", "-I", csrc, "-I",
                           os.path.join(ROOT, "include"), "-o", exe,
                           os.path.join(ROOT, "tests", "native", "conv_lines_check.cu"),
                           os.path.join(csrc, "autotune.cu")])
    return exe


@pytest.mark.parametrize("n,cin,cout,batch,eight", [
    (112, 16, 16, 1, True), (112, 48, 16, 1, True), (112, 16, 32, 2, True),
    (120, 16, 16, 1, True), (120, 32, 32, 1, True), (128, 16, 16, 1, True),
    (128, 48, 16, 1, True), (256, 16, 16, 1, True), (64, 32, 32, 1, True),
    (56, 80, 32, 2, True), (24, 16, 48, 3, True), (112, 16, 48, 1, False)])
def test_every_plan_is_the_plain_convolution(check, n, cin, cout, batch, eight):
    out = subprocess.run([check, str(n), str(cin), str(cout), str(batch)], text=True,
                         capture_output=True, timeout=120)
    assert out.returncode == 0, (out.returncode, out.stderr)
    w = out.stdout.split()
    got = dict(zip(w[::2], map(int, w[1::2])))
    assert got["plans"] >= 3 and got["bad"] == 0 and got["err"] == 0, got
    assert (got["eight"] > 0) == eight, got
