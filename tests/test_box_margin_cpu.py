"""CPU: the float arithmetic's walk enters the box of every triangle that can win.

tests/box_margin_check.c restates a triangle's oriented box, the reference's float distance and the box
distance, and asks the threshold the kernels compile (csrc/box_margin.h) whether the box is entered while
the triangle's own float distance is the best. The derived need is at most 5.2 u c (u = 2^-24, c the
mesh's largest coordinate); the threshold allows 8.
"""

import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ssdf_b200", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("box") / "box_margin_check")
    res = subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-I", CSRC, "-o", exe,
                          os.path.join(HERE, "box_margin_check.c"), "-lm"], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return exe


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_every_winning_box_is_entered(checker, seed):
    out = subprocess.run([checker, "1000000", str(seed)], capture_output=True, text=True, check=True).stdout.split()
    vals = dict(zip(out[0::2], out[1::2]))
    assert int(vals["cases"]) > 900000
    assert int(vals["left_out"]) == 0, vals
    # below the derived bound, and not vacuous
    assert 1.5 < float(vals["largest_need"]) < 5.2, vals
