"""The quotient and reciprocal forms the kernels call (mfg_quot.cuh), compiled
for the host from the same file: the division's bits inside their windows, the
ends of the windows where they are said to be, nothing taken outside them."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "minifs_b200", "csrc")


def build(exe, include):
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(include),
                    "-o", str(exe), os.path.join(HERE, "quotient_check.cpp"), "-lm"], check=True)


def counts(exe, n, seed):
    out = subprocess.run([str(exe), str(n), str(seed)], check=True, capture_output=True, text=True)
    return [int(v) for v in out.stdout.split()]


@pytest.mark.parametrize("seed", [5, 77])
def test_live_forms_against_the_division(tmp_path, seed):
    build(tmp_path / "check", CSRC)
    assert counts(tmp_path / "check", 10_000_000, seed) == [0, 0, 0]


@pytest.mark.parametrize("right, wrong", [
    ("outside_exp(a, 523, 1523)", "outside_exp(a, 523, 1524)"),
    ("outside_exp(a, 523, 1523)", "outside_exp(a, 522, 1523)"),
    ("(hi_mag(a) | __double2loint(a)) == 0", "hi_mag(a) == 0"),
    ("0x80000000;", "0;"),
    ("outside_exp(b, 523, 1523)", "outside_exp(b, 523, 1524)"),
    ("ones == -1 ? -1 : 0", "ones == -2 ? -1 : 0"),
    ("const double q = __fma_rn(r1, y, q1);", "const double q = q0;"),
    ("return __fma_rn(near, r, near);", "return near;"),
], ids=["top", "bottom", "zero", "sign", "divisor", "ones", "quotient", "reciprocal"])
def test_check_sees_a_planted_mistake(tmp_path, right, wrong):
    """In a copy on the host only."""
    with open(os.path.join(CSRC, "mfg_quot.cuh")) as f:
        text = f.read()
    assert text.count(right) == 1
    (tmp_path / "mfg_quot.cuh").write_text(text.replace(right, wrong))
    build(tmp_path / "check", tmp_path)
    assert any(counts(tmp_path / "check", 1_000_000, 5))
