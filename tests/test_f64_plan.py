"""The plain f64 plans (momms_gb300/csrc/f64_plan.h) on the CPU: what a split needs of scratch stays
within what its callers hold, for the model's plans and for tuned split counts; and the rounding
error of the order in which a plan sums is no larger than that of the 128 x 128 grid's."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "test_f64_plan.cpp")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("f64_plan") / "f64_plan")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "momms_gb300", "csrc"), SRC, "-o", out],
                   check=True, capture_output=True, text=True)
    return out


def test_split_plans_fit_the_scratch(exe):
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout


def test_sums_round_no_more_than_the_grids(exe):
    """Ratios of rms errors over 20,000 dot products: each is off by about 1 / sqrt(20000) = 0.7 %
    of itself, so four of that above 1 are allowed."""
    r = subprocess.run([exe, "rms"], capture_output=True, text=True, timeout=300, check=True)
    rows = [line.split() for line in r.stdout.split("\n") if line]
    assert len(rows) == 24
    assert all(float(x[3]) <= 1.03 for x in rows), r.stdout
