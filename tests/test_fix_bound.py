"""The integer pair form's table sums (plum_gb300/csrc/fix_pair.h) stay inside the error
bound that tests/fix_bound_harness.cc derives term by term, over several seeds: the
workloads' systems, r_c = L, weak and very strong screening, a box of 32 r_c. The bound
is reached to between 0.3 and 1 of it, so a term that grew would show."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "plum_gb300", "csrc", "host", "real_tables.cc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fix") / "fix_bound_harness")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "fix_bound_harness.cc"), SRC], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("alpha,box,rc,mode", [
    (0.015625, 40.0, 20.0, 1), (0.0049, 80.0, 40.0, 1), (0.015625, 40.0, 28.0, 2),
    (0.01, 50.0, 34.0, 2), (0.0049, 80.0, 80.0, 2), (0.3, 5.0, 5.0, 2), (1e-4, 10.0, 10.0, 2),
    (1e-5, 30.0, 15.0, 1), (1e-9, 30.0, 15.0, 1), (1.0, 16.0, 8.0, 1), (4.0, 20.0, 10.0, 1),
    (100.0, 3.0, 1.5, 1), (0.04, 31.7, 9.2, 1), (0.01, 320.0, 10.0, 1)])
def test_error_bound(harness, alpha, box, rc, mode):
    out = subprocess.run([harness, repr(alpha), repr(box), repr(rc), "4000", "1", "10"],
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    got = out.stdout.split()
    assert int(got[0]) == mode and 0 < int(got[1]) <= 1280, got
    assert 0.3 <= float(got[4]) <= 1.0, got


@pytest.mark.parametrize("alpha,box,rc,most,far,far_rel", [
    (0.015625, 40.0, 20.0, 1.0e-15, 2.0e-16, 6e-13), (0.0049, 80.0, 40.0, 1.0e-15, 2.2e-16, 3e-12),
    (0.015625, 40.0, 28.0, 8e-15, 1.5e-16, 1e-10), (0.01, 50.0, 34.0, 8e-15, 1.5e-16, 1e-10)])
def test_stated_errors(harness, alpha, box, rc, most, far, far_rel):
    """The figures that the header states for the workloads."""
    out = subprocess.run([harness, repr(alpha), repr(box), repr(rc), "40000", "1", "5"],
                         capture_output=True, text=True, timeout=600)
    got = [float(x) for x in out.stdout.split()]
    assert got[3] <= most and got[5] <= far and got[6] <= far_rel, got
