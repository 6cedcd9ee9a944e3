"""The integer pair form's arithmetic (plum_gb300/csrc/fix_pair.h) on the CPU:
table sums of random pairs, one image and image cells, against long double, with
every index checked against the table. Systems: the 1,000- and 20,000-bead
workloads, the reference's Ewald rule at L = 40 and 50 (r_c = 28, 34), r_c = L,
weak and strong screening, a small box; and systems it must leave alone."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "plum_gb300", "csrc", "host", "real_tables.cc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fix") / "fix_pair_harness")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                        os.path.join(HERE, "fix_pair_harness.cc"), SRC], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("alpha,box,rc,mode", [
    (0.015625, 40.0, 20.0, 1), (0.0049, 80.0, 40.0, 1), (0.015625, 40.0, 28.0, 2),
    (0.01, 50.0, 34.0, 2), (0.0049, 80.0, 80.0, 2), (1e-5, 30.0, 15.0, 1), (1.0, 16.0, 8.0, 1),
    (0.3, 5.0, 3.0, 2), (0.01, 68.854, 34.427, 1), (0.04, 31.7, 9.2, 1), (0.04, 300.0, 10.0, 1),
    (0.015625, 40.0, 41.0, 0), (0.04, 400.0, 10.0, 0)])
def test_table_sums(harness, alpha, box, rc, mode):
    out = subprocess.run([harness, repr(alpha), repr(box), repr(rc), "40000", "5"],
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    got = out.stdout.split()
    assert int(got[0]) == mode, got
    if mode:
        assert int(got[1]) <= 1280
        assert float(got[4]) <= 1.0, got
