"""Division by a tabled reciprocal (x::div_by) rounds as a division does for every count that the
ray tables allow (tests/divby_check.cpp compiled here with g++)."""
import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_rounds_as_a_division(tmp_path):
    out = tmp_path / "divby_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I", os.path.join(PKG_DIR, "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "divby_check.cpp"), "-o", str(out)],
                   check=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, check=True).stdout.split()
    r = dict(zip(r[0::2], map(int, r[1::2])))
    assert r["cases"] > 30_000_000 and r["wrong"] == 0 and r["far"] > 0, r
