"""The FP32 screen of the SEM test for hits of one transmittance (sem_quick_equal) never decides
differently from the 128-bit test (tests/semequal_check.cpp compiled here with g++)."""
import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_screen_agrees_with_the_exact_test(tmp_path):
    out = tmp_path / "semequal_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I", os.path.join(PKG_DIR, "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "semequal_check.cpp"), "-o", str(out)],
                   check=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, check=True).stdout.split()
    r = dict(zip(r[0::2], map(int, r[1::2])))
    assert r["cases"] > 400000 and r["disagree"] == 0 and r["open"] < 0.01 * r["cases"], r
