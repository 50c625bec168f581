"""The shared memory of adaptive_block_kernel: a row's arrays fit what its pass allocates, whatever
the pass's widest detector is (tests/adapt_layout_check.cpp compiled here with g++)."""
import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_every_row_fits_its_pass(tmp_path):
    out = tmp_path / "adapt_layout_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG_DIR, "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "adapt_layout_check.cpp"), "-o", str(out)], check=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, check=True).stdout.split()
    r = dict(zip(r[0::2], map(int, r[1::2])))
    assert r["cases"] > 8_000_000 and r["outside"] == r["empty"] == r["shorter"] == 0, r
