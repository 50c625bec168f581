"""The kept orders of the point sequence (csrc/cpd_orders.h, compiled here with g++ in
tests/orders_check.cpp): complete on the device before a pass is given one, and the ascending order
of any seed's points. And no upload that a pass's stream does not wait for: the slots' streams do
not wait for the legacy stream, where a plain cudaMemcpy from pageable memory may still be running
when it returns."""
import os
import re
import subprocess

import pytest

from conftest import PKG_DIR, ROOT

CSRC = os.path.join(PKG_DIR, "csrc")


@pytest.fixture(scope="module")
def orders_bin(tmp_path_factory):
    out = tmp_path_factory.mktemp("orders") / "orders_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I", CSRC, "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "orders_check.cpp"), "-o", str(out)],
                   check=True)
    return str(out)


def _run(*args):
    r = subprocess.run([str(a) for a in args], capture_output=True, text=True, check=True).stdout.split()
    return dict(zip(r[0::2], map(int, r[1::2])))


def test_an_order_is_on_the_device_before_it_is_given_out(orders_bin):
    r = _run(orders_bin, "early", 1, 2, 31, 1024, 8192, 16384)
    assert r == {"given": 12, "early": 0, "left": 0}


@pytest.mark.parametrize("n", [0, 1, 63, 64, 65, 500])
def test_sizes_seen_once_do_not_keep_a_steady_size_out(orders_bin, n):
    assert _run(orders_bin, "steady", n) == {"given": 2, "kept": 64}


@pytest.mark.parametrize("R", [1, 2, 33, 1000, 16384])
def test_orders_sort_the_points_of_any_seed(orders_bin, R):
    seeds = [0.0, 0.5, 1e-17, 2.0 ** -53, 0.1234567, 0.381966, 0.9, 1.0 - 2.0 ** -53]
    r = _run(orders_bin, "sorted", R, *(repr(s) for s in seeds))
    assert r == {"points": R * len(seeds), "misplaced": 0}


@pytest.mark.parametrize("name", ["cpd_runtime.cu", "cpd_loop.cu"])
def test_uploads_are_on_the_streams_that_read_them(name):
    with open(os.path.join(CSRC, name)) as f:
        calls = re.findall(r"cudaMemcpy\((?:[^;]*?)\bcudaMemcpy(\w+To\w+)\)", f.read())
    assert "HostToDevice" not in calls, calls
