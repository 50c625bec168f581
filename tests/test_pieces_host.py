"""The certified pieces (csrc/cpd_piece.h) against the FP32 fast path, on the host
(tests/piece_check.cpp compiled here with g++): every ray that a piece decides has the
fast path's own outcome, bin, transmittance and no flag, and few rays are left to it."""
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, ROOT
from compound_prism_designer import precision as P
from compound_prism_designer import synth


@pytest.fixture(scope="module")
def piece_bin(tmp_path_factory):
    out = tmp_path_factory.mktemp("piece") / "piece_check"
    csrc = os.path.join(PKG_DIR, "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I", csrc, "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "piece_check.cpp"),
                    os.path.join(csrc, "cpd_host.cpp"), "-o", str(out)], check=True)
    return out


def _run(piece_bin, tmp_path, design, W, R, seed):
    dp, lp, rp = tmp_path / "d.bin", tmp_path / "l.bin", tmp_path / "r.bin"
    dp.write_bytes(bytes(design))
    P.synth_points(seed, W).tofile(lp)
    P.synth_points(seed, R, first=1).tofile(rp)
    out = subprocess.run([str(piece_bin), str(dp), str(W), str(R), str(lp), str(rp)], capture_output=True, text=True,
                         check=True).stdout.split()
    return dict(zip(out[0::2], map(int, out[1::2])))


# the optimizer's ranges; steep faces (total internal reflection, oblique detectors); wide beams (aperture losses);
# strong curvature; a very wide or very fine detector
KINDS = {"plain": ({}, (16, 64, 128)), "steep": ({"angle_range": (0.5, 1.3)}, (32, 128)),
         "wide_beam": ({"beam_width": 6.0}, (64, 500)), "curved": ({"curvature": 0.5}, (8, 33)),
         "thin": ({"height": 6.0}, (64,)), "bins": ({}, (1, 3, 1024))}


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("W,R", [(40, 1024), (16, 8191), (60, 129), (30, 31), (20, 1)])
def test_decided_rays_are_the_fast_paths(piece_bin, tmp_path, kind, W, R):
    kw, bins = KINDS[kind]
    rng = np.random.default_rng([len(kind), R])
    rays = decided = 0
    for B in bins:
        spec, _, _ = synth.random_design(rng, int(rng.integers(2, 7)), B, max_tries=50000, **kw)
        r = _run(piece_bin, tmp_path, spec.design, W, R, float(rng.uniform()))
        assert r["wrong"] == 0, (B, r)
        rays += r["rays"]
        decided += r["decided"]
    if kind == "plain" and R >= 1024:
        assert decided > 0.8 * rays  # else the pieces are of no use


def test_uncoated_design_is_left_to_the_fast_path(piece_bin, tmp_path):
    spec, _, _ = synth.random_design(np.random.default_rng(3), 3, 64, ar_coated=False)
    r = _run(piece_bin, tmp_path, spec.design, 20, 500, 0.2)
    assert r["rays"] > 0 and r["decided"] == 0, r
