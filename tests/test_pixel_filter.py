"""The filtered pixel rule's error bound, checked on the CPU.

tests/pixel_filter_check.cpp compiles the bound the kernels use (csrc/xpr_pixel.cuh) and restates
the kernel's single-precision window coordinates (the hardware reciprocal anywhere within its
documented error): every voxel that the rule decides must get the contract's pixel.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

from xpulse_recon_b200.projector import geometry

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "xpulse_recon_b200", "csrc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("pf") / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-I", CSRC,
                    os.path.join(HERE, "pixel_filter_check.cpp"), "-o", exe], check=True)
    return exe


CASES = {  # geometry, brick, row offset and rows (0: the whole detector), least share decided by the rule
    "untilted": (dict(dwidth=192, dheight=192, projections=18), (32, 16, 8), 0, 0, 0.999),
    "modules": (dict(dwidth=384, dheight=384, projections=36, module_number=3, tilt=2.0), (32, 16, 32), 0, 0, 0.999),
    "large": (dict(dwidth=900, dheight=700, projections=20, module_number=3, tilt=2.0), (32, 16, 8), 0, 0, 0.998),
    "row window": (dict(dwidth=160, dheight=160, projections=24, module_number=2, tilt=1.0), (32, 8, 32), 40, 80, 0.999),
    "wide cone": (dict(dwidth=96, dheight=40, projections=24, so=2.0, sd=4.0, module_number=2, tilt=1.0), (32, 16, 8),
                  0, 0, 0.9),
    "strong tilt": (dict(dwidth=120, dheight=90, projections=24, so=20.0, sd=60.0, module_number=2, tilt=25.0),
                    (32, 16, 32), 0, 0, 0.9),
}


@pytest.mark.parametrize("strict", [1, 0])
@pytest.mark.parametrize("name", sorted(CASES))
def test_decided_pixels_are_the_contracts(check, name, strict):
    g, brick, off, rows, share = CASES[name]
    g = dict(dict(so=100.0, sd=1000.0, px=0.1, rx=0.4, sy=0.7, sit=1), **g)
    tilt = g.pop("tilt", 0.0)
    if tilt:
        rpy = np.random.default_rng(3).uniform(-tilt, tilt, (g["module_number"], 3))
        g["mod_rpy"] = rpy.astype(np.float32).ravel()
    pd, out = geometry(**g)
    origin = [out["orig"][i] + 0.37 * out["vx"] for i in range(3)]
    args = [out["vwidth"], out["vheight"], len(pd), *brick, off, rows or g["dheight"], "%.9g" % out["vx"],
            *("%.9g" % o for o in origin), strict, 150]
    text = "\n".join(" ".join("%.9g" % x for x in r) for r in pd)
    p = subprocess.run([check, *map(str, args)], input=text, capture_output=True, text=True)
    bricks, pairs, decided, wrong = (int(x) for x in p.stdout.split()[:4])
    assert p.returncode == 0 and wrong == 0
    assert bricks > 0 and decided >= share * pairs
