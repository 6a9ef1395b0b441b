"""Offsets inside the engine's device allocations (csrc/host/arena.h), checked on the CPU: every
part on a boundary of its elements for odd image sizes and every pair of storage types, no more
bytes than the parts have when memory is short, and raw images only where there is room to spare."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "xpulse_recon_b200", "csrc", "host")
SOURCE = """
#include "arena.h"
using u64 = unsigned long;
extern "C" int resident(const u64 *bytes, u64 elem, u64 pixels, u64 raw, u64 limit, u64 margin, u64 avail, u64 *out)
{
    xpr::ResidentLayout l = xpr::resident_layout((const uint64_t *)bytes, elem, pixels, raw, limit, margin, avail);
    for (int k = 0; k < 6; ++k) out[k] = l.at[k];
    out[6] = l.raw;
    out[7] = l.total;
    return l.at_once;
}
extern "C" int staging(u64 pixels, u64 elem, u64 avail, u64 *out)
{
    return xpr::staging_layout(pixels, elem, avail, (uint64_t *)out);
}
"""
BIG = 1 << 40


@pytest.fixture(scope="module")
def arena(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("arena")
    (d / "a.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "a.cpp"), "-o", str(d / "a.so")],
                   check=True)
    return C.CDLL(str(d / "a.so"))


def staging(lib, pixels, elem, avail):
    out = (C.c_ulong * 6)()
    return lib.staging(C.c_ulong(pixels), C.c_ulong(elem), C.c_ulong(avail), out), list(out)


def check_parts(at, sizes, elems):
    for k, (n, e) in enumerate(zip(sizes, elems)):
        assert at[k] % e == 0 and at[k] + n <= at[k + 1]


@pytest.mark.parametrize("elem,ratio", [(4, 0), (4, 2), (2, 2), (2, 0)])  # images, ratio (0: the sums are the ratio)
@pytest.mark.parametrize("width,height,per,sit", [(3, 1, 1, 2), (5, 3, 1, 3), (37, 29, 7, 3), (64, 48, 6, 4)])
def test_resident_parts(arena, elem, ratio, width, height, per, sit):
    wh = width * height
    sizes = [4 * width * width * height, 4 * per * wh, 80 * sit * per, sit * per * wh * elem, per * wh * ratio]
    elems = [4, 4, 4, elem, 2]
    stage = 2 * wh * 4 + 8 + 2 * wh * elem
    raw = sit * per * wh * 4
    for avail in [sum(sizes) + k for k in range(0, 3 * 1280 + 2 * stage)] + [BIG]:
        out = (C.c_ulong * 8)()
        once = arena.resident((C.c_ulong * 5)(*sizes), C.c_ulong(elem), C.c_ulong(wh), C.c_ulong(raw), C.c_ulong(BIG),
                              C.c_ulong(64 << 20), C.c_ulong(avail), out)
        at, total = list(out)[:6], out[7]
        check_parts(at, sizes, elems)
        assert total <= avail
        if once:
            assert avail == BIG and out[6] % 256 == 0 and out[6] >= at[5] and total >= out[6] + raw + 8
        else:
            # what is left takes the two images in flight whenever the bare sums do
            left = avail - total
            if sum(sizes) + stage <= avail:
                padded, s = staging(arena, wh, elem, left)
                check_parts(s, [4 * wh, 4 * wh, 8, elem * wh, elem * wh], [4, 4, 4, elem, elem])
                assert s[5] <= left
    assert once


def test_raw_images_leave_a_margin(arena):
    sizes, wh = [4096, 1024, 80, 4096, 0], 256
    raw = 16 * wh * 4
    need = 4096 + 1024 + 256 + 4096 + raw + 8
    for avail, limit, expected in [(need + 1000, raw, 1), (need + 999, raw, 0), (need + 1000, raw - 1, 0), (BIG, raw, 1)]:
        out = (C.c_ulong * 8)()
        assert arena.resident((C.c_ulong * 5)(*sizes), C.c_ulong(4), C.c_ulong(wh), C.c_ulong(raw), C.c_ulong(limit),
                              C.c_ulong(1000), C.c_ulong(avail), out) == expected
    # images that do not lie together
    assert arena.resident((C.c_ulong * 5)(*sizes), C.c_ulong(4), C.c_ulong(wh), C.c_ulong(0), C.c_ulong(BIG),
                          C.c_ulong(0), C.c_ulong(BIG), out) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["naive", "method_1b"])
def test_a_cap_of_exactly_what_a_scan_takes(ctx, method):
    import json

    from xpulse_recon_b200 import _lib
    P, H, W, S = 24, 21, 33, 3
    raw = np.random.default_rng(2).uniform(0.05, 0.98, (P, H, W)).astype(np.float32)
    L = _lib.lib()
    L.xpr_reconstruct_host.argtypes = [C.c_char_p, C.c_void_p, C.c_int64, C.c_uint32, C.c_uint32, C.c_void_p,
                                       C.c_uint64, C.POINTER(C.c_double)]

    def run(cap):
        cfg = {"recon": {"method": method, "it": 1, "sit": S, "seed": 3, "mlog": True, "mem_cap": cap},
               "geometry": {"so": 100.0, "sd": 1000.0, "angle": 360.0}, "detector": {"px": 0.1}}
        out = np.empty((H, W, W), np.float32)
        return L.xpr_reconstruct_host(json.dumps(cfg).encode(), raw.ctypes.data, P, W, H, out.ctypes.data, out.size,
                                      None), out
    images, sums, pd, stage = P * H * W * 4, P // S * H * W * 4, 80 * P, 16 * H * W + 8
    need = (images + 4 * W * W * H if method == "naive" else P // S * H * W * 4) + sums + pd + stage
    rc, out = run(need)
    assert rc == 0, L.xpr_last_error()
    rc, exp = run(0)
    assert rc == 0
    np.testing.assert_array_equal(out.view(np.uint32), exp.view(np.uint32))
    assert run(need - 1)[0] != 0
