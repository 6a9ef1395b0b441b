"""Results above 8 MB into memory that was never touched, starting and ending inside a page: the
same volume as into memory in use, and nothing around it written."""
import ctypes as C
import json
import mmap

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from xpulse_recon_b200 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 1023])  # floats into the first page
def test_result_into_untouched_memory(offset):
    P, H, W = 12, 133, 134  # 9.6 MB
    raw = np.random.default_rng(4).uniform(0.05, 0.98, (P, H, W)).astype(np.float32)
    cfg = json.dumps({"recon": {"method": "naive", "it": 1, "sit": 2, "seed": 3, "mlog": True},
                      "geometry": {"so": 100.0, "sd": 1000.0, "angle": 360.0}, "detector": {"px": 0.1}}).encode()
    L = _lib.lib()
    L.xpr_reconstruct_host.argtypes = [C.c_char_p, C.c_void_p, C.c_int64, C.c_uint32, C.c_uint32, C.c_void_p,
                                       C.c_uint64, C.POINTER(C.c_double)]
    n = H * W * W
    used = np.full(n, 7.0, np.float32)
    _lib.check(L.xpr_reconstruct_host(cfg, raw.ctypes.data, P, W, H, used.ctypes.data, n, None), "run")
    fresh = np.frombuffer(mmap.mmap(-1, 4 * (n + 2048)), np.float32)
    _lib.check(L.xpr_reconstruct_host(cfg, raw.ctypes.data, P, W, H, fresh.ctypes.data + 4 * offset, n, None), "run")
    np.testing.assert_array_equal(fresh[offset:offset + n].view(np.uint32), used.view(np.uint32))
    assert not fresh[:offset].any() and not fresh[offset + n:].any()
