"""The streaming kernels' four-element accesses: remainders, buffers that are not aligned for
them, and values at the ends of the range, against the oracle bit for bit."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from tests.cases import assert_same_bits  # noqa: E402
from xpulse_recon_b200 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 1e-45, -1e-39, 1.1754944e-38, np.inf, -np.inf, np.nan, 3.4e38, -3.4e38, 1.0, -2.5e-7],
                   np.float32)


def stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def at(host, offset, dtype=torch.float32):
    """A device copy of `host` that starts `offset` elements into its buffer."""
    buf = torch.zeros(host.size + offset, dtype=dtype, device="cuda")
    buf[offset:] = torch.from_numpy(host).cuda().to(dtype)
    return buf[offset:]


@pytest.mark.parametrize("n,offset", [(1, 0), (3, 0), (4, 0), (7, 1), (1023, 0), (4099, 0), (4099, 1), (4100, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_error_remainders_and_offsets(ctx, n, offset, dtype):
    rng = np.random.default_rng(n + offset)
    img = rng.uniform(-0.1, 6.0, n).astype(np.float32)
    img[: SPECIAL.size] = SPECIAL[: img.size]
    sums = rng.integers(0, 2 ** 32, n, dtype=np.uint64).astype(np.uint32)
    sums[::5] = 0
    d_img, d_sum = at(img, offset, dtype), at(sums.view(np.int32), offset, torch.int32)
    out = at(np.zeros(n, np.float32), offset, dtype)
    exp = sums.copy()
    O.lib().orc_error(d_img.float().cpu().numpy(), exp, n, 0.9)
    code = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16}[dtype]
    _lib.check(_lib.lib().xpr_error(ctx.handle, d_img.data_ptr(), code, d_sum.data_ptr(), out.data_ptr(), code, n, 0.9,
                                    _lib.ERROR_STD, 1, None, stream()))
    assert_same_bits(out.float().cpu().numpy(), torch.from_numpy(exp.view(np.float32)).to(dtype).float().numpy())
    assert not d_sum.any()


@pytest.mark.parametrize("n,offset", [(1, 0), (5, 0), (8, 0), (4099, 0), (4099, 1), (70001, 3)])
@pytest.mark.parametrize("scale", [1.0, 6e4, 1e-30, 1e30])
def test_preprocess_remainders_and_offsets(ctx, n, offset, scale):
    rng = np.random.default_rng(n)
    raw = (rng.uniform(0.01, 1.0, n) * scale).astype(np.float32)
    raw[: SPECIAL.size:2] = SPECIAL[: raw.size:2]
    mn, mx = C.c_float(3.4028234663852886e38), C.c_float(-3.4028234663852886e38)
    O.lib().orc_minmax_normal(raw, n, C.byref(mn), C.byref(mx))
    d_raw = at(raw, offset)
    d_mm = torch.tensor([3.4028234663852886e38, -3.4028234663852886e38], device="cuda")
    L = _lib.lib()
    _lib.check(L.xpr_preprocess_minmax(ctx.handle, d_raw.data_ptr(), n, d_mm.data_ptr(), stream()))
    np.testing.assert_array_equal(d_mm.cpu().numpy(), np.array([mn.value, mx.value], np.float32))
    for normalize, mlog in ((1, 1), (1, 0), (0, 1)):
        exp = raw.copy()
        O.lib().orc_preprocess(exp, n, normalize, mn.value, mx.value, mlog)
        out = at(np.zeros(n, np.float32), offset)
        _lib.check(L.xpr_preprocess_apply(ctx.handle, d_raw.data_ptr(), out.data_ptr(), _lib.F32, n, normalize,
                                          d_mm.data_ptr(), mlog, stream()))
        assert_same_bits(out.cpu().numpy(), exp)
