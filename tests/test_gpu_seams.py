"""Modules whose viewport does not start on a 4-pixel column while the detector's width is a
multiple of 4 (the forward's bulk flush starts its tile rows on 16 bytes): a voxel left of the
viewport belongs to the neighbouring module's share of the sums only."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from tests.cases import assert_same_bits  # noqa: E402
from xpulse_recon_b200 import _lib  # noqa: E402
from xpulse_recon_b200.batch import Batch, Problem  # noqa: E402
from xpulse_recon_b200.projector import Reconstruction, geometry  # noqa: E402

pytestmark = pytest.mark.gpu

WIDTHS = [(44, 2), (100, 2), (84, 4)]  # modules of 22, 50 and 21 pixels


@pytest.mark.parametrize("arith", [O.STRICT, O.FAST])
@pytest.mark.parametrize("tilt", [0.0, 1.5])
@pytest.mark.parametrize("width,modules", WIDTHS)
def test_forward_sums_at_module_seams(ctx, width, modules, tilt, arith):
    g = dict(so=100.0, sd=1000.0, px=0.1, sit=1, dwidth=width, dheight=36, projections=9, module_number=modules)
    rng = np.random.default_rng(width)
    rpy = rng.uniform(-tilt, tilt, (modules, 3)).astype(np.float32).ravel() if tilt else None
    pd, out = geometry(mod_rpy=rpy, **g)
    W, H, P = out["vwidth"], out["vheight"], g["projections"]
    origin = [float(np.float32(out["orig"][i]) + np.float32(0.4 * out["vx"])) for i in range(3)]
    vol = rng.uniform(0.0, 2.0, W * H * W).astype(np.float32)
    L, keep = O.make_launch((0, 0, 0), (W, H, W), origin, [out["vx"]] * 3, width, 36, 0, P, modules, arith=arith)
    sums = np.zeros(P * 36 * width, np.uint32)
    O.forward(vol, sums, pd, L)
    r = Reconstruction(ctx, arith=arith)
    r.set_image_parameters(width, 36, P)
    r.set_volume_parameters((0, 0, 0), (W, H, W), [out["vx"]] * 3)
    r.set_angle_number(P, modules)
    r.set_origin(origin)
    r.set_projdata_buffer(torch.from_numpy(pd).cuda())
    d_vol, d_sum = torch.from_numpy(vol).cuda(), torch.zeros(sums.size, dtype=torch.int32, device="cuda")
    r.set_volume_buffer(d_vol)
    r.set_sum_images_buffer(d_sum)
    r.forward()
    np.testing.assert_array_equal(d_sum.cpu().numpy().view(np.uint32), sums)


@pytest.mark.parametrize("layers", [8, 16])
@pytest.mark.parametrize("width,modules", WIDTHS[:2])
def test_batched_forward_at_module_seams(ctx, width, modules, layers):
    raw = np.random.default_rng(width).uniform(0.05, 0.98, (12, 24, width)).astype(np.float32)
    p = Problem.from_raw(ctx, raw, dict(module_number=modules), 1, 3, seed=5)
    b = Batch(ctx, [p], arith=_lib.STRICT, use_graph=False, autotune=False, fwd_layers=layers)
    b.run()
    imgs = raw.ravel().copy()
    O.lib().orc_preprocess(imgs, imgs.size, 0, 0.0, 0.0, 1)
    gp = O.geom_params(dwidth=width, dheight=24, projections=12, sit=3, module_number=modules)
    rp = O.ReconParams(1, 3, 1.0, 0.9, 5, O.STRICT, 0)
    exp = np.zeros(p.vol.numel(), np.float32)
    assert O.lib().orc_recon_naive(C.byref(gp), C.byref(rp), imgs, exp) == 0
    assert_same_bits(p.vol.cpu().numpy(), exp)
    b.close()
