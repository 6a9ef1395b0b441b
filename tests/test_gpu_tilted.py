"""Units that walk tilted projections: the switch from the untilted pass (also when the first
tilted projection comes after the first chunk of 32), the filtered pixel rule inside and at the
viewport's edges, footprints beyond a tile, and projections the rule does not take."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from tests.cases import assert_same_bits  # noqa: E402
from xpulse_recon_b200.projector import Reconstruction, geometry  # noqa: E402

pytestmark = pytest.mark.gpu

SCANS = {  # geometry, largest tilt (degrees), entries left untilted in front
    "three modules": (dict(dwidth=96, dheight=40, projections=14, module_number=3), 2.0, 0),
    "late": (dict(dwidth=72, dheight=37, projections=25, module_number=2), 1.5, 40),
    "ragged": (dict(dwidth=61, dheight=35, projections=9, module_number=2, rx=-0.7), 1.0, 0),
    "strong": (dict(dwidth=64, dheight=48, projections=7, so=20.0, sd=60.0, module_number=2), 30.0, 0),
    "one module": (dict(dwidth=48, dheight=32, projections=8), 2.0, 3),
    "wide": (dict(dwidth=80, dheight=48, projections=6, so=2.0, sd=4.0, module_number=2), 3.0, 0),
}


@pytest.mark.parametrize("arith", [O.STRICT, O.FAST])
@pytest.mark.parametrize("name", sorted(SCANS))
def test_tilted_forward_and_backward_match_the_oracle(ctx, name, arith):
    g, tilt, plain = SCANS[name]
    g = dict(dict(so=100.0, sd=1000.0, px=0.1, sit=1), **g)
    M = g.get("module_number", 1)
    rng = np.random.default_rng(17)
    rpy = rng.uniform(-tilt, tilt, (M, 3)).astype(np.float32)
    pd, out = geometry(mod_rpy=rpy.ravel(), **g)
    if plain:
        pd[:plain] = geometry(**g)[0][:plain]
    W, H, P = out["vwidth"], out["vheight"], g["projections"]
    origin = [float(np.float32(out["orig"][i]) + np.float32(0.4 * out["vx"])) for i in range(3)]
    vol = rng.uniform(0.0, 2.0, W * H * W).astype(np.float32)
    ratio = rng.uniform(-0.2, 0.2, P * g["dheight"] * g["dwidth"]).astype(np.float32)
    L, keep = O.make_launch((0, 0, 0), (W, H, W), origin, [out["vx"]] * 3, g["dwidth"], g["dheight"], 0, P, M, arith=arith)
    sums = np.zeros(ratio.size, np.uint32)
    O.forward(vol, sums, pd, L)
    back = vol.copy()
    O.backward(back, ratio, pd, L)

    r = Reconstruction(ctx, arith=arith)
    r.set_image_parameters(g["dwidth"], g["dheight"], P)
    r.set_volume_parameters((0, 0, 0), (W, H, W), [out["vx"]] * 3)
    r.set_angle_number(P, M)
    r.set_origin(origin)
    r.set_projdata_buffer(torch.from_numpy(pd).cuda())
    d_vol, d_sum = torch.from_numpy(vol).cuda(), torch.zeros(ratio.size, dtype=torch.int32, device="cuda")
    r.set_volume_buffer(d_vol)
    r.set_sum_images_buffer(d_sum)
    r.forward()
    np.testing.assert_array_equal(d_sum.cpu().numpy().view(np.uint32), sums)
    r.set_ratio_buffer(torch.from_numpy(ratio).cuda())
    r.backward()
    assert_same_bits(d_vol.cpu().numpy(), back)
