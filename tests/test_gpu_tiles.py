"""Brick footprints of every size against the oracle: forward tiles of the fixed pitch, wider ones
with a pitch of their own and bricks that go straight to the detector; windows that the filtered
pixel rule takes and ones too large for it; untilted projections among tilted ones."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from tests.cases import assert_same_bits  # noqa: E402
from xpulse_recon_b200.projector import Reconstruction, geometry  # noqa: E402

pytestmark = pytest.mark.gpu

MODULES = {"one": (1, 0.0), "two": (2, 0.0), "tilted": (2, 1.5), "last tilted": (2, 1.5)}  # number, tilt


@pytest.mark.parametrize("arith", [O.STRICT, O.FAST])
@pytest.mark.parametrize("modules", sorted(MODULES))
@pytest.mark.parametrize("voxel", [1.0, 1.3, 1.45, 1.7, 4.5])  # of the pixel at the axis
def test_footprints_of_every_size(ctx, voxel, modules, arith):
    M, tilt = MODULES[modules]
    g = dict(so=100.0, sd=1000.0, px=0.1, sit=1, dwidth=300, dheight=72, projections=19, module_number=M)
    rng = np.random.default_rng(7)
    rpy = rng.uniform(-tilt, tilt, (M, 3)).astype(np.float32) if tilt else None
    if modules == "last tilted":
        rpy[0] = 0.0
    pd, out = geometry(mod_rpy=None if rpy is None else rpy.ravel(), **g)
    W, H, P = int(out["vwidth"] / (2 * voxel)), int(out["vheight"] / voxel), g["projections"]
    vx = float(np.float32(out["vx"] * voxel))
    origin = [float(np.float32(-0.5 * n * vx + 0.3 * out["vx"])) for n in (W, H, W)]
    vol = rng.uniform(0.0, 2.0, W * H * W).astype(np.float32)
    ratio = rng.uniform(-0.2, 0.2, P * 72 * 300).astype(np.float32)
    L, keep = O.make_launch((0, 0, 0), (W, H, W), origin, [vx] * 3, 300, 72, 0, P, M, arith=arith)
    sums = np.zeros(ratio.size, np.uint32)
    O.forward(vol, sums, pd, L)
    back = vol.copy()
    O.backward(back, ratio, pd, L)

    r = Reconstruction(ctx, arith=arith)
    r.set_image_parameters(300, 72, P)
    r.set_volume_parameters((0, 0, 0), (W, H, W), [vx] * 3)
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


@pytest.mark.parametrize("arith", [O.STRICT, O.FAST])
@pytest.mark.parametrize("flat", [0, 1, 2])  # modules without tilt
def test_lists_and_row_windows_of_mixed_modules(ctx, flat, arith):
    """Index lists in any order, entries repeated, NaN ratios, a box and a row window, on three
    modules of which some are tilted."""
    from tests.cases import make_case, oracle_backward, oracle_forward
    from tests.test_gpu_parity import gpu_backward, gpu_forward
    c = make_case("modules3_rpy", sit=1, seed=3, row_window=(6, 20), box=((3, 2, 1), (58, 27, 60)))
    pd = c["pd_all"].reshape(-1, c["M"], 20)
    untilted = make_case("modules2", sit=1)["pd_all"].reshape(-1, 2, 20)
    for m in range(flat):  # an untilted module's matrix rows, this scan's viewports
        pd[:, m, :16] = untilted[np.arange(len(pd)) % len(untilted), 0, :16]
    rng = np.random.default_rng(flat)
    n, images = 70, 4
    lists = (rng.integers(0, len(pd) * c["M"], n).astype(np.uint16), rng.integers(0, images, n).astype(np.uint16))
    np.testing.assert_array_equal(gpu_forward(ctx, c, arith, lists=lists),
                                  oracle_forward(c, arith, lists=lists, pd=c["pd_all"]))
    n_img = max(int(lists[1].max()) + 1, c["Pc"])
    ratio = rng.uniform(-0.3, 0.3, n_img * c["Wd"] * c["rows"]).astype(np.float32)
    ratio[rng.random(ratio.size) < 0.05] = np.nan
    for skip in (0, 1):
        r = ratio if skip else np.nan_to_num(ratio)
        assert_same_bits(gpu_backward(ctx, c, r, arith, lists=lists, nan_skip=bool(skip)),
                         oracle_backward(c, r, arith, nan_skip=skip, lists=lists, pd=c["pd_all"]))
