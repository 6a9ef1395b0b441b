"""What a program built on this package spends its time in, as cases that can be timed.

Each case is one call (or the few calls of one sub-iteration) through the public entry points:
the operator seam ``projector.Reconstruction``, the whole device-resident runs ``batch.Problem``
/ ``batch.Batch``, the preprocessing of the C ABI, and the whole call ``xpr_reconstruct_host``
on host data.  Sizes follow the package's own configurations (192^3 x 18 projections per
sub-iteration, 768^3 x 72, 3 tilted modules of 128 px, many 96 x 64 x 96 problems) and odd ones
between them.  Measured images are analytic line integrals of seeded spheres with 1 % noise, so
a sub-iteration works on consistent data; volumes are the same spheres, disturbed, over a faint
background, as an iterate looks after a few sub-iterations.
"""
from __future__ import annotations

import ctypes as C
import json
import math

import numpy as np
import torch

from xpulse_recon_b200 import _lib
from xpulse_recon_b200.batch import Batch, Problem, torch_dtype
from xpulse_recon_b200.projector import Context, Reconstruction, geometry

EPS = 1.0 / 4194304.0  # the smallest positive detector sum
STORAGE = {"fp32": _lib.F32, "bf16": _lib.BF16, "fp16": _lib.F16}
ARITH = {"strict": _lib.STRICT, "fast": _lib.FAST}
SPHERES = 6

_ctx = None


def _context() -> Context:
    """A program keeps one device context."""
    global _ctx
    if _ctx is None:
        _ctx = Context(torch.cuda.current_device())
    return _ctx


# what an operator case leaves out: a plain scan on one detector in the default contract
PLAIN = dict(dw=192, dh=192, proj=18, rx=0.0, sx=0.0, sy=0.0, modules=1, tilt=0.0, angle=360.0, arith="strict",
             ratio="fp32", images="fp32", layers=0, lists=False)


def _op(name, op, **kw):
    return dict(PLAIN, op=op, name=name, **kw)


def listed():
    return [
        # a whole call of the smallest scan, as the command line makes it: raw projections in host memory
        # in, the volume in host memory out (192^3 voxels, 180 projections, 10 sub-iterations)
        dict(name="reconstruct_192", op="reconstruct", dw=192, dh=192, proj=180, sit=10, it=1, modules=1, tilt=0.0,
             method="naive"),
        # the headline scan's forward: 768^3 voxels, 72 projections of 768 x 768
        _op("forward_768", "forward", dw=768, dh=768, proj=72, rx=1.5, sx=-2.0, sy=3.0),
        # and its backward
        _op("backward_768", "backward", dw=768, dh=768, proj=72, rx=1.5, sx=-2.0, sy=3.0),
        # a cropped detector: widths that are no multiple of 4, a short scan, an offset axis
        _op("forward_odd", "forward", dw=501, dh=387, proj=41, rx=-2.3, sy=1.5, angle=200.0),
        # the reduced storage form (FP16 ratio) on two abutted modules, odd sizes again
        _op("backward_f16", "backward", dw=454, dh=301, proj=45, modules=2, rx=0.7, ratio="fp16"),
        # a whole sub-iteration (forward, error, backward) of the smallest scan, where launch latency counts
        _op("sub_192", "sub"),
        # a multi-module detector with mounting errors (roll / pitch / yaw) in the default contract
        _op("sub_tilted", "sub", dw=384, dh=384, proj=36, modules=3, tilt=2.0),
        # the relaxed contract with BF16 images and ratio: the fastest form a user can ask for
        _op("sub_fast_bf16", "sub", dw=512, dh=480, proj=50, arith="fast", ratio="bf16", images="bf16", rx=1.5),
        # one slab of the out-of-core method that projects by index lists and skips NaN ratios
        _op("sub_slab_lists", "sub", dw=640, dh=512, proj=40, layers=48, lists=True),
        # many small scans on tilted modules in one batched run: 2 iterations of 10 sub-iterations
        dict(name="batch_small", op="batch", count=48, dw=96, dh=64, dw_max=96, proj=180, sit=10, it=2, modules=3,
             tilt=2.0, arith="fast", ratio="bf16", images="bf16"),
        # a mix of ordinary scans in the default contract, FP16 images as the request loop stores them
        dict(name="batch_mixed", op="batch", count=6, dw=96, dh=72, dw_max=252, proj=120, sit=6, it=1, modules=1,
             tilt=0.0, arith="strict", ratio="fp32", images="fp16"),
        # raw counts of a whole scan to attenuations: minimum and maximum, normalisation, -log
        dict(name="preprocess", op="preprocess", dw=768, dh=768, proj=240, normalize=True, images="fp32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["forward", "backward", "sub", "sub", "batch", "preprocess", "reconstruct"])
    if op == "preprocess":
        return dict(op=op, dw=_log_int(rng, 90, 800), dh=_log_int(rng, 60, 800), proj=_log_int(rng, 20, 200),
                    normalize=rng.random() < 0.6, images=rng.choice(["fp32", "fp32", "fp16", "bf16"]))
    if op == "reconstruct":
        return dict(op=op, dw=_log_int(rng, 60, 260), dh=_log_int(rng, 60, 200), proj=rng.randrange(60, 240),
                    sit=rng.randrange(4, 12), it=rng.choice([1, 2]), modules=1, tilt=0.0,
                    method=rng.choice(["naive", "method_1b", "method_1c", "method_2"]))
    if op == "batch":
        modules = rng.choice([1, 1, 3])
        dw = rng.randrange(48, 160)
        return dict(op=op, count=rng.randrange(2, 40), dw=dw, dh=rng.randrange(32, 120),
                    dw_max=min(200, dw + rng.randrange(0, 60)), proj=rng.randrange(60, 200), sit=rng.randrange(4, 12),
                    it=rng.choice([1, 2]), modules=modules, tilt=2.0 if modules > 1 else 0.0,
                    arith=rng.choice(["strict", "fast"]), ratio=rng.choice(["fp32", "bf16", "fp16"]),
                    images=rng.choice(["fp32", "bf16", "fp16"]))
    modules = rng.choice([1, 1, 1, 2, 3])
    c = dict(PLAIN, op=op, dw=_log_int(rng, 100, 700), dh=_log_int(rng, 80, 560), proj=rng.randrange(10, 70),
             rx=round(rng.uniform(-3, 3), 2), sx=round(rng.uniform(-2, 2), 2), sy=round(rng.uniform(-3, 3), 2),
             modules=modules, tilt=round(rng.uniform(0.2, 2.0), 2) if modules > 1 and rng.random() < 0.6 else 0.0,
             angle=rng.choice([360.0, 360.0, 200.0]), arith=rng.choice(["strict", "strict", "fast"]),
             ratio=rng.choice(["fp32", "fp32", "fp16", "bf16"]), images=rng.choice(["fp32", "fp32", "fp16", "bf16"]))
    if rng.random() < 0.25:
        c["layers"] = rng.randrange(7, c["dh"] // 2)
        c["lists"] = rng.random() < 0.5
    return c


# ------------------------------------------------------------------------------ inputs
def _spheres(seed):
    """(centre x, y, z, radius, attenuation) of a phantom in the unit cube [-1, 1]^3."""
    r = np.random.default_rng(seed)
    return [(*r.uniform(-0.45, 0.45, 3), r.uniform(0.08, 0.4), r.uniform(0.2, 1.0)) for _ in range(SPHERES)]


def _plan(c, seed):
    """The ProjData of one sub-iteration's angles, the grid and the origin a program keeps."""
    M = c["modules"]
    r = np.random.default_rng(seed + 17)
    rpy = r.uniform(-c["tilt"], c["tilt"], (M, 3)).astype(np.float32) if c["tilt"] else None
    pd, g = geometry(so=100.0, sd=1000.0, angle=c.get("angle", 360.0), px=0.1, rx=c.get("rx", 0.0),
                     sx=c.get("sx", 0.0), sy=c.get("sy", 0.0), module_number=M, dwidth=c["dw"], dheight=c["dh"],
                     projections=c["proj"], sit=1, mod_rpy=None if rpy is None else rpy.ravel())
    # the sub-voxel shift that a program draws for each sub-iteration
    origin = [float(np.float32(np.float32(g["orig"][i]) + np.float32(r.uniform(0, g["vx"])))) for i in range(3)]
    return pd, g, origin


def _scale(g):
    """Attenuation per mm of a unit sphere value: line integrals of about 1 through the object."""
    return 1.0 / (g["vwidth"] * g["vx"])


def _volume(g, seed, layers, gen):
    """The phantom on layers [y0, y1) of the grid, disturbed, over a faint background; flat (y, z, x)."""
    y0, y1 = layers
    W, H = g["vwidth"], g["vheight"]
    ax = (torch.arange(W, device="cuda", dtype=torch.float32) + 0.5) * (2.0 / W) - 1.0
    ay = ((torch.arange(y0, y1, device="cuda", dtype=torch.float32) + 0.5) * 2.0 - H) / W
    vol = torch.full((y1 - y0, W, W), 0.02, device="cuda")
    for x, y, z, rad, mu in _spheres(seed):
        r2 = (ay - y * H / W).square()[:, None, None] + (ax - z).square()[None, :, None] + \
            (ax - x).square()[None, None, :]
        vol += (r2 < rad * rad) * mu
        del r2
    vol *= _scale(g) * g["vx"]
    vol *= torch.empty_like(vol).uniform_(0.9, 1.1, generator=gen)
    return vol.reshape(-1)


def _images(c, g, pd, seed, gen):
    """Line integrals of the phantom along every pixel's ray, with 1 % noise: float32 [P, H, W]."""
    W, H, M, P = c["dw"], c["dh"], c["modules"], c["proj"]
    half = 0.5 * g["vwidth"] * g["vx"]
    m = torch.from_numpy(pd.astype(np.float64)).cuda().view(P, M, 20)
    out = torch.zeros(P, H, W, device="cuda")
    u = torch.arange(W, device="cuda", dtype=torch.float64)
    v = torch.arange(H, device="cuda", dtype=torch.float64)
    up = g["vheight"] / g["vwidth"]
    for k in range(M):
        cu, cv, cw = m[:, k, 0:3], m[:, k, 4:7], m[:, k, 12:15]
        src = torch.linalg.solve(torch.stack([cu, cv, cw], 1), -m[:, k, [3, 7, 15]])
        left, right = max(0, math.ceil(pd.reshape(P, M, 20)[0, k, 16])), min(W, math.ceil(pd.reshape(P, M, 20)[0, k, 17]))
        n1 = u[left:right, None, None] * cw - cu          # [U, P, 3]: the plane of a detector column
        n2 = v[:, None, None] * cw - cv                   # [V, P, 3]: the plane of a detector row
        for p in range(P):
            d = torch.linalg.cross(n1[None, :, p], n2[:, None, p]).float()
            d = d / d.norm(dim=-1, keepdim=True)
            for x, y, z, rad, mu in _spheres(seed):
                t = torch.tensor([x, y * up, z], device="cuda", dtype=torch.float64) * half - src[p]
                b = (d * t.float()).sum(-1)
                h2 = (rad * half) ** 2 - (float(t.square().sum()) - b.square())
                out[p, :, left:right] += (2.0 * mu * _scale(g)) * h2.clamp_min(0.0).sqrt()
    out *= torch.empty_like(out).normal_(1.0, 0.01, generator=gen)
    return out.add_(0.01).clamp_min_(EPS)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _layers(c, g):
    n = c["layers"] or g["vheight"]
    y0 = (g["vheight"] - n) // 2
    return y0, y0 + n


def _op_inputs(c, seed):
    """Everything an operator call reads, as device tensors."""
    gen = _gen(seed)
    pd, g, origin = _plan(c, seed)
    layers = _layers(c, g)
    s = dict(pd=pd, g=g, origin=origin, layers=layers, vol=_volume(g, seed, layers, gen))
    npix = c["proj"] * c["dh"] * c["dw"]
    if c["op"] == "sub":
        s["images"] = _images(c, g, pd, seed, gen).reshape(-1).to(torch_dtype(STORAGE[c["images"]]))
    if c["op"] == "backward":
        # log ratios of a late sub-iteration: a few per mille
        s["ratio"] = torch.empty(npix, device="cuda").normal_(0.0, 3e-3, generator=gen) \
            .to(torch_dtype(STORAGE[c["ratio"]]))
    return s


def prepare(c, seed):
    op = c["op"]
    if op == "preprocess":
        n = c["proj"] * c["dh"] * c["dw"]
        return dict(op=op, c=c, raw=_raw(c, seed), n=n, ctx=_context(),
                    out=torch.empty(n, device="cuda", dtype=torch_dtype(STORAGE[c["images"]])),
                    start=torch.tensor([3.4028234e38, -3.4028234e38], device="cuda"),
                    minmax=torch.empty(2, device="cuda"))
    if op == "reconstruct":
        pd, g, _ = _plan(c, seed)
        raw = _images(c, g, pd, seed, _gen(seed)).neg_().exp_().cpu().numpy()
        params = {"recon": {"method": c["method"], "it": c["it"], "sit": c["sit"], "seed": 11, "mlog": True},
                  "geometry": {"so": 100.0, "sd": 1000.0, "angle": 360.0}, "detector": {"px": 0.1}}
        L = _lib.lib()
        L.xpr_reconstruct_host.argtypes = [C.c_char_p, C.c_void_p, C.c_int64, C.c_uint32, C.c_uint32, C.c_void_p,
                                           C.c_uint64, C.POINTER(C.c_double)]
        return dict(op=op, c=c, raw=raw, params=json.dumps(params).encode(),
                    out=np.empty((g["vheight"], g["vwidth"], g["vwidth"]), np.float32))
    if op == "batch":
        probs = [_problem(c, k, seed) for k in range(c["count"])]
        b = Batch(_context(), probs, arith=ARITH[c["arith"]], storage=STORAGE[c["ratio"]],
                  image_storage=STORAGE[c["images"]])
        return dict(op=op, batch=b, probs=probs)
    s = _op_inputs(c, seed)
    rec = Reconstruction(_context(), arith=ARITH[c["arith"]])
    g, (y0, y1) = s["g"], s["layers"]
    npix = c["proj"] * c["dh"] * c["dw"]
    rec.set_image_parameters(c["dw"], c["dh"], c["proj"])
    rec.set_volume_parameters((0, y0, 0), (g["vwidth"], y1, g["vwidth"]), [g["vx"]] * 3)
    rec.set_angle_number(c["proj"], c["modules"])
    rec.set_origin(s["origin"])
    rec.set_volume_buffer(s["vol"])
    rec.set_projdata_buffer(torch.from_numpy(s["pd"]).cuda())
    if c["lists"]:
        e = torch.arange(c["proj"] * c["modules"], device="cuda")
        rec.set_angle_list(e.to(torch.uint16), (e // c["modules"]).to(torch.uint16), nan_skip=True)
    s.update(op=op, rec=rec)
    if op in ("forward", "sub"):
        s["sums"] = torch.zeros(npix, dtype=torch.int32, device="cuda")
        rec.set_sum_images_buffer(s["sums"])
    if op == "backward":
        rec.set_ratio_buffer(s["ratio"])
    if op == "sub":
        s["ratio"] = torch.empty(npix, dtype=torch_dtype(STORAGE[c["ratio"]]), device="cuda")
        rec.set_ratio_buffer(s["ratio"])
        rec.set_images_buffer(s["images"])
        rec.set_weight(0.9)
    torch.cuda.synchronize()
    return s


def _raw(c, seed):
    """Detector counts of a scan, a few dead pixels among them."""
    gen = _gen(seed)
    n = c["proj"] * c["dh"] * c["dw"]
    raw = torch.empty(n, device="cuda").uniform_(0.0, 2.0, generator=gen).neg_().exp_()
    raw *= torch.empty(n, device="cuda").normal_(1.0, 0.01, generator=gen)
    raw[torch.randint(0, n, (max(1, n // 50000),), device="cuda", generator=gen)] = 0.0
    return raw * 6e4 if c["normalize"] else raw


def _problem(c, k, seed):
    """Problem k of a batch: its detector between dw and dw_max, images in subset-major order."""
    f = k / max(1, c["count"] - 1)
    dw = int(round(c["dw"] + f * (c["dw_max"] - c["dw"])))
    if c["modules"] > 1:
        dw -= dw % c["modules"]
    one = dict(c, dw=dw, dh=int(round(c["dh"] * dw / c["dw"])))
    sit, Pc = c["sit"], c["proj"] // c["sit"]
    one["proj"] = sit * Pc
    pd, g, _ = _plan(one, seed + 1009 * k)
    order = [s + j * sit for s in range(sit) for j in range(Pc)]
    pd = np.ascontiguousarray(pd.reshape(one["proj"], -1, 20)[order].reshape(-1, 20))
    gen = _gen(seed + k)
    # smooth attenuations between 0.05 and 1: what they depict does not matter to the run's cost
    small = torch.rand(1, one["proj"], max(2, one["dh"] // 8), max(2, dw // 8), device="cuda", generator=gen)
    img = torch.nn.functional.interpolate(small, size=(one["dh"], dw), mode="bilinear")
    vw, vh = int(g["vwidth"]), int(g["vheight"])
    return Problem(vol=torch.ones(vw * vh * vw, device="cuda"),
                   images=(img * 0.95 + 0.05).reshape(-1).to(torch_dtype(STORAGE[c["images"]])),
                   projdata=torch.from_numpy(pd).cuda(), det_w=dw, det_h=one["dh"], per_subset=Pc,
                   modules=c["modules"], sit=sit, it=c["it"], vwidth=vw, vheight=vh, voxel=float(g["vx"]),
                   orig=tuple(float(x) for x in g["orig"]), seed=5489 + k)


# ------------------------------------------------------------------------------ one pass
def run(s):
    op = s["op"]
    if op == "preprocess":
        L, c, sp = _lib.lib(), s["c"], C.c_void_p(torch.cuda.current_stream().cuda_stream)
        h = s["ctx"].handle
        if c["normalize"]:
            s["minmax"].copy_(s["start"])
            _lib.check(L.xpr_preprocess_minmax(h, s["raw"].data_ptr(), s["n"], s["minmax"].data_ptr(), sp), "minmax")
        _lib.check(L.xpr_preprocess_apply(h, s["raw"].data_ptr(), s["out"].data_ptr(), STORAGE[c["images"]], s["n"],
                                          int(c["normalize"]), s["minmax"].data_ptr() if c["normalize"] else None, 1,
                                          sp), "preprocess")
        return s["out"]
    if op == "reconstruct":
        c = s["c"]
        _lib.check(_lib.lib().xpr_reconstruct_host(s["params"], s["raw"].ctypes.data, c["proj"], c["dw"], c["dh"],
                                                   s["out"].ctypes.data, s["out"].size, None), "reconstruct")
        return s["out"]
    if op == "batch":
        s["batch"].run()
        return [p.vol for p in s["probs"]]
    rec = s["rec"]
    if op == "forward":
        s["sums"].zero_()
        rec.forward()
        return s["sums"]
    if op == "backward":
        rec.backward()
        return s["vol"]
    s["sums"].zero_()
    rec.forward()
    rec.error()
    rec.backward()
    return dict(vol=s["vol"], sums=s["sums"], ratio=s["ratio"])


# ------------------------------------------------------------------------------ work and values
def work(c):
    px = 4 if c.get("images") == "fp32" else 2
    if c["op"] == "preprocess":
        n = c["proj"] * c["dh"] * c["dw"]
        return {"bytes": n * (4 + px), "flops": 20.0 * n}
    if c["op"] == "reconstruct":
        vox, n = c["dw"] * c["dw"] * c["dh"], c["proj"] * c["dh"] * c["dw"]
        return {"bytes": 4.0 * (vox + n), "flops": 44.0 * vox * (c["proj"] // c["sit"]) * c["sit"] * c["it"]}
    rt = 4 if c["ratio"] == "fp32" else 2
    if c["op"] == "batch":
        b = f = 0.0
        for k in range(c["count"]):
            t = k / max(1, c["count"] - 1)
            dw = int(round(c["dw"] + t * (c["dw_max"] - c["dw"])))
            if c["modules"] > 1:
                dw -= dw % c["modules"]
            dh = int(round(c["dh"] * dw / c["dw"]))
            vox, npix, steps = dw * dh * dw, dw * dh * (c["proj"] // c["sit"]), c["it"] * c["sit"]
            b += npix * c["sit"] * px + 4.0 * vox
            f += 44.0 * vox * (c["proj"] // c["sit"]) * steps
        return {"bytes": b, "flops": f}
    # the grid is as wide as the detector and as tall as it has rows (voxel = pixel at the axis)
    vox, npix = c["dw"] * c["dw"] * (c["layers"] or c["dh"]), c["proj"] * c["dh"] * c["dw"]
    pairs = float(vox) * c["proj"]
    if c["op"] == "forward":
        return {"bytes": 4.0 * vox + 4.0 * npix, "flops": 22.0 * pairs}
    if c["op"] == "backward":
        return {"bytes": 8.0 * vox + rt * npix, "flops": 22.0 * pairs}
    return {"bytes": 8.0 * vox + (px + 4.0 + rt) * npix, "flops": 44.0 * pairs}


def _pixels(s, c, e, ys):
    """Flat detector index and in-bounds mask of the voxels of layers ys for ProjData entry e, in 64 bits."""
    g = s["g"]
    m = s["pd"][e].astype(np.float64)
    W = g["vwidth"]
    p = [torch.arange(W, device="cuda", dtype=torch.float64) * g["vx"] + s["origin"][i] for i in (0, 2)]
    py = ys.double() * g["vx"] + s["origin"][1]

    def row(r):
        return (py * m[r + 1])[:, None, None] + (p[1] * m[r + 2])[None, :, None] + \
            (p[0] * m[r] + m[r + 3])[None, None, :]

    w = row(12)
    iu, iv = (row(0) / w + 0.5).floor_(), (row(4) / w + 0.5).floor_()
    l, r, b, t = (math.ceil(x) for x in s["pd"][e][16:20])
    ok = (iu >= max(l, 0)) & (iu < min(r, c["dw"])) & (iv >= max(b, 0)) & (iv < min(t, c["dh"]))
    idx = (iv * c["dw"] + iu).long()
    idx += (e // c["modules"]) * c["dw"] * c["dh"]
    return torch.where(ok, idx, 0), ok


def _slabs(s):
    y0, y1 = s["layers"]
    step = max(1, (1 << 25) // s["g"]["vwidth"] ** 2)
    for a in range(y0, y1, step):
        yield a - y0, torch.arange(a, min(y1, a + step), device="cuda")


def _sums64(s, c):
    W = s["g"]["vwidth"]
    out = torch.zeros(c["proj"] * c["dh"] * c["dw"], dtype=torch.float64, device="cuda")
    for a, ys in _slabs(s):
        val = s["vol"].view(-1, W, W)[a:a + len(ys)].double()
        for e in range(c["proj"] * c["modules"]):
            idx, ok = _pixels(s, c, e, ys)
            out.index_add_(0, idx.reshape(-1), (val * ok).reshape(-1))
    return out


def _update64(s, c, ratio):
    W = s["g"]["vwidth"]
    out = s["vol"].double().view(-1, W, W).clone()
    for a, ys in _slabs(s):
        acc = torch.zeros(len(ys), W, W, dtype=torch.float64, device="cuda")
        cnt = torch.zeros_like(acc)
        for e in range(c["proj"] * c["modules"]):
            idx, ok = _pixels(s, c, e, ys)
            acc += ratio[idx] * ok
            cnt += ok
        out[a:a + len(ys)] *= (acc / cnt).exp()
    return out.reshape(-1)


def exact(c, seed):
    if c["op"] == "preprocess":
        x = _raw(c, seed)
        tiny = x.abs() < 1.1754944e-38  # dead pixels take the middle value
        x = x.double()
        if c["normalize"]:
            mn, mx = x[~tiny].min(), x[~tiny].max()
            x = torch.where(tiny, (mx + mn) / 2.0, (x - mn) / (mx - mn))
        return -x.clamp(EPS, 1.0 - EPS).log()
    if c["op"] in ("batch", "reconstruct", "forward"):
        return None  # whole runs amplify each nearest-pixel choice; detector sums are whole numbers
    s = _op_inputs(c, seed)
    if c["op"] == "backward":
        return _update64(s, c, s["ratio"].double())
    if float(work(c)["flops"]) > 6e11:
        return None
    sums = _sums64(s, c)
    ratio = (s["images"].double() / sums.clamp_min(EPS)).clamp_min(EPS).log() * 0.9
    return dict(vol=_update64(s, c, ratio), sums=None, ratio=ratio)
