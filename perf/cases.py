"""The work a program has this framework do, as cases that can be timed.

A case names one public entry point, its sizes, sample type and options;
`prepare` makes its seeded inputs on the GPU (on the host where the call takes
host buffers), `run` is one call, `work` the bytes that call cannot do
without, and `exact` a plain float64 restatement of the float results.

The cases share one `Context`, as a program that processes one image set after
another does, with new images (and buffers) from set to set.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "enblend-enfuse_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import enbgpu  # noqa: E402
from enbgpu import synthetic  # noqa: E402

_TORCH = {"u8": torch.uint8, "u16": torch.uint16, "f32": torch.float32}
_BYTES = {"u8": 1, "u16": 2, "f32": 4}

_context = None


def _ctx():
    global _context
    if _context is None:
        _context = enbgpu.Context(0)
    _context.set_stream(torch.cuda.current_stream().cuda_stream)
    return _context


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def _enfuse(k, w, h, dtype, con=0, ent=0, alpha=False, wrap=False, hard=False, host=False):
    """enfuse of k exposures; con / ent: window sizes of the contrast and entropy weights, 0 leaves them out."""
    return {"call": "enfuse", "k": k, "w": w, "h": h, "dtype": dtype, "con": con, "ent": ent, "alpha": alpha,
            "wrap": wrap, "hard": hard, "host": host}


def _enblend(w, h, offset, dtype, rgba=True, pitched=False, wrap=False, host=False):
    """enblend of two w x h images `offset` columns apart; rgba: alpha in the 4th component, else in planes."""
    return {"call": "enblend", "w": w, "h": h, "offset": offset, "dtype": dtype, "rgba": rgba, "pitched": pitched,
            "wrap": wrap, "host": host}


def listed():
    return [
        # a camera's bracket fused for a preview: the smallest call, all latency and launches
        dict(_enfuse(3, 251, 187, "u8"), name="enfuse_preview_u8"),
        # the common bracket of three 8-bit exposures, exposure and saturation weights
        dict(_enfuse(3, 1024, 768, "u8"), name="enfuse_3x1024x768_u8"),
        # a full-frame 16-bit bracket with every weight (5x5 windows)
        dict(_enfuse(9, 6000, 4000, "u16", con=5, ent=5), name="enfuse_9x6000x4000_u16"),
        # focus stacking of aligned, so ragged, 16-bit frames: alpha holes, contrast alone decides, hard masks
        dict(_enfuse(5, 2047, 1535, "u16", con=5, alpha=True, hard=True), name="enfuse_focus_u16_alpha"),
        # one float bracket (raw development) with every weight
        dict(_enfuse(4, 1601, 1203, "f32", con=5, ent=5), name="enfuse_4x1601x1203_f32"),
        # the panorama step: two 16-bit images into one canvas, rows padded as the host staging pads them
        dict(_enblend(4096, 3072, 2867, "u16", pitched=True), name="enblend_2x4096x3072_u16"),
        # a small 360-degree panorama step of 8-bit RGB images with alpha planes, dense odd rows
        dict(_enblend(1001, 753, 701, "u8", rgba=False, wrap=True), name="enblend_u8_wrap"),
        # what the command line does with each image: host buffers in, host buffers out
        dict(_enblend(2048, 1536, 1434, "u8", host=True), name="enblend_host_u8"),
        # a day's brackets of all sizes fused as one batch
        {"call": "stacks", "n": 16, "lo": 512, "hi": 4096, "layout": 4, "name": "stacks_16_f32"},
        # one optimisation step of the fuse's parameters and per-pixel logits
        {"call": "grad", "k": 8, "w": 2048, "h": 2048, "con": 5, "name": "grad_8x2048x2048"},
        # the seam of a panorama step from the two footprints
        {"call": "seam", "w": 4096, "h": 3072, "offset": 2867, "wrap": False, "name": "seam_6963x3072"},
        # the pyramid calls one by one, as the C++ adaptor's users make them
        {"call": "pyramids", "w": 1921, "h": 1081, "dtype": "u16", "wrap": False, "name": "pyramids_1921x1081_u16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["enfuse", "enfuse", "enfuse", "enblend", "enblend", "stacks", "grad", "seam", "pyramids"])
    if call == "enfuse":
        dtype = rng.choice(["u8", "u16", "f32"])
        w, h, k = _log(rng, 160, 6000), _log(rng, 120, 4000), rng.randint(2, 9)
        if dtype == "f32":  # the float fuse is drawn up to the largest single stack of a batch
            w, h, k = min(w, 4096), min(h, 4096), min(k, 7)
        c = _enfuse(k, w, h, dtype, con=rng.choice([0, 3, 5, 5]), ent=rng.choice([0, 0, 3, 5]))
        if dtype != "f32":
            c.update(alpha=rng.random() < 0.3, wrap=rng.random() < 0.2, hard=rng.random() < 0.2,
                     host=rng.random() < 0.2)
        return c
    if call == "enblend":
        w, h = _log(rng, 400, 4096), _log(rng, 300, 3072)
        c = _enblend(w, h, int(w * rng.uniform(0.5, 0.8)), rng.choice(["u8", "u16"]), rgba=rng.random() < 0.6,
                     pitched=rng.random() < 0.5, wrap=rng.random() < 0.3)
        if rng.random() < 0.25:
            c.update(host=True, pitched=False)
        return c
    if call == "stacks":
        return {"call": "stacks", "n": rng.randint(2, 16), "lo": 512, "hi": _log(rng, 1024, 3072),
                "layout": rng.randrange(1 << 16)}
    if call == "grad":
        return {"call": "grad", "k": rng.randint(2, 8), "w": _log(rng, 300, 2048), "h": _log(rng, 300, 2048),
                "con": rng.choice([3, 5])}
    if call == "seam":
        w = _log(rng, 400, 4096)
        return {"call": "seam", "w": w, "h": _log(rng, 300, 3072), "offset": int(w * rng.uniform(0.5, 0.8)),
                "wrap": rng.random() < 0.3}
    return {"call": "pyramids", "w": _log(rng, 200, 4096), "h": _log(rng, 200, 3072),
            "dtype": rng.choice(["u8", "u16"]), "wrap": rng.random() < 0.3}


def _specs(case):
    """The batch's stacks: (height, width, exposure values) from the case alone."""
    rng = np.random.default_rng(case["layout"])
    out = []
    for _ in range(case["n"]):
        w, h = (int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]))))) for _ in range(2))
        k = int(rng.integers(3, 8))
        out.append((h, w, [float(e) for e in np.linspace(1 - k, k - 1, k)]))
    return out


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _quantise(v, dtype):
    """Samples in [0, 1] as the sample type."""
    v = v.clamp(0.0, 1.0)
    if dtype == "f32":
        return v.contiguous()
    q = torch.round(v * (255.0 if dtype == "u8" else 65535.0)).to(torch.int32)
    return q.to(torch.uint8).contiguous() if dtype == "u8" else q.to(torch.int16).view(torch.uint16).contiguous()


def _scene(h, w, stops, seed):
    """Log radiance of a scene; the generator's noise grid wants 512 pixels a side, small scenes are cut from that."""
    return synthetic.log_radiance_torch(max(h, 512), max(w, 512), stops, seed)[:h, :w].contiguous()


def _exposures(w, h, k, dtype, seed, spread=None):
    """k exposures of one scene, one stop apart (or over +-spread), sensor noise before quantisation."""
    lr = _scene(h, w, 12.0 if k > 5 else 8.0, seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 7919)
    spread = (k - 1) / 2.0 if spread is None else spread
    out = []
    for ev in np.linspace(-spread, spread, k):
        v = torch.exp2(lr + float(ev)) ** (1.0 / 2.2)
        if dtype != "f32":
            v += 2.0 ** -12 * torch.randn(v.shape, generator=gen, device="cuda")
        out.append(_quantise(v, dtype))
    return out


def _footprint(w, h, angle, margin):
    """1 inside a slightly rotated rectangle of the canvas (the frame of an aligned image), else 0."""
    y = (torch.arange(h, device="cuda", dtype=torch.float32) - (h - 1) / 2)[:, None]
    x = (torch.arange(w, device="cuda", dtype=torch.float32) - (w - 1) / 2)[None, :]
    c, s = math.cos(angle), math.sin(angle)
    return (((c * x + s * y).abs() <= w * (0.5 - margin)) & ((c * y - s * x).abs() <= h * (0.5 - margin)))


def _panorama(case, seed):
    """Two overlapping images on their union canvas, the 0/255 seam mask and the two alpha planes."""
    h, w, off = case["h"], case["w"], case["offset"]
    wu = w + off
    rng = np.random.default_rng(seed)
    lr = _scene(h, wu, 8.0, seed)
    one = {"u8": 255, "u16": 65535}[case["dtype"]]
    images, alphas = [], []
    for x0 in (off, 0):
        pix = _quantise(float(rng.uniform(0.9, 1.1)) * torch.exp2(lr) ** (1.0 / 2.2), case["dtype"])
        alpha = torch.zeros((h, wu), dtype=torch.uint8, device="cuda")
        alpha[:, x0:x0 + w] = 255
        wide = pix.to(torch.int32) * (alpha != 0)[..., None]
        if case["rgba"]:
            wide = torch.cat([wide, (alpha != 0).to(torch.int32)[..., None] * one], dim=2)
        images.append(wide.to(torch.uint8).contiguous() if one == 255
                      else wide.to(torch.int16).view(torch.uint16).contiguous())
        alphas.append(alpha)
    walk = (off + w) // 2 + np.cumsum(rng.integers(-1, 2, size=h))
    seam = torch.from_numpy(np.clip(walk, off + 1, w - 1)).cuda()
    mask = (torch.arange(wu, device="cuda")[None, :] >= seam[:, None]).to(torch.uint8) * 255
    return images[0], images[1], mask, alphas


def _params(case, float_range=1.0):
    kw = dict(saturation_weight=0.2, float_range=float_range)
    if case.get("hard"):  # focus stacking: contrast alone
        kw.update(exposure_weight=0.0, saturation_weight=0.0, contrast_weight=1.0, contrast_window_size=case["con"] or 5)
        return enbgpu.enfuse_params(**kw)
    if case["con"]:
        kw.update(contrast_weight=0.5, contrast_window_size=case["con"])
    if case.get("ent"):
        kw.update(entropy_weight=0.3, entropy_window_size=case["ent"])
    return enbgpu.enfuse_params(**kw)


def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    call = case["call"]
    if call == "enfuse":
        w, h, k, dtype = case["w"], case["h"], case["k"], case["dtype"]
        images, alphas = _exposures(w, h, k, dtype, seed), None
        if case["alpha"]:
            rng = np.random.default_rng(seed)
            alphas = [_footprint(w, h, float(rng.uniform(-0.02, 0.02)), 0.01).to(torch.uint8) * 255 for _ in range(k)]
        out = torch.zeros((h, w, 3), dtype=_TORCH[dtype], device="cuda")
        out_alpha = torch.zeros((h, w), dtype=torch.uint8, device="cuda")
        if case["host"]:
            images, out, out_alpha = [_host(x) for x in images], _host(out), _host(out_alpha)
            alphas = [_host(a) for a in alphas] if alphas else None
        return {"case": case, "ctx": _ctx(), "images": images, "alphas": alphas, "out": out, "out_alpha": out_alpha,
                "params": _params(case)}
    if call == "enblend":
        white, black, mask, alphas = _panorama(case, seed)
        alphas = [None, None] if case["rgba"] else alphas
        out, out_alpha = torch.zeros_like(black), torch.zeros_like(mask)
        if case["host"]:
            white, black, mask, out, out_alpha = (_host(x) for x in (white, black, mask, out, out_alpha))
            alphas = [a if a is None else _host(a) for a in alphas]
        elif case["pitched"]:
            white, black, mask, out, out_alpha = (enbgpu.pitched(x) for x in (white, black, mask, out, out_alpha))
            alphas = [a if a is None else enbgpu.pitched(a) for a in alphas]
        return {"case": case, "ctx": _ctx(), "white": white, "black": black, "mask": mask, "alphas": alphas,
                "out": out, "out_alpha": out_alpha}
    if call == "stacks":
        stacks = [_exposures(w, h, len(evs), "f32", seed * 1000 + i, spread=evs[-1])
                  for i, (h, w, evs) in enumerate(_specs(case))]
        return {"case": case, "ctx": _ctx(), "stacks": stacks, "outs": [torch.zeros_like(s[0]) for s in stacks],
                "params": enbgpu.enfuse_params(saturation_weight=0.2, contrast_weight=0.5, entropy_weight=0.3,
                                               contrast_window_size=5, entropy_window_size=5, float_range=1.0)}
    if call == "grad":
        w, h, k = case["w"], case["h"], case["k"]
        lr = _scene(h, w, 8.0, seed)
        rad = torch.exp2(lr)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed + 17)
        return {"case": case, "ctx": _ctx(), "images": _exposures(w, h, k, "f32", seed),
                "target": ((rad / (1.0 + rad)) ** (1.0 / 2.2)).contiguous(),
                "logits": [0.1 * torch.randn((h, w), generator=gen, device="cuda") for _ in range(k)],
                "out": torch.zeros((h, w, 3), device="cuda"),
                "grad_logits": [torch.zeros((h, w), device="cuda") for _ in range(k)], "params": _params(case)}
    if call == "seam":
        w, h, off = case["w"], case["h"], case["offset"]
        rng = np.random.default_rng(seed)
        planes = []
        for x0 in (off, 0):
            a = torch.zeros((h, w + off), dtype=torch.uint8, device="cuda")
            a[:, x0:x0 + w] = _footprint(w, h, float(rng.uniform(-0.02, 0.02)), 0.01).to(torch.uint8) * 255
            planes.append(a)
        return {"case": case, "ctx": _ctx(), "white": planes[0], "black": planes[1], "mask": torch.zeros_like(planes[0])}
    w, h, dtype = case["w"], case["h"], case["dtype"]
    white, black = _exposures(w, h, 2, dtype, seed)
    rng = np.random.default_rng(seed)
    alphas = [_footprint(w, h, float(rng.uniform(-0.02, 0.02)), 0.01).to(torch.uint8) * 255 for _ in range(2)]
    mask = (_footprint(w, h, float(rng.uniform(-0.2, 0.2)), 0.25).to(torch.uint8) * 255).contiguous()
    return {"case": case, "ctx": _ctx(), "white": white, "black": black, "alphas": alphas, "mask": mask,
            "union": (alphas[0] | alphas[1]).contiguous(), "out": torch.zeros_like(black),
            "levels": enbgpu.num_levels(w, h)}


# --------------------------------------------------------------------------
# one call
# --------------------------------------------------------------------------

def _samples(x):
    """16-bit pixels as the int16 view of the same bits (torch does not index uint16)."""
    if isinstance(x, np.ndarray):
        return x.view(np.int16) if x.dtype == np.uint16 else x
    return x.view(torch.int16) if x.dtype == torch.uint16 else x


def run(s):
    case, ctx = s["case"], s["ctx"]
    call = case["call"]
    if call == "enfuse":
        out, alpha = ctx.enfuse(s["images"], s["alphas"], params=s["params"], out=s["out"], out_alpha=s["out_alpha"],
                                wrap=case["wrap"], hard_mask=case["hard"])
        return {"out": _samples(out), "alpha": alpha}
    if call == "enblend":
        out, alpha = ctx.enblend(s["white"], s["black"], s["mask"], *s["alphas"], out=s["out"],
                                 out_alpha=s["out_alpha"], wrap=case["wrap"])
        return {"out": _samples(out), "alpha": alpha}
    if call == "stacks":
        return ctx.fuse_stacks(s["stacks"], params=s["params"], outs=s["outs"])
    if call == "grad":
        r = ctx.fuse_grad(s["images"], s["target"], params=s["params"], logits=s["logits"], out=s["out"],
                          grad_logits=s["grad_logits"])
        return {"scalars": r, "out": s["out"], "grad_logits": s["grad_logits"]}
    if call == "seam":
        return ctx.nft_mask(s["white"], s["black"], mask=s["mask"], wrap=case["wrap"])
    wrap, levels = case["wrap"], s["levels"]
    u8 = case["dtype"] == "u8"
    frac = 7 if u8 else 15
    gp = ctx.gaussian_pyramid(s["mask"], levels, wrap=wrap, frac_bits=frac, dtype=enbgpu.ENB_I16 if u8 else enbgpu.ENB_I32)
    wl = ctx.laplacian_pyramid(s["white"], levels, alpha=s["alphas"][0], wrap=wrap)
    bl = ctx.laplacian_pyramid(s["black"], levels, alpha=s["alphas"][1], wrap=wrap)
    ctx.blend_pyramids(gp, wl, bl, 255 << frac)
    ctx.collapse_pyramid(bl, wrap=wrap)
    ctx.from_pyramid(bl, 0, s["union"], s["out"])
    for p in (gp, wl, bl):
        p.free()
    return _samples(s["out"])


def work(case):
    """Each input read once, each output written once."""
    call = case["call"]
    if call == "enfuse":
        px = case["w"] * case["h"]
        b = px * (3 * _BYTES[case["dtype"]] + (1 if case["alpha"] else 0))
        return {"bytes": case["k"] * b + px * (3 * _BYTES[case["dtype"]] + 1), "flops": 0}
    if call == "enblend":
        px = (case["w"] + case["offset"]) * case["h"]
        b = (4 if case["rgba"] else 3) * _BYTES[case["dtype"]]
        return {"bytes": px * (3 * b + 2 + (0 if case["rgba"] else 2)), "flops": 0}
    if call == "stacks":
        return {"bytes": sum(h * w * 12 * (len(evs) + 1) for h, w, evs in _specs(case)), "flops": 0}
    if call == "grad":
        return {"bytes": case["w"] * case["h"] * (case["k"] * (12 + 4 + 4) + 24), "flops": 0}
    if call == "seam":
        return {"bytes": 3 * (case["w"] + case["offset"]) * case["h"], "flops": 0}
    return {"bytes": case["w"] * case["h"] * (9 * _BYTES[case["dtype"]] + 4), "flops": 0}


# --------------------------------------------------------------------------
# the float results in 64 bits
# --------------------------------------------------------------------------

def _windows(x, n):
    """The n*n shifted views of the last two axes."""
    H, W = x.shape[-2:]
    return [x[..., i:H - n + 1 + i, j:W - n + 1 + j] for i in range(n) for j in range(n)]


def _inside(x, n, like):
    out = torch.zeros_like(like)
    b = n // 2
    out[..., b:like.shape[-2] - b, b:like.shape[-1] - b] = x
    return out


def _weight64(img, con, ent, theta):
    """Weight of one (3, H, W) float64 exposure; theta: optimum, width, exposure, saturation, contrast weight."""
    opt, width, w_exp, w_sat, w_con = theta
    gray = img.sum(0) / 3.0
    e = w_exp * torch.exp(-0.5 * ((gray - opt) / width) ** 2)
    if con:
        ws = _windows(gray, con)
        mean = sum(ws) / len(ws)
        var = sum((v - mean) ** 2 for v in ws) / (len(ws) - 1)
        on = var > 1e-20
        e = e + w_con * _inside(torch.where(on, torch.sqrt(torch.where(on, var, torch.ones_like(var))),
                                            torch.zeros_like(var)), con, gray)
    mx, mn = img.max(0).values, img.min(0).values
    den = torch.where(mx + mn <= 1.0, mx + mn, 2.0 - mx - mn)
    on = mx != mn
    e = e + w_sat * torch.where(on, (mx - mn) / torch.where(on, den, torch.ones_like(den)), torch.zeros_like(den))
    if ent:
        low = None
        for c in range(3):
            ws = _windows(img[c].float().contiguous(), ent)  # equality of float samples: float32 holds them exactly
            plog, bins = 0.0, 0.0
            for a in ws:
                n = torch.zeros(a.shape, dtype=torch.uint8, device=a.device)
                for b in ws:
                    n += a == b
                n = n.double()
                plog = plog - torch.log(n / len(ws))
                bins = bins + 1.0 / n
            bins = bins.round()
            hh = torch.where(bins > 1, plog / len(ws) / torch.log(bins.clamp(min=2.0)), torch.zeros_like(plog))
            low = hh if low is None else torch.minimum(low, hh)
        e = e + 0.3 * _inside(low, ent, gray)
    return e


def _down1(x, dim):
    """The opaque 5-tap reduce along one axis, normalised at the ends."""
    x = x.transpose(dim, -1)
    n = x.shape[-1]
    m = (n + 1) // 2
    pad = torch.nn.functional.pad
    xp = pad(x, (2, 2 * m + 1 - n))
    one = pad(torch.ones(n, dtype=x.dtype, device=x.device), (2, 2 * m + 1 - n))
    num = sum(k * xp[..., t:t + 2 * m - 1:2] for t, k in enumerate((1.0, 4.0, 6.0, 4.0, 1.0)))
    den = sum(k * one[t:t + 2 * m - 1:2] for t, k in enumerate((1.0, 4.0, 6.0, 4.0, 1.0)))
    return (num / den).transpose(dim, -1)


def _up1(x, n, dim):
    """The (1, 6, 1) / (4, 4) expand along one axis to n samples."""
    x = x.transpose(dim, -1)
    m = x.shape[-1]
    xp = torch.nn.functional.pad(x, (1, 1))
    one = torch.nn.functional.pad(torch.ones(m, dtype=x.dtype, device=x.device), (1, 1))
    even = (xp[..., :m] + 6.0 * xp[..., 1:m + 1] + xp[..., 2:]) / (one[:m] + 6.0 + one[2:])
    odd = (xp[..., 1:m + 1] + xp[..., 2:]) / (1.0 + one[2:])
    return torch.stack([even, odd], dim=-1).flatten(-2)[..., :n].transpose(dim, -1)


def _down(x):
    return _down1(_down1(x, -2), -1)


def _up(x, like):
    return _up1(_up1(x, like.shape[-2], -2), like.shape[-1], -1)


def _levels(w, h):
    short, n = min(w, h), 1
    while short > 8:
        short, n = (short + 1) // 2, n + 1
    return n


def _merge64(images, masks, levels):
    """Collapsed sum of the exposures' Laplacian pyramids times their mask pyramids; images of (3, H, W)."""
    total = None
    for img, m in zip(images, masks):
        g = torch.log1p(img)  # the pyramid value less 1, which no level of the merge sees
        lp = []
        for _ in range(levels - 1):
            nxt = _down(g)
            lp.append(g - _up(nxt, g))
            g = nxt
        lp.append(g)
        parts = []
        for l in range(levels):
            parts.append(lp[l] * m)
            if l + 1 < levels:
                m = _down(m)
        total = parts if total is None else [a + b for a, b in zip(total, parts)]
    c = total[-1]
    for l in range(levels - 2, -1, -1):
        c = total[l] + _up(c, total[l])
    return torch.where(c >= 0, torch.expm1(c.clamp(min=0.0)), 1.0 - 1.0 / (1.0 + c.clamp(max=0.0)))


def _fuse64(images, con, ent):
    """The fused float image: weights, soft masks, merge."""
    theta = (0.5, 0.2, 1.0, 0.2, 0.5)
    planes = [x.permute(2, 0, 1).double() for x in images]
    masks = [_weight64(x, con, ent, theta) for x in planes]
    norm = sum(masks)
    h, w = norm.shape
    out = _merge64(planes, [(m / norm) for m in masks], _levels(w, h))
    return out.permute(1, 2, 0).contiguous()


def exact(case, seed):
    call = case["call"]
    if call == "enfuse" and case["dtype"] == "f32":
        with torch.no_grad():
            return {"out": _fuse64(prepare(case, seed)["images"], case["con"], case["ent"]), "alpha": None}
    if call == "stacks":
        with torch.no_grad():
            return [_fuse64(st, 5, 5) for st in prepare(case, seed)["stacks"]]
    if call == "grad":
        s = prepare(case, seed)
        theta = torch.tensor([0.5, 0.2, 1.0, 0.2, 0.5 if case["con"] else 0.0], dtype=torch.float64, device="cuda",
                             requires_grad=True)
        logits = [a.double().requires_grad_(True) for a in s["logits"]]
        planes = [x.permute(2, 0, 1).double() for x in s["images"]]
        ws = [_weight64(x, case["con"], 0, theta) * torch.exp(a) for x, a in zip(planes, logits)]
        norm = sum(ws)
        out = _merge64(planes, [w / norm for w in ws], _levels(case["w"], case["h"]))
        loss = ((out - s["target"].permute(2, 0, 1).double()) ** 2).mean()
        loss.backward()
        g = theta.grad.tolist()
        return {"scalars": {"loss": float(loss.detach()), "d_exp_optimum": g[0], "d_exp_width": g[1],
                            "d_w_exposure": g[2], "d_w_saturation": g[3], "d_w_contrast": g[4] if case["con"] else 0.0},
                "out": out.detach().permute(1, 2, 0).contiguous(), "grad_logits": [a.grad for a in logits]}
    return None  # integer samples: equal or not
