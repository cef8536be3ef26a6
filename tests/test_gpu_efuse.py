"""The fused enfuse driver (enb_efuse.cu) against the oracle and against the
per-operation pass structure (enb_fuse_options.plain).

The fused passes must give the same integers as the reference's pass
structure: the collapsed level 0 and the dithered pixels are compared bit for
bit.  Cases cover 8- and 16-bit RGB, RGBA (alpha thresholded from the 4th
component), gray and explicit alpha planes, 1 to 16 exposures, odd and tiny
canvases (2 to 9 pyramid levels), wrap-around, the hard mask, --load-masks and
the exposure and entropy cutoffs; more than 16 exposures take the
per-operation passes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

W_ALL = dict(exposure_weight=1.0, saturation_weight=0.2, contrast_weight=0.5, entropy_weight=0.3,
             contrast_window_size=5, entropy_window_size=5)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _stack(dt, h, w, K, seed, S=3):
    from enbgpu import synthetic
    imgs = synthetic.exposure_stack(h, w, list(np.linspace(-3.0, 3.0, K)), dt, 8.0, seed=seed)
    if S == 4:
        rng = np.random.default_rng(seed)
        top = np.iinfo(dt).max
        imgs = [np.concatenate([x, np.full((h, w, 1), top, dt)], axis=2) for x in imgs]
        for i, x in enumerate(imgs):
            x[rng.random((h, w)) < 0.1, 3] = top // 3
            x[2 + i: 9 + i, 3:17, 3] = 0
    if S == 1:
        imgs = [np.ascontiguousarray(x[..., 1]) for x in imgs]
    return imgs


def _run(ctx, imgs, kw, **opt):
    import enbgpu
    h, w = imgs[0].shape[:2]
    C = 3 if imgs[0].ndim == 3 else 1
    l0 = torch.zeros((h, w, C), dtype=torch.int32, device="cuda")
    out, oa = ctx.enfuse([_dev(x) for x in imgs], params=enbgpu.enfuse_params(**kw) if kw is not None else None,
                         level0=l0, **opt)
    return l0.cpu().numpy(), out.cpu().numpy(), oa.cpu().numpy()


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("S", [3, 4, 1])
@pytest.mark.parametrize("geom", [(75, 97, 3), (40, 33, 1), (6, 7, 2), (130, 257, 5), (33, 64, 16)])
def test_fused_enfuse_against_oracle(ctx, orc, dt, S, geom):
    h, w, K = geom
    imgs = _stack(dt, h, w, K, seed=h + w + K, S=S)
    kw = W_ALL if min(h, w) >= 5 else dict(exposure_weight=1.0, saturation_weight=0.2)
    ref = orc.enfuse(imgs, None, orc.params(**kw), seed=17, want_level0=True)
    ctx.profile(True)
    l0, out, oa = _run(ctx, imgs, kw, seed=17)
    names = set(ctx.profile_report())
    ctx.profile(False)
    # a canvas whose short side is at most 8 pixels has one pyramid level,
    # which the per-operation passes take
    assert ("ef_out0" in names) == (orc.num_levels(w, h) >= 2), names
    C = 3 if S != 1 else 1
    assert np.array_equal(l0 if C == 3 else l0[..., 0], ref["level0"] if C == 3 else ref["level0"][..., 0])
    assert np.array_equal(oa, ref["alpha"])
    assert np.array_equal(out, ref["out"])


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("variant", ["hard", "wrap", "levels3", "alpha_planes", "cutoffs", "nearest"])
def test_fused_enfuse_equals_plain_passes(ctx, dt, variant):
    """The fused passes and one kernel per reference operation give the same bits."""
    h, w, K = 61, 83, 4
    imgs = _stack(dt, h, w, K, seed=5)
    kw, opt = dict(W_ALL), {}
    if variant == "hard":
        opt["hard_mask"] = True
    elif variant == "wrap":
        opt["wrap"] = True
    elif variant == "levels3":
        opt["levels"] = 3
    elif variant == "alpha_planes":
        rng = np.random.default_rng(9)
        opt["alphas"] = [_dev(((rng.random((h, w)) < 0.9) * 255).astype(np.uint8)) for _ in range(K)]
    elif variant == "cutoffs":
        kw.update(exposure_cutoff=((5.0, True), (95.0, True)), entropy_cutoff=((10.0, True), (90.0, True)))
    elif variant == "nearest":
        opt["dither"] = "nearest"
    a = _run(ctx, imgs, kw, seed=3, **opt)
    b = _run(ctx, imgs, kw, seed=3, plain=True, **opt)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("hard", [False, True])
def test_fused_enfuse_loaded_masks(ctx, orc, dt, hard):
    """--load-masks: the weights come from the caller; all-zero weights take
    the integer 255/K fallback (soft) or 255/K (hard)."""
    h, w, K = 50, 66, 3
    imgs = _stack(dt, h, w, K, seed=22)
    rng = np.random.default_rng(4)
    masks = [rng.random((h, w)).astype(np.float32) for _ in imgs]
    for m in masks:
        m[:5, :7] = 0.0
    ref = orc.enfuse(imgs, None, masks=masks, hard_mask=hard, seed=5, want_level0=True)
    l0, out, oa = _run(ctx, imgs, None, masks=[_dev(m) for m in masks], hard_mask=hard, seed=5)
    assert np.array_equal(l0, ref["level0"])
    assert np.array_equal(out, ref["out"])
    assert np.array_equal(oa, ref["alpha"])


def test_more_than_sixteen_exposures_take_the_plain_passes(ctx, orc):
    h, w, K = 24, 31, 17
    imgs = _stack(np.uint8, h, w, K, seed=8)
    kw = dict(exposure_weight=1.0, saturation_weight=0.2)
    ref = orc.enfuse(imgs, None, orc.params(**kw), seed=2, want_level0=True)
    ctx.profile(True)
    l0, out, oa = _run(ctx, imgs, kw, seed=2)
    names = set(ctx.profile_report())
    ctx.profile(False)
    assert "ef_out0" not in names
    assert np.array_equal(l0, ref["level0"])
    assert np.array_equal(out, ref["out"])


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
def test_fused_enfuse_host_buffers(ctx, orc, dt):
    h, w, K = 45, 70, 3
    imgs = _stack(dt, h, w, K, seed=12, S=4)
    ref = orc.enfuse(imgs, None, orc.params(**W_ALL), seed=6)
    import enbgpu
    out, oa = ctx.enfuse(imgs, params=enbgpu.enfuse_params(**W_ALL), seed=6)
    assert np.array_equal(out, ref["out"])
    assert np.array_equal(oa, ref["alpha"])


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("w,h,K,wrap,chans", [(65, 33, 2, False, 3), (64, 16, 5, False, 3), (129, 31, 16, False, 3),
                                              (130, 47, 3, True, 3), (131, 49, 4, True, 4), (63, 95, 9, True, 3),
                                              (257, 63, 3, False, 4), (66, 34, 4, True, 1)])
def test_level_tiles_at_their_edges(ctx, dtype, w, h, K, wrap, chans):
    """The level passes at tile edges, odd and periodic levels, one and four channels, many exposures, and output
    rows that allow paired stores or not, against the per-operation passes: every sample of level 0 and the pixels."""
    rng = np.random.default_rng(w * 1000 + h)
    maxv = np.iinfo(dtype).max
    shape = (h, w) if chans == 1 else (h, w, chans)
    imgs = [rng.integers(0, maxv + 1, shape).astype(dtype) for _ in range(K)]
    if chans == 4:
        for im in imgs:
            im[..., 3] = maxv
    alphas = [np.where(rng.random((h, w)) < 0.9, 255, 0).astype(np.uint8) for _ in range(K)]
    import enbgpu
    prm = enbgpu.enfuse_params(saturation_weight=0.2, contrast_weight=0.5)
    got = []
    for plain in (False, True):
        l0 = np.zeros((h, w, min(chans, 3)), np.int32)
        out, alpha = ctx.enfuse(imgs, alphas, params=prm, wrap=wrap, seed=9, level0=l0, plain=plain)
        got.append((l0, out, alpha))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    # device rows one sample off the pair's alignment
    pad = [torch.from_numpy(np.pad(im, [(0, 0), (0, 1)] + [(0, 0)] * (im.ndim - 2))).cuda()[:, :w] for im in imgs]
    out = torch.from_numpy(np.zeros_like(np.pad(imgs[0], [(0, 0), (0, 1)] + [(0, 0)] * (imgs[0].ndim - 2)))).cuda()[:, :w]
    ctx.enfuse(pad, [torch.from_numpy(a).cuda() for a in alphas], params=prm, wrap=wrap, seed=9, out=out)
    ctx.synchronize()
    assert np.array_equal(out.cpu().numpy(), got[0][1])


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("con,ent", [(0, 0), (5, 0), (3, 0), (0, 5), (0, 3), (5, 5), (3, 5), (5, 3), (3, 3)])
@pytest.mark.parametrize("chans", [3, 4])
def test_weight_kernels_against_single_operations(ctx, dtype, con, ent, chans):
    """The RGB weight kernels (points, 2x2 quads) against the per-image kernel behind the plain passes: few distinct
    values (long runs of equal keys), random and flat samples, saturated and black ones, alpha holes and edges in
    planes and in the 4th component, images smaller than a tile, ragged rows; level 0 and pixels bit for bit."""
    import enbgpu
    rng = np.random.default_rng(100 * con + 10 * ent + chans)
    maxv = np.iinfo(dtype).max
    prm = enbgpu.enfuse_params(saturation_weight=0.2, contrast_weight=0.5 if con else 0.0, entropy_weight=0.3 if ent else 0.0,
                               contrast_window_size=con or 5, entropy_window_size=ent or 3)
    for (w, h, K) in [(9, 11, 2), (33, 31, 3), (67, 64, 4), (130, 35, 2)]:
        shape = (h, w, chans)
        kinds = [rng.integers(0, maxv + 1, shape), rng.integers(0, 3, shape) * (maxv // 2), rng.integers(0, 25, shape),
                 np.full(shape, maxv), maxv - rng.integers(0, 300, shape) % (maxv // 4)]
        imgs = [np.ascontiguousarray(kinds[(i + w) % len(kinds)].astype(dtype)) for i in range(K)]
        for im in imgs:
            im[h // 2:, : w // 3] = 0
        for alpha in ("none", "planes") if chans == 3 else ("channel", "planes"):
            alphas = None
            if chans == 4:
                for im in imgs:
                    im[..., 3] = np.where(rng.random((h, w)) < (0.9 if alpha == "channel" else 2.0), maxv, maxv // 3)
                    im[: h // 4, w // 2:, 3] = 0 if alpha == "channel" else maxv
            if alpha == "planes":
                alphas = [np.where((np.add.outer(np.arange(h), 2 * np.arange(w)) > 12) & (rng.random((h, w)) < 0.97), 255, 0)
                          .astype(np.uint8) for _ in range(K)]
            got = []
            for plain in (False, True):
                l0 = np.zeros((h, w, 3), np.int32)
                out, oa = ctx.enfuse(imgs, alphas, params=prm, seed=9, level0=l0, plain=plain)
                got.append((l0, out, oa))
            for a, b in zip(*got):
                assert np.array_equal(a, b), (w, h, alpha)


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("samples", [(3, 4, 3), (4, 3, 4)])
@pytest.mark.parametrize("windows", [0, 5])
def test_exposures_of_rgb_and_rgba_mixed(ctx, dt, samples, windows):
    """A stack of RGB and RGBA images, all with alpha planes: the same result as the stack of their RGB samples, whose
    exposures all have one layout (bit for bit, as every pass is in integers)."""
    h, w = 45, 70
    imgs = _stack(dt, h, w, len(samples), seed=61)
    rng = np.random.default_rng(61)
    alphas = [np.where(rng.random((h, w)) < 0.9, 255, 0).astype(np.uint8) for _ in samples]
    kw = W_ALL if windows else dict(exposure_weight=1.0, saturation_weight=0.2)
    l0, out, oa = _run(ctx, imgs, kw, seed=3, alphas=[_dev(a) for a in alphas])
    mixed = [x if s == 3 else np.concatenate([x, rng.integers(0, 256, (h, w, 1)).astype(dt)], axis=2)
             for x, s in zip(imgs, samples)]
    l0m, outm, oam = _run(ctx, mixed, kw, seed=3, alphas=[_dev(a) for a in alphas])
    assert np.array_equal(l0m, l0)
    assert np.array_equal(outm[..., :3], out)
    assert np.array_equal(oam, oa)


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("window", [3, 5])
@pytest.mark.parametrize("holes", [0.02, 0.3, 0.9])
def test_entropy_windows_with_transparent_taps(ctx, orc, dt, window, holes):
    """Entropy of windows with transparent taps, whose keys sort as the largest sample: few distinct samples with the
    type's maximum among them, from a few holes to a few opaque pixels, against the oracle bit for bit."""
    h, w, K = 39, 71, 2
    rng = np.random.default_rng(window)
    top = np.iinfo(dt).max
    imgs = [rng.choice(np.array([0, 1, top // 2, top - 1, top], dt), (h, w, 3)) for _ in range(K)]
    alphas = [np.where(rng.random((h, w)) < holes, 0, 255).astype(np.uint8) for _ in range(K)]
    kw = dict(exposure_weight=0.2, entropy_weight=1.0, entropy_window_size=window, contrast_weight=0.3, contrast_window_size=5)
    ref = orc.enfuse(imgs, alphas, orc.params(**kw), seed=9, want_level0=True)
    l0, out, oa = _run(ctx, imgs, kw, seed=9, alphas=[_dev(a) for a in alphas])
    assert np.array_equal(l0, ref["level0"])
    assert np.array_equal(oa, ref["alpha"])
    assert np.array_equal(out, ref["out"])
