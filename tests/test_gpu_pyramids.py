"""Whole pyramids (build, blend, collapse) against the CPU oracle level by
level, bit for bit: the last reduces in one launch, level 0 of a Laplacian
pyramid straight from the pixels, the chained expands and the blend of all
levels, at shapes on both sides of each of these rules (long thin levels, more
levels than one launch takes, odd sizes, periodic seams).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(200, 130, 6), (257, 300, 8), (64, 64, 6), (65, 70, 8), (1030, 9, 4), (2101, 17, 5), (9, 455, 4), (333, 21, 1), (65, 33, 2)]


def _chain(orc, level0, alpha, levels, bits, wrap):
    out, a = [level0], alpha
    for _ in range(1, levels):
        if a is None:
            out.append(orc.reduce(out[-1], None, bits, wrap))
        else:
            r, a = orc.reduce(out[-1], a, bits, wrap)
            out.append(r)
    return out


def _laplacian(orc, g, bits, wrap):
    return [orc.expand(g[l + 1], g[l], False, bits, wrap) for l in range(len(g) - 1)] + [g[-1]]


def _same(pyr, ref, what):
    for l, r in enumerate(ref):
        got = np.transpose(pyr.read(l), (1, 2, 0)).astype(np.int32)
        assert np.array_equal(got, r), (what, l, r.shape)


def _pixels(rng, h, w, stride, dtype, pad):
    """Device pixels with the given samples a pixel in rows of w + pad pixels, and their colour samples."""
    a = rng.integers(0, np.iinfo(dtype).max + 1, size=(h, w + pad, stride)).astype(dtype)
    t = torch.from_numpy(a.view(np.int16) if dtype == np.uint16 else a).cuda()
    if dtype == np.uint16:
        t = t.view(torch.uint16)
    t = t[:, :w]
    c = 1 if stride == 1 else 3
    return (t[:, :, 0] if c == 1 else t), a[:, :w, :c].astype(np.int32)


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("wrap", [False, True])
@pytest.mark.parametrize("stride,pad", [(3, 0), (4, 0), (1, 0), (3, 1)])
def test_pyramids(ctx, orc, dtype, wrap, stride, pad):
    import enbgpu
    u8 = dtype == np.uint8
    bits, frac, mfrac = (16, 7, 7) if u8 else (32, 7, 15)
    white_value = 255 << mfrac
    rng = np.random.default_rng(31 + stride)
    for (w, h, levels) in SHAPES:
        pyr, ref = [], []
        for _ in range(2):
            dev, px = _pixels(rng, h, w, stride, dtype, pad)
            a = (rng.random((h, w)) < 0.8).astype(np.uint8) * 255
            g = _chain(orc, px << frac, a, levels, bits, wrap)
            gp = ctx.gaussian_pyramid(dev, levels, alpha=torch.from_numpy(a).cuda(), wrap=wrap)
            _same(gp, g, ("gaussian", w, h))
            lp = ctx.laplacian_pyramid(dev, levels, alpha=torch.from_numpy(a).cuda(), wrap=wrap)
            lref = _laplacian(orc, g, bits, wrap)
            _same(lp, lref, ("laplacian", w, h))
            bare = ctx.laplacian_pyramid(dev, levels, wrap=wrap)
            _same(bare, _laplacian(orc, _chain(orc, px << frac, None, levels, bits, wrap), bits, wrap), ("bare", w, h))
            pyr.append(lp)
            ref.append(lref)
        mask = np.zeros((h, w), np.uint8)
        mask[:, w // 2:] = 255
        mask[rng.random((h, w)) < 0.05] = 128
        mdev = torch.from_numpy(mask).cuda()
        gp = ctx.gaussian_pyramid(mdev, levels, wrap=wrap, frac_bits=mfrac,
                                  dtype=enbgpu.ENB_I16 if u8 else enbgpu.ENB_I32)
        gm = _chain(orc, mask[..., None].astype(np.int32) << mfrac, None, levels, bits, wrap)
        _same(gp, gm, ("mask", w, h))
        ctx.blend_pyramids(gp, pyr[0], pyr[1], white_value)
        out = [orc.blend(gm[l], ref[0][l], ref[1][l], white_value, bits) for l in range(levels)]
        _same(pyr[1], out, ("blend", w, h))
        ctx.collapse_pyramid(pyr[1], wrap=wrap)
        for l in range(levels - 2, -1, -1):
            out[l] = orc.expand(out[l + 1], out[l], True, bits, wrap)
        _same(pyr[1], out, ("collapse", w, h))


# The fused drivers' small levels: long thin ones, levels of exactly 304 tiles
# of 64x16 and of a row of tiles more, level areas around 4096 pixels.
FUSED = [(455, 11), (13, 700), (2048, 608), (2048, 610), (128, 128), (130, 127), (4100, 33)]


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("wrap", [False, True])
@pytest.mark.parametrize("stride", [1, 3, 4])
def test_fused_small_levels(ctx, dtype, wrap, stride):
    rng = np.random.default_rng(77 + stride)
    for (w, h) in FUSED:
        imgs = [_pixels(rng, h, w, stride, dtype, 0)[0] for _ in range(3)]
        alphas = [torch.from_numpy((rng.random((h, w)) < 0.9).astype(np.uint8) * 255).cuda() for _ in range(3)]
        mask = torch.from_numpy((rng.random((h, w)) < 0.5).astype(np.uint8) * 255).cuda()
        got, want = (ctx.enblend(imgs[0], imgs[1], mask, alphas[0], alphas[1], wrap=wrap, seed=5, plain=plain)
                     for plain in (False, True))
        assert torch.equal(got[1], want[1]) and np.array_equal(got[0].cpu().numpy(), want[0].cpu().numpy()), (w, h)
        for a in (None, alphas):
            got, want = (ctx.enfuse(imgs, a, wrap=wrap, seed=5, plain=plain) for plain in (False, True))
            assert torch.equal(got[1], want[1]) and np.array_equal(got[0].cpu().numpy(), want[0].cpu().numpy()), (w, h)
