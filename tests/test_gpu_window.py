"""Window operators through umi_launch (umi_gb300/csrc/window_ops.cuh) against
a direct numpy evaluation of the descriptor: images of another size than P,
offsets that leave the image on every side, PAD / clamp per dimension, strides
(negative ones too), windows wider than a 16-byte piece and taller than a
thread's rows, ragged right and bottom edges, unaligned outputs with a row
stride of their own, and the plans that stay with the generic kernel (several
accumulation blocks, a batch dimension).  Integers exactly; the float sums
within 1e-5 of the sum of |x w| (at most 13 * 13 FMAs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PAD, WRAP = 0, 1


def _read(img, y, x, mode, pad):
    h, w = img.shape
    cy, cx = np.clip(y, 0, h - 1), np.clip(x, 0, w - 1)
    out = ((cy != y) & (mode[0] == PAD)) | ((cx != x) & (mode[1] == PAD))
    return np.where(out, pad, img[cy, cx])


def _case(umi, dev, strat, g, P, img, oy, ox, ky, kx, sy, sx, mode, block=(0, 0), ostride=0, oshift=0):
    import torch
    h, w = P
    isf = strat == umi.STRATEGY_WEIGHTED_SUM_F32
    weighted = strat in (umi.STRATEGY_WEIGHTED_SUM_F32, umi.STRATEGY_WEIGHTED_SUM_I32)
    pad = 7.5 if isf else -3
    yy, xx = np.mgrid[:h, :w]
    wts = g.normal(size=(ky, kx)).astype(np.float32) if isf else g.integers(-4, 5, (ky, kx)).astype(np.int32)
    vals = [(ay, ax, _read(img, yy + ay * sy + oy, xx + ax * sx + ox, mode, pad)) for ay in range(ky) for ax in range(kx)]
    c0 = {umi.STRATEGY_NEIGHBOUR_SUM_I32: [5, 3], umi.STRATEGY_MAX_I32: [-2 ** 31], umi.STRATEGY_MIN_I32: [2 ** 31 - 1],
          umi.STRATEGY_CENSUS_I32: None}.get(strat, [2])
    if strat == umi.STRATEGY_CENSUS_I32:
        centre = _read(img, yy + 1, xx - 1, mode, pad)
        want = np.zeros((h, w), np.uint32)
        for _, _, v in vals:
            want = (want << np.uint32(1)) | (v < centre).astype(np.uint32)
        want = want.view(np.int32)
    elif strat == umi.STRATEGY_NEIGHBOUR_SUM_I32:
        want = ((5 + sum(v.astype(np.int64) for _, _, v in vals)) * 3).astype(np.int32)
    elif weighted:
        want = 2 + sum(v.astype(np.float64 if isf else np.int64) * wts[ay, ax] for ay, ax, v in vals)
    else:
        want = np.stack([v for _, _, v in vals])
        want = want.max(0) if strat == umi.STRATEGY_MAX_I32 else want.min(0)
    view = [(), (), (2, oy, sy), (3, ox, sx)]
    phys = [(1, PAD), (1, PAD), (img.shape[0], mode[0]), (img.shape[1], mode[1])]
    mems = [dict(p_view=[(), (), (2, 0, 1), (3, 0, 1)], a_view=view, phys=phys, stage=1)]
    ins, pads = [torch.from_numpy(img).to(dev)], [pad]
    if strat == umi.STRATEGY_CENSUS_I32:
        mems.insert(0, dict(p_view=[(), (), (2, 1, 1), (3, -1, 1)], phys=phys, stage=0))
        ins, pads = ins * 2, pads * 2
    if weighted:
        mems.append(dict(p_view=[(), (), (), ()], a_view=[(), (), (2, 0, 1), (3, 0, 1)],
                         phys=[(1, PAD), (1, PAD), (ky, PAD), (kx, PAD)], stage=1))
        ins, pads = ins + [torch.from_numpy(wts).to(dev)], pads + [0]
    os_ = max(ostride, w)
    flat = torch.full((oshift + h * os_,), 77, dtype=torch.float32 if isf else torch.int32, device=dev)
    out = flat[oshift:oshift + h * os_].view(h, os_)
    mems.append(dict(p_view=[(), (), (2, 0, 1), (3, 0, 1)], phys=[(), (), (h, PAD), (os_, PAD)], stage=2, out=True))
    d = umi.make_desc(p=[(1, 1, 1, 1), (1, 1, 1, 1), (h, 8, 1, 1), (w, 32, 32, 1)],
                      a=[(1, 1), (1, 1), (ky, block[0] or ky), (kx, block[1] or kx)], mems=mems)
    umi.launch(d, strat, ins, [out], pads=pads, consts=c0)
    got = out.cpu().numpy()
    assert (got[:, w:] == 77).all() and (flat[:oshift] == 77).all().item()
    if isf:
        scale = 2 + sum(np.abs(v * wts[ay, ax]) for ay, ax, v in vals)
        assert (np.abs(got[:, :w] - want) <= 1e-5 * scale).all()
    else:
        assert np.array_equal(got[:, :w], want)


@pytest.mark.parametrize("k", range(10))
@pytest.mark.parametrize("name", ["CENSUS_I32", "MAX_I32", "MIN_I32", "NEIGHBOUR_SUM_I32", "WEIGHTED_SUM_I32",
                                  "WEIGHTED_SUM_F32"])
def test_window_forms(umi, dev, name, k):
    strat = getattr(umi, "STRATEGY_" + name)
    g = np.random.default_rng(100 * k + len(name))
    (P, isz, off, win, stride, mode, more) = [
        ((40, 200), (40, 200), (-2, -2), (5, 5), (1, 1), (WRAP, WRAP), {}),
        ((33, 129), (33, 129), (-1, -1), (3, 3), (1, 1), (PAD, PAD), {}),
        ((1, 1), (1, 1), (-3, -4), (7, 9), (1, 1), (PAD, WRAP), {}),
        ((64, 130), (50, 90), (4, 7), (1, 13), (1, 1), (WRAP, PAD), dict(ostride=133, oshift=1)),
        ((70, 127), (70, 127), (-6, 0), (13, 1), (1, 1), (WRAP, WRAP), dict(ostride=128)),
        ((37, 260), (41, 270), (3, 5), (2, 4), (1, 1), (PAD, PAD), {}),
        ((45, 140), (46, 141), (-7, -7), (2, 2), (15, 15), (WRAP, WRAP), {}),
        ((30, 150), (30, 150), (4, 3), (3, 5), (-2, -1), (PAD, WRAP), {}),
        ((26, 70), (26, 70), (-2, -2), (5, 5), (1, 1), (WRAP, WRAP), dict(block=(2, 3))),
        ((9, 300), (200, 40), (150, -300), (4, 6), (0, 3), (WRAP, PAD), {}),
    ][k]
    dt = np.float32 if name.endswith("F32") else np.int32
    img = (g.normal(size=isz) if dt == np.float32 else g.integers(-9, 10, isz)).astype(dt)
    if more.get("block") and name == "CENSUS_I32":
        more = {}  # another order of the bits
    _case(umi, dev, strat, g, P, img, off[0], off[1], win[0], win[1], stride[0], stride[1], mode, **more)


@pytest.mark.parametrize("h,w", [(33, 129), (32, 128), (65, 257), (1, 385), (97, 131)])
def test_window_last_tiles(umi, dev, h, w):
    """Tiles of which the image fills one row or one column: only what their
    outputs use is staged."""
    import torch
    from umi_gb300 import apps
    x = np.random.default_rng(h + w).integers(-1000, 1000, (h, w)).astype(np.int32)
    xd = torch.from_numpy(x).to(dev)
    for r in (1, 3, 6):
        p = np.pad(x, r, mode="edge")
        win = np.stack([p[i:i + h, j:j + w] for i in range(2 * r + 1) for j in range(2 * r + 1)])
        assert np.array_equal(apps.dilate(xd, r).cpu().numpy(), win.max(0))
        assert np.array_equal(apps.erode(xd, r).cpu().numpy(), win.min(0))
    c = np.zeros((h, w), np.uint32)
    p = np.pad(x, 2, mode="edge")
    for i in range(5):
        for j in range(5):
            c = (c << 1) | (p[i:i + h, j:j + w] < x)
    assert np.array_equal(apps.census(xd, 2).cpu().numpy().view(np.uint32), c.astype(np.uint32))
