"""The exact elimination search (umi_gb300/csrc/full_me_elim.cu) against the
CPU oracle, bit for bit, where it can go wrong: ranges at the edges of its row
passes (nd = 2r + 1 below, at and above 33 and 66 rows, one and two threads
per column), runs of several blocks and ragged last runs, frames whose rows
are not 4- or 16-byte aligned, content at every cell scale (nearly flat,
full contrast), blocks it has to search exhaustively beside blocks it does
not, ties, and the largest SADs.  Integer results: no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _t(a, dev, shift=0):
    """The array on the GPU, its first byte `shift` past a 256-byte boundary."""
    import torch
    flat = torch.zeros(a.size + 256, dtype=torch.uint8, device=dev)
    v = flat[shift:shift + a.size].view(a.shape)
    v.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return v


def _scene(g, h, w, contrast):
    """Blurred noise (moved by (3, -2) with a little noise), a noise corner and a flat corner."""
    from umi_gb300.workloads import gaussian_blur
    a = gaussian_blur(g.normal(0, 1, (h + 8, w + 8)).astype(np.float32), 1.5)
    a = a / a.std()
    x = np.clip(128 + contrast * a, 0, 255)
    ref, cur = x[4:4 + h, 4:4 + w].copy(), x[7:7 + h, 2:2 + w].copy()
    cur += g.normal(0, 1, cur.shape)
    cur[:h // 3, :w // 3] = g.integers(0, 256, cur[:h // 3, :w // 3].shape)
    ref[-(h // 3):, -(w // 3):] = 90
    return np.clip(cur, 0, 255).astype(np.uint8), np.clip(ref, 0, 255).astype(np.uint8)


@pytest.mark.parametrize("h,w,r", [(80, 208, 8), (64, 176, 15), (64, 320, 16), (80, 144, 17), (64, 160, 24),
                                   (64, 96, 33), (48, 80, 48), (48, 96, 63), (33, 71, 7), (50, 203, 16), (70, 101, 32),
                                   (40, 90, 64), (20, 18, 3)])
def test_elim_matches_oracle(umi, orc, dev, h, w, r):
    g = np.random.default_rng(h * 1000 + w + r)
    for contrast, shift in ((2.0, 0), (12.0, 1), (90.0, 4)):
        cur, ref = _scene(g, h, w, contrast)
        got = umi.full_me_u8(_t(cur, dev, shift), _t(ref, dev, shift), 16, r).cpu().numpy()
        assert np.array_equal(got, orc.full_me_u8(cur, ref, 16, r)), contrast


@pytest.mark.parametrize("r", [9, 16, 40])
def test_elim_ties_and_extremes(umi, orc, dev, r):
    import torch
    full = lambda v, h=96, w=160: torch.full((h, w), v, dtype=torch.uint8, device=dev)  # noqa: E731
    for a, b in ((7, 9), (0, 255), (255, 255)):
        got = umi.full_me_u8(full(a), full(b), 16, r).cpu().numpy()
        assert np.all(got[:, 2] == 256 * abs(a - b)) and np.all(got[:, :2] == -r)
    # period 4 in both directions: many exact matches, the first in raster order wins
    y, x = np.mgrid[:96, :160]
    p = (40 * (y % 4) + 15 * (x % 4)).astype(np.uint8)
    assert np.array_equal(umi.full_me_u8(_t(p, dev), _t(p, dev), 16, r).cpu().numpy(), orc.full_me_u8(p, p, 16, r))


@pytest.mark.parametrize("h,w,r", [(112, 144, 16), (96, 131, 21)])
def test_elim_list_and_centers(umi, orc, dev, h, w, r):
    import torch
    g = np.random.default_rng(r)
    cur, ref = _scene(g, h, w, 12.0)
    nbx, n = w // 16, (h // 16) * (w // 16)
    centers = g.integers(-13, 14, (n, 2)).astype(np.int32)
    blocks = g.permutation(n).astype(np.int32)
    count = n // 2
    out = torch.full((n, 3), -9, dtype=torch.int32, device=dev)
    umi.full_me_u8_list(_t(cur, dev), _t(ref, dev), torch.from_numpy(blocks).to(dev),
                        torch.tensor([count], dtype=torch.int32, device=dev), out, 16, r,
                        centers=torch.from_numpy(centers).to(dev))
    got = out.cpu().numpy()
    assert np.all(got[blocks[count:]] == -9)
    for i in blocks[:count].tolist()[:10]:
        by, bx = divmod(i, nbx)
        best = min((orc.block_sad_u8(cur, ref, 16, by, bx, dy, dx), dy, dx)
                   for dy in range(centers[i, 0] - r, centers[i, 0] + r + 1)
                   for dx in range(centers[i, 1] - r, centers[i, 1] + r + 1))
        assert tuple(got[i]) == (best[1], best[2], best[0]), i


@pytest.mark.parametrize("r", [33, 34, 64])
@pytest.mark.parametrize("n", [1, 150, 153, 400])
def test_list_of_any_length(umi, orc, dev, r, n):
    """Lists with wide windows: up to one block per SM every thread of a CTA
    serves one block, beyond that two teams share the CTA; the length is read on
    the GPU.  Blocks that are not listed keep what they held."""
    import torch
    g = np.random.default_rng(r + n)
    h, w = 16 * 21, 16 * 20
    cur, ref = _scene(g, h, w, 40)
    nblk = (h // 16) * (w // 16)
    blocks = g.permutation(nblk)[:n].astype(np.int32)
    want = orc.full_me_u8(cur, ref, 16, r, blocks=blocks)
    padded = np.full(nblk, -5, np.int32)
    padded[:n] = blocks
    mv = torch.full((nblk, 3), -99, dtype=torch.int32, device=dev)
    umi.full_me_u8_list(_t(cur, dev), _t(ref, dev), torch.from_numpy(padded).to(dev),
                        torch.tensor([n], dtype=torch.int32, device=dev), mv, 16, r)
    got = mv.cpu().numpy()
    assert np.array_equal(got[blocks], want)
    rest = np.setdiff1d(np.arange(nblk), blocks)
    assert (got[rest] == -99).all()
