"""Full search of 8x8 blocks at their own places (strips of up to 32 blocks, a
lane a block) against the oracle: ranges whose last group of displacements or
of rows is whole and not, strips of every width class, any row alignment."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _t(a, dev, shift):
    """A CUDA tensor with a's bytes, its first byte `shift` past a 256-byte boundary."""
    import torch
    flat = torch.zeros(a.size + 256, dtype=torch.uint8, device=dev)
    t = flat[shift:shift + a.size].view(a.shape)
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t


# few blocks (the general kernel for wide ranges), many (strips with split
# warps) and enough for whole strips of 32
@pytest.mark.parametrize("h,w,r", [(8, 8, 1), (9, 15, 2), (24, 264, 3), (40, 256, 4), (16, 72, 7), (24, 135, 8),
                                   (40, 531, 13), (24, 50, 63), (160, 531, 13), (200, 264, 16), (136, 267, 17),
                                   (160, 201, 31), (97, 801, 32), (184, 182, 63), (184, 180, 64), (717, 1278, 16),
                                   (720, 1030, 7), (344, 1801, 33)])
@pytest.mark.parametrize("shift", [0, 3])
def test_full_me_8_matches_oracle(umi, orc, dev, h, w, r, shift):
    g = np.random.default_rng(h * 1000 + w + r)
    ref = g.integers(0, 256, (h, w), dtype=np.uint8)
    dy, dx = min(r, h - 1), min(r, w - 1) // 2
    moved = np.roll(ref, (dy, -dx), (0, 1))
    noisy = np.clip(moved.astype(int) + g.integers(-20, 21, (h, w)), 0, 255).astype(np.uint8)
    few = g.integers(0, 3, (h, w), dtype=np.uint8)  # many equal sums: the first in raster order
    extreme = np.where(g.random((h, w)) < 0.5, 0, 255).astype(np.uint8)
    scenes = ((moved, ref), (noisy, ref), (few, few[::-1].copy()), (extreme, 255 - extreme))
    for c, f in scenes[:2] if h * w > 200000 else scenes:
        got = umi.full_me_u8(_t(c, dev, shift), _t(f, dev, shift), 8, r).cpu().numpy()
        assert np.array_equal(got, orc.full_me_u8(c, f, 8, r))
