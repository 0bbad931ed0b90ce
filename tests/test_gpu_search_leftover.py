"""8x8 searches whose leftover columns (beyond a multiple of 32) are taken in groups
of rows that end below the window's staged rows: lists, centres and small
frames, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [19, 25, 35, 40, 45, 53, 58])
def test_leftover_columns(umi, orc, dev, r):
    import torch
    h, w = 24, 168
    g = np.random.default_rng(r)
    ref = g.integers(0, 256, (h, w), dtype=np.uint8)
    cur = np.roll(ref, (2, -3), (0, 1))
    c, f = torch.from_numpy(cur).to(dev), torch.from_numpy(ref).to(dev)
    n = (h // 8) * (w // 8)
    want = orc.full_me_u8(cur, ref, 8, r)
    assert np.array_equal(umi.full_me_u8(c, f, 8, r).cpu().numpy(), want)
    zero = torch.zeros((n, 2), dtype=torch.int32, device=dev)
    assert np.array_equal(umi.full_me_u8(c, f, 8, r, centers=zero).cpu().numpy(), want)
    out = torch.empty((n, 3), dtype=torch.int32, device=dev)
    umi.full_me_u8_list(c, f, torch.arange(n, dtype=torch.int32, device=dev),
                        torch.tensor([n], dtype=torch.int32, device=dev), out, 8, r)
    assert np.array_equal(out.cpu().numpy(), want)
