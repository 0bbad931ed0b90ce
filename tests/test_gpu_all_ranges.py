"""Every range of the operators whose shared memory grows with it, at small
frames: each launches and equals the oracle or the plain evaluation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(dev, h, w, seed):
    import torch
    g = np.random.default_rng(seed)
    ref = g.integers(0, 256, (h, w), dtype=np.uint8)
    cur = np.roll(ref, (1, -2), (0, 1))
    cur[:, w // 2:] = g.integers(0, 256, cur[:, w // 2:].shape)
    return cur, ref, torch.from_numpy(cur).to(dev), torch.from_numpy(ref).to(dev)


@pytest.mark.parametrize("block,h,w", [(16, 32, 80), (16, 33, 101), (8, 16, 64), (8, 64, 200), (8, 240, 320)])
def test_search_ranges(umi, orc, dev, block, h, w):
    cur, ref, c, r = _pair(dev, h, w, block + w)
    for rad in range(1, 65):
        if h * w > 20000 and rad % 5:
            continue
        assert np.array_equal(umi.full_me_u8(c, r, block, rad).cpu().numpy(), orc.full_me_u8(cur, ref, block, rad)), rad


@pytest.mark.parametrize("block", [8, 16])
def test_list_and_volume_ranges(umi, orc, dev, block):
    import torch
    cur, ref, c, r = _pair(dev, 32, 80, block)
    n = (32 // block) * (80 // block)
    blocks = torch.arange(n, dtype=torch.int32, device=dev)
    count = torch.tensor([n], dtype=torch.int32, device=dev)
    out = torch.empty((n, 3), dtype=torch.int32, device=dev)
    for rad in range(1, 65):
        want = orc.full_me_u8(cur, ref, block, rad)
        umi.full_me_u8_list(c, r, blocks, count, out, block, rad)
        assert np.array_equal(out.cpu().numpy(), want), rad
        vol = umi.full_me_sad_u8(c, r, block, rad).reshape(n, -1).min(1).values.cpu().numpy()
        assert np.array_equal(vol, want[:, 2]), rad
        zero = torch.zeros((n, 2), dtype=torch.int32, device=dev)
        assert np.array_equal(umi.full_me_u8(c, r, block, rad, centers=zero).cpu().numpy(), want), rad


def test_window_and_blur_ranges(umi, dev):
    import torch
    from umi_gb300 import apps
    x = torch.randint(-999, 999, (40, 150), dtype=torch.int32, device=dev)
    f = torch.rand(40, 150, device=dev)
    for rad in range(0, 48):
        p = torch.nn.functional.pad(x[None, None].double(), (rad,) * 4, mode="replicate")
        want = torch.nn.functional.max_pool2d(p, 2 * rad + 1, 1)[0, 0].int()
        assert torch.equal(apps.dilate(x, rad), want), rad
        k = torch.from_numpy(apps.gaussian_kernel(2.0, rad)).to(dev).double()
        q = torch.nn.functional.pad(f[None, None].double(), (rad,) * 4, mode="replicate")
        q = torch.nn.functional.conv2d(torch.nn.functional.conv2d(q, k.view(1, 1, 1, -1)), k.view(1, 1, -1, 1))[0, 0]
        assert torch.allclose(apps.gaussian(f, 2.0, rad).double(), q, rtol=0, atol=1e-5), rad  # sums of weights 1, at most 190 FMAs
