"""Integral image and box sum with every workspace size that was ever named for
them: two arrays of column sums (uint16, per band of 8 rows and per group of 128)
serve any frame; wider frames are named more.  Nothing outside the workspace is
written, less is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _two_arrays(h, w):
    al = lambda b: (b + 255) // 256 * 256  # noqa: E731
    groups, wpad = -(-(-(-h // 8)) // 16), -(-w // 8) * 8
    return al(groups * 16 * wpad * 2) + al(groups * wpad * 2)


@pytest.mark.parametrize("h,w", [(1, 1), (9, 11), (130, 257), (300, 1923), (65, 2048), (33, 2049), (140, 2500), (17, 5000),
                                 (130, 4096), (1000, 3840), (8, 8200), (129, 6145)])
@pytest.mark.parametrize("off", [0, 1])
def test_iimg_workspaces(umi, dev, h, w, off):
    import torch
    from umi_gb300 import apps
    x = np.random.default_rng(h + w).integers(0, 256, (h, w), dtype=np.uint8)
    buf = torch.full((h * w + 64,), 255, dtype=torch.uint8, device=dev)
    inp = buf[off:off + h * w].view(h, w)
    inp.copy_(torch.from_numpy(x))
    want = x.astype(np.int64).cumsum(0).cumsum(1)
    least, named = _two_arrays(h, w), umi.iimg_workspace_bytes(h, w)
    assert least <= named and (w > 2048 or least == named)
    for nb in (least, named):
        ws = torch.full((nb + 256,), 0xA5, dtype=torch.uint8, device=dev)
        flat = torch.full((h * w + 64,), -7, dtype=torch.int32, device=dev)
        out = flat[4 * off:4 * off + h * w].view(h, w)
        umi.iimg_u8_i32(inp, out=out, workspace=ws[:nb])
        assert np.array_equal(out.cpu().numpy(), want)
        assert (ws[nb:] == 0xA5).all() and (flat[:4 * off] == -7).all() and (flat[4 * off + h * w:] == -7).all()
        box = apps.box_sum(inp, 2, workspace=ws[:nb])
        assert np.array_equal(box.cpu().numpy(), apps.box_sum(inp, 2).cpu().numpy())
    with pytest.raises(umi.UmiError):
        umi.iimg_u8_i32(inp, workspace=torch.empty(least - 256, dtype=torch.uint8, device=dev))
