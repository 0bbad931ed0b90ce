"""Integral image: segments of 1024 columns (frames wider than 2048), rows and
outputs at any alignment (three-word loads, stores through shared memory,
32-, 16- and 4-byte stores), bands cut by the last row.  Bit-exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,off,ooff", [(130, 2056, 0, 0), (33, 2049, 1, 1), (300, 3075, 3, 2), (17, 5000, 2, 4),
                                          (140, 2500, 5, 1), (8, 1024, 1, 0), (9, 11, 2, 3), (1, 4099, 0, 0),
                                          (65, 257, 3, 0), (1000, 3840, 8, 4)])
def test_iimg_segments(umi, dev, h, w, off, ooff):
    import torch
    x = np.random.default_rng(h + w).integers(0, 256, (h, w), dtype=np.uint8)
    buf = torch.full((h * w + 64,), 255, dtype=torch.uint8, device=dev)
    inp = buf[off:off + h * w].view(h, w)
    inp.copy_(torch.from_numpy(x))
    obuf = torch.full((h * w + 64,), -7, dtype=torch.int32, device=dev)
    out = obuf[ooff:ooff + h * w].view(h, w)
    ws = torch.full((umi.iimg_workspace_bytes(h, w),), 0xA5, dtype=torch.uint8, device=dev)
    umi.iimg_u8_i32(inp, out=out, workspace=ws)
    assert np.array_equal(out.cpu().numpy(), x.astype(np.int64).cumsum(0).cumsum(1))
    assert (obuf[:ooff] == -7).all().item() and (obuf[ooff + h * w:] == -7).all().item()
