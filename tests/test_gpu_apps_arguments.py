"""Radii of the window applications as numpy scalars, 0-d arrays and tensors: the
results of the plain number, also after the array or tensor has been changed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["census", "dilate", "erode", "box_sum"])
def test_radius(umi, dev, name):
    import torch
    from umi_gb300 import apps
    f = getattr(apps, name)
    dt = torch.uint8 if name == "box_sum" else torch.int32
    x = torch.randint(0, 256, (37, 150), device=dev).to(dt)
    for kind in (np.array, np.int64, torch.tensor):
        r = kind(1)
        assert torch.equal(f(x, r), f(x, 1))
        r += 1
        assert torch.equal(f(x, r), f(x, 2))
    with pytest.raises(TypeError):
        f(x, 1.5)
