"""The Gaussian's kept weights on the CPU: sigma and radius may be numpy scalars,
0-d arrays or (radius) tensors, and one that its owner changes between calls is
read again."""
import numpy as np
import pytest


@pytest.mark.parametrize("kind", [np.array, "tensor", np.int64, float, str])
def test_radius_of_any_kind(umi, kind):
    import torch
    from umi_gb300 import apps
    kind = torch.tensor if kind == "tensor" else kind
    for r in (1, 2):
        assert np.array_equal(apps.gaussian_kernel(1.5, kind(r)), apps.gaussian_kernel(1.5, r))


def test_sigma_of_any_kind(umi):
    from umi_gb300 import apps
    want = apps.gaussian_kernel(1.5)
    for sigma in (np.array(1.5), np.float64(1.5), np.float32(1.5)):
        assert np.allclose(apps.gaussian_kernel(sigma), want, rtol=1e-6)


def test_changed_arguments_are_read_again(umi):
    import torch
    from umi_gb300 import apps
    for r in (torch.tensor(1), np.array(1)):
        assert apps.gaussian_kernel(1.5, r).size == 3
        r += 2
        assert apps.gaussian_kernel(1.5, r).size == 7
    s = np.array(1.0)
    a = apps.gaussian_kernel(s, 3)
    s += 1.0
    assert not np.array_equal(a, apps.gaussian_kernel(s, 3))
