"""The window operators of umi_gb300/apps.py (census, box sums via the
integral image, separable Gaussian, dilation / erosion: four more members of
the UMI example family on the generic operator) against numpy restatements
of their definitions.  Integer outputs bit-exact; the Gaussian within
rel 1e-5 of an FP64 separable filter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(37, 53), (1, 1), (16, 16), (130, 300), (5, 200)]


def _t(a, dev):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def _windows(x, r, mode):
    """(k*k, h, w) stack of the window elements in row-major order."""
    p = np.pad(x, r, mode=mode) if mode == "edge" else np.pad(x, r, mode="constant")
    h, w = x.shape
    return np.stack([p[dy:dy + h, dx:dx + w] for dy in range(2 * r + 1) for dx in range(2 * r + 1)])


@pytest.mark.parametrize("h,w", SIZES)
@pytest.mark.parametrize("r", [1, 2])
def test_census(umi, dev, h, w, r):
    from umi_gb300 import apps
    x = np.random.default_rng(h * w + r).integers(0, 8, (h, w)).astype(np.int32)  # many ties
    got = apps.census(_t(x, dev), r).cpu().numpy().view(np.uint32)
    want = np.zeros((h, w), np.uint64)
    for win in _windows(x, r, "edge"):
        want = (want << np.uint64(1)) | (win < x).astype(np.uint64)
    assert np.array_equal(got, (want & np.uint64(0xffffffff)).astype(np.uint32))


@pytest.mark.parametrize("h,w", SIZES)
@pytest.mark.parametrize("r", [1, 3])
def test_dilate_erode(umi, dev, h, w, r):
    from umi_gb300 import apps
    x = np.random.default_rng(h + w * 3 + r).integers(-1000, 1000, (h, w)).astype(np.int32)
    win = _windows(x, r, "edge")
    assert np.array_equal(apps.dilate(_t(x, dev), r).cpu().numpy(), win.max(0))
    assert np.array_equal(apps.erode(_t(x, dev), r).cpu().numpy(), win.min(0))


@pytest.mark.parametrize("h,w", SIZES + [(1080, 1920)])
@pytest.mark.parametrize("r", [0, 2, 7])
def test_box_sum(umi, dev, h, w, r):
    from umi_gb300 import apps
    x = np.random.default_rng(h * 7 + w + r).integers(0, 256, (h, w), dtype=np.uint8)
    c = np.pad(x.astype(np.int64), r, mode="constant").cumsum(0).cumsum(1)
    c = np.pad(c, ((1, 0), (1, 0)))
    k = 2 * r + 1
    want = c[k:k + h, k:k + w] - c[0:h, k:k + w] - c[k:k + h, 0:w] + c[0:h, 0:w]
    got = apps.box_sum(_t(x, dev), r).cpu().numpy()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("h,w", SIZES)
@pytest.mark.parametrize("sigma", [0.8, 2.0])
def test_gaussian(umi, dev, h, w, sigma):
    from umi_gb300 import apps
    x = np.random.default_rng(h + w).random((h, w), dtype=np.float32)
    k = apps.gaussian_kernel(sigma).astype(np.float64)
    r = k.size // 2
    p = np.pad(x.astype(np.float64), r, mode="edge")
    hz = sum(k[i] * p[:, i:i + w] for i in range(k.size))          # (h + 2r, w)
    want = sum(k[i] * hz[i:i + h, :] for i in range(k.size))
    got = apps.gaussian(_t(x, dev), sigma).cpu().numpy()
    assert np.max(np.abs(got - want) / np.maximum(np.abs(want), 1e-3)) <= 1e-5


@pytest.mark.parametrize("h,w", [(1, 1), (5, 3), (31, 127), (32, 128), (33, 129), (97, 260), (70, 514)])
@pytest.mark.parametrize("radius", [0, 1, 3, 4, 6, 15, 16])
def test_gaussian_one_launch_equals_two(umi, dev, h, w, radius):
    """The one-launch blur (up to 31 weights) gives the bits of the two window
    sums, also in tmp; overlapping buffers and wider windows take two."""
    import torch
    from umi_gb300 import apps
    g = torch.Generator(device="cpu").manual_seed(h * 1000 + w + radius)
    x = torch.randn(h, w, generator=g)
    x[0, 0], x[h // 2, w // 2], x[h - 1, w - 1] = float("inf"), -0.0, 1e30
    x = x.to(dev)
    wt = torch.from_numpy(apps.gaussian_kernel(2.0, radius)).to(dev)
    across, down = apps._gaussian_plans(h, w, 2 * radius + 1)
    tmp, want = torch.empty_like(x), torch.empty_like(x)
    across((x, wt), (tmp,))
    down((tmp, wt), (want,))
    same = lambda a, b: torch.equal(a.view(torch.int32), b.view(torch.int32))  # noqa: E731
    assert same(apps.gaussian(x, 2.0, radius=radius), want)
    flat = torch.full((2, h * w + 17), -7.0, device=dev)
    o, t = flat[0, 1:1 + h * w].view(h, w), flat[1, 4:4 + h * w].view(h, w)  # out one word past a boundary
    apps.gaussian(x, 2.0, radius=radius, out=o, tmp=t)
    assert same(o, want) and same(t, tmp)
    assert (flat[0, 0] == -7) and (flat[0, 1 + h * w:] == -7).all() and (flat[1, 4 + h * w:] == -7).all()
    y = x.clone()
    apps.gaussian(y, 2.0, radius=radius, out=y)
    assert same(y, want)


@pytest.mark.parametrize("h,w", [(1, 1), (2, 5), (8, 127), (9, 129), (70, 300), (33, 2100)])
@pytest.mark.parametrize("r", [0, 1, 7, 40, 5000])
def test_box_sum_reads_corners_or_j(umi, dev, h, w, r):
    """Corners straight from the integral image, with and without J, equal the
    clipped sums; J's interior is filled, nothing outside the buffers written;
    overlapping buffers take the way through J."""
    import torch
    from umi_gb300 import apps
    x = np.random.default_rng(h * 7 + w + r).integers(0, 256, (h, w), dtype=np.uint8)
    c = np.pad(x.astype(np.int64).cumsum(0).cumsum(1), ((1, 0), (1, 0)))
    y0, y1 = np.maximum(np.arange(h) - r, 0), np.minimum(np.arange(h) + r + 1, h)
    x0, x1 = np.maximum(np.arange(w) - r, 0), np.minimum(np.arange(w) + r + 1, w)
    want = c[y1][:, x1] - c[y1][:, x0] - c[y0][:, x1] + c[y0][:, x0]
    xd = _t(x, dev)
    assert apps._box_direct(xd, r, None, None, None) == (r <= 1 << 20)
    assert np.array_equal(apps.box_sum(xd, r).cpu().numpy(), want)
    flat = torch.full((3, (h + 1) * (w + 1) + 16), -7, dtype=torch.int32, device=dev)
    o, ii, J = flat[0, :h * w].view(h, w), flat[1, :h * w].view(h, w), flat[2, :(h + 1) * (w + 1)].view(h + 1, w + 1)
    J.zero_()
    assert apps._box_direct(xd, r, o, J, ii) and not apps._box_direct(xd, r, ii, J, ii)
    got = apps.box_sum(xd, r, out=o, J=J, ii=ii)
    assert got is o and np.array_equal(o.cpu().numpy(), want)
    assert np.array_equal(J.cpu().numpy(), c) and np.array_equal(ii.cpu().numpy(), c[1:, 1:])
    assert (flat[0, h * w:] == -7).all() and (flat[1, h * w:] == -7).all() and (flat[2, (h + 1) * (w + 1):] == -7).all()
    assert np.array_equal(apps.box_sum(xd, r, out=ii, J=J, ii=ii).cpu().numpy(), want)
