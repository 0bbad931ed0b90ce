"""Window operators of the UMI family on the generic operator (umi_launch).

The reference ships eight example applications; these are four more of the
same kind, each a descriptor with a built-in strategy, which umi_launch serves
from staged image tiles where the window allows it and else by the closed-form
generic kernel:

* ``census``: census transform, one bit per window pixel (row-major), set
  where the pixel is below the centre (CENSUS_I32); edges replicated.
* ``box_sum``: sums over (2r+1)^2 windows clipped to the image, from the
  integral image (``iimg_u8_i32``): four corner reads of the zero-bordered
  integral image with weights +1 -1 -1 +1 (WEIGHTED_SUM_I32 over a 2 x 2
  accumulation view of stride 2r+1, coordinates clamped); buffers that do
  not overlap take the same sums straight from the integral image
  (``umi_box_sum_u8``).
* ``gaussian``: separable Gaussian blur, a horizontal then a vertical pass
  of WEIGHTED_SUM_F32 with the normalised 1-D kernel; edges replicated.  Up
  to 31 weights both passes are one launch (``umi_separable_f32``, same bits).
* ``dilate`` / ``erode``: grey-level max / min over (2r+1)^2 windows
  (MAX_I32 / MIN_I32); edges replicated.

All take and return CUDA tensors of shape (h, w) and run on the current
stream.

A plan depends on the sizes alone and takes Python longer to build than the
GPU needs for the whole call (0.09 ms of a 0.05 ms kernel), so the last few
sizes' plans are kept (they are only read).
"""
from __future__ import annotations

import functools
import math
import operator

import numpy as np

import umi_gb300 as U

PAD, WRAP = 0, 1


_CONST = {}  # small constant tensors (weights) per (device, key): made once, so calls can be graph-captured


def _const(dev, key, make):
    import torch
    k = (str(dev), key)
    if k not in _CONST:
        _CONST[k] = torch.from_numpy(np.ascontiguousarray(make())).to(dev)
    return _CONST[k]


def _p(h, w):
    return [(1, 1, 1, 1), (1, 1, 1, 1), (h, 16, 4, 1), (w, 16, 8, 1)]


def _img(h, w, mode=WRAP, a_view=None, stage=1, out=False):
    m = dict(p_view=[(), (), (2, 0, 1), (3, 0, 1)], phys=[(1, mode), (1, mode), (h, mode), (w, mode)], stage=stage)
    if a_view is not None:
        m["a_view"] = a_view
    if out:
        m["out"] = True
    return m


def _int(v):
    """v as a plain int: plans are kept by value, never by an array's or a tensor's identity."""
    return v if type(v) is int else operator.index(v)


@functools.lru_cache(maxsize=64, typed=True)
def _census_plan(h, w, radius):
    k = 2 * radius + 1
    d = U.make_desc(p=_p(h, w), a=[(1, 1), (1, 1), (k, k), (k, k)],
                    mems=[_img(h, w, stage=0), _img(h, w, a_view=_window(radius)), _img(h, w, PAD, stage=2, out=True)])
    return U.PlannedLaunch(d, U.STRATEGY_CENSUS_I32)


@functools.lru_cache(maxsize=64, typed=True)
def _extremum_plan(h, w, radius, strategy, init):
    k = 2 * radius + 1
    d = U.make_desc(p=_p(h, w), a=[(1, 1), (1, 1), (k, k), (k, k)],
                    mems=[_img(h, w, a_view=_window(radius)), _img(h, w, PAD, stage=2, out=True)])
    return U.PlannedLaunch(d, strategy, [init])


@functools.lru_cache(maxsize=64, typed=True)
def _box_plan(h, w, radius):
    k = 2 * radius + 1
    # corner (a_y, a_x) of point (y, x): J[clamp(y - r + a_y k)][clamp(x - r + a_x k)]
    jmem = dict(p_view=[(), (), (2, -radius, 1), (3, -radius, 1)], a_view=[(), (), (2, 0, k), (3, 0, k)],
                phys=[(1, WRAP), (1, WRAP), (h + 1, WRAP), (w + 1, WRAP)], stage=1)
    wmem = dict(p_view=[(), (), (), ()], a_view=[(), (), (2, 0, 1), (3, 0, 1)],
                phys=[(1, PAD), (1, PAD), (2, PAD), (2, PAD)], stage=1)
    d = U.make_desc(p=_p(h, w), a=[(1, 1), (1, 1), (2, 2), (2, 2)], mems=[jmem, wmem, _img(h, w, PAD, stage=2, out=True)])
    return U.PlannedLaunch(d, U.STRATEGY_WEIGHTED_SUM_I32, [0])


@functools.lru_cache(maxsize=64, typed=True)
def _gaussian_plans(h, w, k):
    r = k // 2
    dh = U.make_desc(p=_p(h, w), a=[(1, 1), (1, 1), (1, 1), (k, k)],
                     mems=[_img(h, w, a_view=[(), (), (), (3, -r, 1)]),
                           dict(p_view=[(), (), (), ()], a_view=[(), (), (), (3, 0, 1)],
                                phys=[(1, PAD), (1, PAD), (1, PAD), (k, PAD)], stage=1),
                           _img(h, w, PAD, stage=2, out=True)])
    dv = U.make_desc(p=_p(h, w), a=[(1, 1), (1, 1), (k, k), (1, 1)],
                     mems=[_img(h, w, a_view=[(), (), (2, -r, 1), ()]),
                           dict(p_view=[(), (), (), ()], a_view=[(), (), (2, 0, 1), ()],
                                phys=[(1, PAD), (1, PAD), (k, PAD), (1, PAD)], stage=1),
                           _img(h, w, PAD, stage=2, out=True)])
    return tuple(U.PlannedLaunch(d, U.STRATEGY_WEIGHTED_SUM_F32, [0.0]) for d in (dh, dv))


def _window(r):
    return [(), (), (2, -r, 1), (3, -r, 1)]


def census(img, radius: int = 1, out=None, stream=None):
    """Census transform of an int32 image over (2 radius + 1)^2 windows
    (radius <= 2 keeps every bit: at most 32)."""
    import torch
    h, w = img.shape
    if out is None:
        out = torch.empty((h, w), dtype=torch.int32, device=img.device)
    _census_plan(h, w, _int(radius))((img, img), (out,), stream)
    return out


def _extremum(img, radius, strategy, init, out, stream):
    import torch
    h, w = img.shape
    if out is None:
        out = torch.empty((h, w), dtype=torch.int32, device=img.device)
    _extremum_plan(h, w, _int(radius), strategy, init)((img,), (out,), stream)
    return out


def dilate(img, radius: int = 1, out=None, stream=None):
    """Grey-level dilation (window maximum) of an int32 image."""
    return _extremum(img, radius, U.STRATEGY_MAX_I32, -(1 << 31), out, stream)


def erode(img, radius: int = 1, out=None, stream=None):
    """Grey-level erosion (window minimum) of an int32 image."""
    return _extremum(img, radius, U.STRATEGY_MIN_I32, (1 << 31) - 1, out, stream)


def _box_direct(img, radius, out, J, ii):
    """Whether the windows' corners can be read straight from the integral
    image: buffers of its shape that do not overlap (through J, each step had
    read its input before the next one wrote)."""
    h, w = img.shape
    if not (0 < h <= 500000 and 0 < w and 0 <= radius <= 1 << 20):
        return False
    if (J is not None and tuple(J.shape) != (h + 1, w + 1)) or any(
            t is not None and tuple(t.shape) != (h, w) for t in (out, ii)):
        return False
    at = sorted((t.data_ptr(), t.numel()) for t in (out, J, ii) if t is not None)
    return all(a + 4 * n <= b for (a, n), (b, _) in zip(at, at[1:]))


def box_sum(img_u8, radius: int, out=None, J=None, ii=None, workspace=None, stream=None):
    """Sums of a uint8 image over (2 radius + 1)^2 windows clipped to the
    image (int32), from its integral image.  J ((h+1, w+1) int32, first row
    and column zero), ii ((h, w) int32) and the iimg workspace may be passed
    in to avoid allocations."""
    import torch
    h, w = img_u8.shape
    dev = img_u8.device
    radius = _int(radius)
    if _box_direct(img_u8, radius, out, J, ii):
        U._need(img_u8, torch.uint8, "inp")
        ii = torch.empty((h, w), dtype=torch.int32, device=dev) if ii is None else ii
        out = torch.empty((h, w), dtype=torch.int32, device=dev) if out is None else out
        for name, t in (("out", ii), ("memory 0", J), ("memory 2", out)):
            if t is not None:
                U._need(t, torch.int32, name)
        if workspace is None:
            workspace = torch.empty(max(U.iimg_workspace_bytes(h, w), 16), dtype=torch.uint8, device=dev)
        U.check(U.lib().umi_box_sum_u8(U._ptr(img_u8), h, w, radius, U._ptr(ii), U._ptr(J), U._ptr(out),
                                       U._ptr(workspace), workspace.numel(), U._stream_ptr(stream)), "umi_box_sum_u8")
        return out
    if J is None:
        J = torch.zeros((h + 1, w + 1), dtype=torch.int32, device=dev)  # J[y][x] = sum of img[:y, :x]
    J[1:, 1:] = U.iimg_u8_i32(img_u8, out=ii, workspace=workspace, stream=stream)
    wts = _const(dev, "box", lambda: np.array([[1, -1], [-1, 1]], np.int32))
    if out is None:
        out = torch.empty((h, w), dtype=torch.int32, device=dev)
    _box_plan(h, w, radius)((J, wts), (out,), stream)
    return out


def gaussian_kernel(sigma: float, radius: int | None = None) -> np.ndarray:
    """Normalised 1-D Gaussian weights exp(-i^2 / (2 sigma^2)), i = -r..r
    (r = ceil(3 sigma) by default), as float32."""
    return _gaussian_kernel(sigma, radius).copy()


def _gaussian_kernel(sigma, radius) -> np.ndarray:
    if type(sigma) is not float and isinstance(sigma, np.ndarray):
        sigma = sigma[()]
    return _kernel_of(sigma, radius if radius is None or type(radius) is int else int(radius))


@functools.lru_cache(maxsize=64, typed=True)
def _kernel_of(sigma: float, radius: int | None) -> np.ndarray:
    r = int(math.ceil(3 * sigma)) if radius is None else radius
    t = np.arange(-r, r + 1, dtype=np.float64)
    k = np.exp(-t * t / (2.0 * sigma * sigma))
    return (k / k.sum()).astype(np.float32)


def _one_launch(img, tmp, out, k):
    """Whether both passes can go in one launch: few enough weights, and no
    buffer overlaps another (each pass alone may then write what it has read)."""
    if k > 31 or not 0 < img.shape[0] <= 1 << 20 or img.shape[1] == 0:
        return False
    n = 4 * img.shape[0] * img.shape[1]
    at = [t.data_ptr() for t in (img, tmp, out) if t is not None]
    return all(abs(a - b) >= n for i, a in enumerate(at) for b in at[:i])


def gaussian(img, sigma: float, radius: int | None = None, out=None, tmp=None, stream=None):
    """Separable Gaussian blur of a float32 image (edges replicated)."""
    import torch
    h, w = img.shape
    kern = _gaussian_kernel(sigma, radius)
    k = kern.size
    dev = img.device
    wt = _const(dev, ("gauss", float(sigma), k), lambda: kern)
    if out is None:
        out = torch.empty((h, w), dtype=torch.float32, device=dev)
    if _one_launch(img, tmp, out, k):
        U._check_memories(U.STRATEGY_WEIGHTED_SUM_F32, (img, wt), (out,) if tmp is None else (tmp, out))
        U.check(U.lib().umi_separable_f32(U._ptr(img), U._ptr(wt), k, h, w, U._ptr(tmp), U._ptr(out),
                                          U._stream_ptr(stream)), "umi_separable_f32")
        return out
    if tmp is None:
        tmp = torch.empty((h, w), dtype=torch.float32, device=dev)
    across, down = _gaussian_plans(h, w, k)
    across((img, wt), (tmp,), stream)
    down((tmp, wt), (out,), stream)
    return out
