"""Window operators on images that are not contiguous: a plan's row strides are
the caller's to set (the rows of a pitched image, every other element, rows
from the last to the first), for the image and for the centre, and every
strategy reads the elements the plan names."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
WRAP = 1


@pytest.mark.parametrize("pitch,step,flip", [(150, 1, False), (300, 2, False), (133, 1, True)])
@pytest.mark.parametrize("name", ["CENSUS_I32", "MAX_I32", "NEIGHBOUR_SUM_I32", "WEIGHTED_SUM_I32", "WEIGHTED_SUM_F32"])
@pytest.mark.parametrize("stride", [1, 2])
def test_window_of_a_pitched_image(umi, dev, name, stride, pitch, step, flip):
    import torch
    h, w, k = 40, 131, 3
    strat = getattr(umi, "STRATEGY_" + name)
    isf = name.endswith("F32")
    g = np.random.default_rng(pitch + len(name))
    buf = g.integers(-50, 51, (h, pitch)).astype(np.float32 if isf else np.int32)
    img = buf[::-1 if flip else 1, :step * (w - 1) + 1:step]
    store = torch.from_numpy(buf).to(dev)
    mem = dict(p_view=[(), (), (2, 0, 1), (3, 0, 1)], a_view=[(), (), (2, -1, stride), (3, -1, stride)],
               phys=[(1, WRAP), (1, WRAP), (h, WRAP), (w, WRAP)], stage=1)
    mems, weighted = [mem], name.startswith("WEIGHTED")
    if name == "CENSUS_I32":
        mems.insert(0, dict(p_view=mem["p_view"], phys=mem["phys"], stage=0))
    images = len(mems)
    wts = g.integers(-4, 5, (k, k)).astype(buf.dtype)
    if weighted:
        mems.append(dict(p_view=[(), (), (), ()], a_view=[(), (), (2, 0, 1), (3, 0, 1)],
                         phys=[(1, 0), (1, 0), (k, 0), (k, 0)], stage=1))
    mems.append(dict(p_view=mem["p_view"], phys=[(), (), (h, 0), (w, 0)], stage=2, out=True))
    plan = umi.plan_build(umi.make_desc(p=[(1, 1, 1, 1), (1, 1, 1, 1), (h, 8, 1, 1), (w, 32, 32, 1)],
                                        a=[(1, 1), (1, 1), (k, k), (k, k)], mems=mems))
    for m in range(images):
        plan.mem[m].rowstride[2] = -pitch if flip else pitch
        plan.mem[m].rowstride[3] = step
    first = store.data_ptr() + (4 * (h - 1) * pitch if flip else 0)
    weights = torch.from_numpy(wts).to(dev)
    inp = (ctypes.c_void_p * 2)(*[first] * images)
    if weighted:
        inp[images] = weights.data_ptr()
    out = torch.full((h, w), 77, dtype=store.dtype, device=dev)
    consts = {"NEIGHBOUR_SUM_I32": (ctypes.c_int32 * 2)(5, 3), "MAX_I32": (ctypes.c_int32 * 1)(-2 ** 31),
              "WEIGHTED_SUM_I32": (ctypes.c_int32 * 1)(2), "WEIGHTED_SUM_F32": (ctypes.c_float * 1)(2.0)}.get(name)
    umi.check(umi.lib().umi_launch(ctypes.byref(plan), strat, inp, None, (ctypes.c_void_p * 1)(out.data_ptr()), consts,
                                   ctypes.sizeof(consts) if consts is not None else 0, umi._stream_ptr()), "umi_launch")
    yy, xx = np.mgrid[:h, :w]
    at = lambda dy, dx: img[np.clip(yy + dy, 0, h - 1), np.clip(xx + dx, 0, w - 1)]  # noqa: E731
    vals = [at(-1 + stride * i, -1 + stride * j) for i in range(k) for j in range(k)]
    if name == "CENSUS_I32":
        want = np.zeros((h, w), np.uint32)
        for v in vals:
            want = (want << np.uint32(1)) | (v < at(0, 0)).astype(np.uint32)
        want = want.view(np.int32)
    elif name == "MAX_I32":
        want = np.maximum.reduce(vals)
    elif weighted:  # whole numbers below 2^24: exact in either type
        want = 2 + sum(v * c for v, c in zip(vals, wts.ravel()))
    else:
        want = (5 + sum(vals)) * 3
    assert np.array_equal(out.cpu().numpy(), want)
