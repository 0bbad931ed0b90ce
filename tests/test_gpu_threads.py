"""Host threads calling one operator at sizes that need different amounts of
shared memory, on a stream each: no call fails, every result is that of a call
alone.  (A launch whose shared memory exceeds what its kernel was last allowed
is refused by the CUDA runtime before it reaches the GPU.)"""
import sys
import threading

import pytest

pytestmark = pytest.mark.gpu


def _run(umi, name, calls, outs, n=4000):
    """n calls of the library's function `name` per thread; calls: its arguments
    before the stream, one list per thread."""
    import torch
    fn, want = getattr(umi.lib(), name), []
    for args, out in zip(calls, outs):
        assert fn(*args, umi._stream_ptr()) == 0
        want.append(out.clone())
    torch.cuda.synchronize()
    failed, start = [], threading.Barrier(len(calls))

    def work(args):
        stream = torch.cuda.Stream()
        ptr = umi._stream_ptr(stream)
        start.wait()
        for i in range(n):
            status = fn(*args, ptr)
            if status:
                failed.append((status, umi.lib().umi_last_error_string()))
                break
        stream.synchronize()
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        ts = [threading.Thread(target=work, args=(c,)) for c in calls]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    torch.cuda.synchronize()
    assert not failed, failed[:3]
    for out, w in zip(outs, want):
        assert torch.equal(out, w)


def test_blur(umi, dev):
    import torch
    x = torch.rand(33, 130, device=dev)
    outs, calls = [], []
    for k in (9, 31, 17, 29):
        w = torch.rand(k, device=dev)
        outs.append(torch.empty_like(x))
        calls.append([umi._ptr(x), umi._ptr(w), k, 33, 130, None, umi._ptr(outs[-1])])
        outs[-1].weights = w
    _run(umi, "umi_separable_f32", calls, outs)


@pytest.mark.parametrize("block,h,radii", [(16, 96, (9, 16, 24, 31)), (16, 48, (48, 64, 56, 60)), (8, 160, (7, 8, 5, 3)),
                                           (8, 160, (33, 64, 50, 40))])
def test_search(umi, dev, block, h, radii):
    import torch
    g = torch.Generator(device=dev).manual_seed(block)
    c, r = (torch.randint(0, 256, (h, 640), dtype=torch.uint8, device=dev, generator=g) for _ in range(2))
    outs = [torch.empty(((h // block) * (640 // block), 3), dtype=torch.int32, device=dev) for _ in radii]
    calls = [[umi._ptr(c), umi._ptr(r), h, 640, block, rad, None, umi._ptr(o)] for rad, o in zip(radii, outs)]
    _run(umi, "umi_full_me_u8", calls, outs)


def test_search_volume(umi, dev):
    import torch
    c, r = (torch.randint(0, 256, (32, 64), dtype=torch.uint8, device=dev) for _ in range(2))
    outs = [torch.empty((8, 2 * rad + 1, 2 * rad + 1), dtype=torch.int32, device=dev) for rad in (36, 64, 40, 50)]
    calls = [[umi._ptr(c), umi._ptr(r), 32, 64, 16, rad, umi._ptr(o)] for rad, o in zip((36, 64, 40, 50), outs)]
    _run(umi, "umi_full_me_sad_u8", calls, outs)


def test_window(umi, dev):
    import ctypes

    import torch
    from umi_gb300 import apps
    x = torch.randint(-99, 99, (48, 200), dtype=torch.int32, device=dev)
    outs, calls = [], []
    for rad in (20, 24, 30, 36):
        outs.append(torch.empty_like(x))
        plan = apps._extremum_plan(48, 200, rad, umi.STRATEGY_MAX_I32, -(1 << 31))
        calls.append([plan._ref, umi.STRATEGY_MAX_I32, (ctypes.c_void_p * 1)(x.data_ptr()), None,
                      (ctypes.c_void_p * 1)(outs[-1].data_ptr()), plan._consts, plan._bytes])
    _run(umi, "umi_launch", calls, outs)
