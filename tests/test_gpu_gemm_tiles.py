"""Every form of the half-precision product: one-CTA tiles of each width and
pairs of CTAs of each width, the one-CTA ones and the wide pairs with three or
more tiles per CTA (each accumulator used again), ragged in M and N, with and
without TMA stores.  The launcher's choice is asserted, so that another cost
model cannot leave a form without its test."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _tile(umi, M, N, K):
    w, p = ctypes.c_int32(), ctypes.c_int32()
    umi.check(umi.lib().umi_gemm_tile(M, N, K, ctypes.byref(w), ctypes.byref(p)), "umi_gemm_tile")
    return w.value, p.value


# (tile, pair, rounds of the grid at 152 SMs)
@pytest.mark.parametrize("M,N,K,width,pair,rounds", [
    (300, 9997, 64, 64, 0, 3), (1200, 5999, 256, 128, 0, 3), (1200, 11996, 136, 224, 0, 3), (1200, 13995, 136, 256, 0, 3),
    (2048, 1025, 1032, 128, 1, 1), (1200, 11996, 264, 224, 1, 3), (1200, 13995, 264, 256, 1, 3), (2047, 2045, 1000, 256, 1, 1)])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
def test_every_tile(umi, dev, M, N, K, width, pair, rounds, dt):
    import torch
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    if sms == 152:
        assert _tile(umi, M, N, K) == (width, pair)
        assert -(-M // (256 if pair else 128)) * -(-N // width) > (rounds - 1) * (76 if pair else 152)
    tdt = torch.bfloat16 if dt == "bf16" else torch.float16
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    A, B = (torch.randn(n, K, generator=g, device=dev).to(tdt) for n in (M, N))
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    flat = torch.full((M * N + 64,), -7.0, device=dev)
    C = umi.gemm(A, B, out=flat[:M * N].view(M, N), err=err)
    assert int(err.item()) == 0 and (flat[M * N:] == -7.0).all() and torch.isfinite(C).all()
    # whole rows and columns of every block of 32 rows against FP64, 1e-5 of the sum of |a b| (the other products' bound)
    a, b = A.double(), B.double()
    rows = torch.arange(0, M, 31, device=dev)
    cols = torch.arange(0, N, 61, device=dev)
    for i, j in ((rows, slice(None)), (slice(None), cols)):
        want, scale = a[i] @ b[j].T, a[i].abs() @ b[j].abs().T
        got = C[i][:, j] if isinstance(i, slice) else C[i]
        assert ((got.double() - want).abs() <= 1e-5 * scale).all()
