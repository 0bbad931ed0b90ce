"""Every GEMM kernel's way out when the epilogue's wait for an accumulator gives
up: one-CTA tiles of each width and pairs of CTAs, several tiles per CTA.  The
bit comes back, the kernel returns, and the next call on the stream is right."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(300, 9997, 64), (1200, 5999, 256), (1200, 11996, 136), (1200, 13995, 136),
                                   (2048, 1025, 1032), (1200, 11996, 264), (1200, 13995, 264), (64, 64, 8192)])
def test_gemm_gives_up_and_recovers(umi, dev, M, N, K):
    import torch
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g, device=dev).to(torch.bfloat16)
    B = torch.randn(N, K, generator=g, device=dev).to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    want = umi.gemm(A, B, err=err).clone()
    umi.check_err(err)
    umi.gemm_bf16_wait_limit(A, B, 1, err=err)
    bits = int(err.item())
    assert bits & 4 and bits & ~15 == 0, bits
    with pytest.raises(umi.UmiError):
        umi.check_err(err)
    err.zero_()
    assert torch.equal(umi.gemm(A, B, err=err), want)
    umi.check_err(err)
