"""The network's passes in a workspace of the size that was named for them
before the gradients took bf16 parts, as in one of the size named now: the
same predictions, gradients and searches, nothing written behind it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _former(h, w):
    al = lambda b: (b + 255) // 256 * 256  # noqa: E731
    P, nblk, head = h * w // 16, (h // 16) * (w // 16), -(-(h * w // 256) // 8)
    wb = [2 * 32 * c * 9 for c in (2, 32, 32, 32)]
    tiles = -(-(w // 4) // 32) * -(-(h // 4) // 4)
    parts = ([8 * P] + [128 * P] * 4 + [128 * P] * 2 + wb + wb + [8 * nblk, 8 * nblk, 4 * nblk, 16, 4 * nblk, 12 * nblk]
             + [4 * tiles * (32 * 32 * 9 + 32), 4 * head * (2 * 512 + 2), 4 * head] + [64 * P] * 2 + [18432] * 4 + [4])
    return sum(al(b) for b in parts)


@pytest.mark.parametrize("h,w", [(16, 16), (16, 64), (48, 32), (64, 64), (32, 656), (256, 1024), (720, 1280)])
def test_former_workspace(umi, dev, h, w):
    import torch
    g = np.random.default_rng(h + w)
    cur, ref = (torch.from_numpy(g.integers(0, 256, (h, w), dtype=np.uint8)).to(dev) for _ in range(2))
    tgt = torch.from_numpy(g.integers(-40, 40, ((h // 16) * (w // 16), 2)).astype(np.int32)).to(dev)
    net = umi.MeNet(h, w, device=dev, seed=3)

    def passes():
        pred = net.forward(cur, ref).clone()
        infer = net.infer(cur, ref).clone()
        net.forward(cur, ref)
        grads = net.backward(tgt).clone()
        again = net.backward(tgt).clone()  # the forward pass's activations are still there
        assert torch.equal(grads, again)
        found = net.estimate(cur, ref, 4, 16, sad_threshold=9000, audit_stride=3)
        return pred, infer, net.loss.clone(), grads, found
    want = passes()
    flat = torch.full((_former(h, w) + 512,), 0xFF, dtype=torch.uint8, device=dev)
    net.ws = flat[:_former(h, w)]
    got = passes()
    assert (flat[_former(h, w):] == 0xFF).all()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert all(torch.equal(a, b) for a, b in zip(got[4], want[4]))
    # other numbers of partial sums: fp32 sums of at most h w / 16 products
    assert torch.allclose(got[2], want[2], rtol=1e-5)
    layers, wh, bh, _ = umi.param_layout()
    for a, b in [(wo, bo) for wo, bo in layers] + [(bo, bo + 32) for _, bo in layers] + [(wh, bh), (bh, bh + 2)]:
        assert (got[3][a:b] - want[3][a:b]).abs().max() <= 1e-5 * want[3][a:b].abs().max() + 1e-12
    net.ws = flat[:4096]
    with pytest.raises(umi.UmiError):
        net.forward(cur, ref)
