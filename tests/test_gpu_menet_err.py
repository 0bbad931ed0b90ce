"""The network's backward pass when a device wait gives up: the bits reach the
caller's word, the gradients of the layers below are NaN (the head's and the
last layer's need no data gradient), and the next pass is whole again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(64, 96), (272, 656)])
def test_backward_reports_waits_that_gave_up(umi, dev, h, w):
    import torch
    g = np.random.default_rng(h)
    cur, ref = (torch.from_numpy(g.integers(0, 256, (h, w), dtype=np.uint8)).to(dev) for _ in range(2))
    tgt = torch.from_numpy(g.integers(-40, 40, ((h // 16) * (w // 16), 2)).astype(np.int32)).to(dev)
    net = umi.MeNet(h, w, device=dev, seed=1)
    net.ws.fill_(0xFF)  # an error word that holds bits before the first pass
    net.forward(cur, ref)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    want = net.backward(tgt, err=err).clone()
    umi.check_err(err, "backward")
    assert torch.isfinite(want).all()
    net.backward(tgt, err=err, wait_ns=1)
    bits = int(err.item())
    assert bits & 4  # a row that was not finished in time
    with pytest.raises(umi.UmiError):
        umi.check_err(err, "backward")
    layers, wh, bh, total = umi.param_layout()
    assert torch.isnan(net.grads[:layers[2][1] + 32]).all()
    assert torch.equal(net.grads[layers[3][0]:], want[layers[3][0]:])
    err.zero_()
    assert torch.equal(net.backward(tgt, err=err), want)
    assert int(err.item()) == 0
