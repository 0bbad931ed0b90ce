"""The exact elimination search where a CTA takes a run of several blocks (at
least two runs per SM, so frames of 306 runs and more on 152 SMs): runs of 2 to
8 blocks with a ragged last one, rows of any alignment, blocks that are searched
exhaustively beside blocks that are not.  Against the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# blocks per run: 8 (17 = 8 + 8 + 1 in a row), 7 and 6 (+-16; two runs of 7 in a
# row would leave SMs idle), 5, 4 and 3 (+-32), 2 (+-33, +-35); one width each
# that is a multiple of 16 and one that is not
@pytest.mark.parametrize("h,w,r", [(1632, 272, 8), (1639, 277, 8), (1632, 240, 16), (1633, 245, 16), (1632, 211, 16),
                                   (1632, 176, 24), (1632, 189, 24), (1632, 144, 32), (1640, 150, 32), (1632, 115, 32),
                                   (1632, 80, 33), (1637, 83, 35)])
def test_runs_match_oracle(umi, orc, dev, h, w, r):
    import torch
    from umi_gb300.workloads import gaussian_blur
    g = np.random.default_rng(h + w + r)

    def tensor(a, shift):
        flat = torch.zeros(a.size + 256, dtype=torch.uint8, device=dev)
        t = flat[shift:shift + a.size].view(a.shape)
        t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
        return t
    a = gaussian_blur(g.normal(0, 1, (h + 8, w + 8)).astype(np.float32), 1.5)
    x = np.clip(128 + 30 * a / a.std(), 0, 255)
    ref, cur = x[4:4 + h, 4:4 + w].copy(), x[7:7 + h, 2:2 + w] + g.normal(0, 2, (h, w))
    for i in range(0, h, 48):  # noise and flat patches of one to three blocks, at changing places of the rows
        at = int(g.integers(0, w - 16))
        cur[i:i + 16, at:at + 40] = g.integers(0, 256, cur[i:i + 16, at:at + 40].shape)
        ref[i + 16:i + 40, at // 2:at // 2 + 70] = 90 + g.normal(0, 1, ref[i + 16:i + 40, at // 2:at // 2 + 70].shape)
    cur, ref = (np.clip(v, 0, 255).astype(np.uint8) for v in (cur, ref))
    shift = 0 if w % 16 == 0 else 5
    got = umi.full_me_u8(tensor(cur, shift), tensor(ref, shift), 16, r).cpu().numpy()
    assert np.array_equal(got, orc.full_me_u8(cur, ref, 16, r))
