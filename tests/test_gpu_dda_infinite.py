"""One infinite sample, of either sign, in every view in turn: the DDA transpose and
the normalised backprojection are infinite, with its sign, on the pixels that its
ray meets, and what they are without it on all others, as the walk leaves them
(an image side less one that is a power of two makes an axis-aligned view's step
exact in FP32).  A ray may pass a pixel's corner by less than rounding, there
either value stands."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pyraft_gb300 as rg  # noqa: E402

DDA = rg.radon_method.BRESENHAM
FULL = (0.0, 1.0, math.pi, -1.0)


@pytest.mark.parametrize("n,r,a,sc", [
    (65, 46, 31, FULL),                               # reflected views, axis-aligned ones at both ends
    (64, 64, 30, (0.013, 1.0, 0.013 + math.pi, -1.0)),
    (40, 57, 21, (0.0, 1.2, 3.0, -1.1))])             # four taps
def test_infinite_samples_keep_to_their_rays(orc, n, r, a, sc):
    rng = np.random.default_rng(n)
    y = (rng.random((r, a)) + 0.5).astype(np.float32)
    ops = [lambda g: rg.radon_transpose(g, (n, n), DDA), lambda g: rg.backprojection(g, (DDA, (n, n), 0))]
    dev = lambda v: rg.gpu_image(torch.from_numpy(v).cuda(), sc[:2], sc[2:])
    plain = [op(dev(y)).data.cpu().numpy() for op in ops]
    for j in range(a):
        k = r // 2 + (5 * j) % 7 - 3
        one = np.zeros((r, a))
        one[k, j] = 1.0
        w = orc.radon_transpose_bresenham(one, (n, n), (-1.0, 1.0, 1.0, -1.0), sc)
        meets, off = w > 1e-5 * w.max(), w == 0.0
        assert meets.any()
        for v in (np.inf, -np.inf):
            s = y.copy()
            s[k, j] = v
            for op, want in zip(ops, plain):
                got = op(dev(s)).data.cpu().numpy()
                assert np.all(got[meets] == v), (j, k, v)
                assert np.all(np.isfinite(got[off]))
                assert np.all(np.abs(got[off] - want[off]) <= 1e-5 * np.abs(want[off]).max())
