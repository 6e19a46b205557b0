"""The normalised DDA backprojection is as near to 64 bits as its FP32 result allows:
the walk's two FP64 sums are two FP32 numbers each here, with the rounding errors
of the products.  What is left are the weights, rounded twice or so to 2^-25: rms
1.3e-8 of a weight of 0.6 at the mean, over 2 A rays per pixel and samples that
spread about as much as they average, 1e-9 at 200 views, beside 2.5e-8 for the
rounding of the result: under 0.1 %, and 0.2 % is allowed.  (One rounding of
every product makes 0.7 to 1.3 %.)"""
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


@pytest.mark.parametrize("n,r,a,ic,sc", [
    (300, 300, 200, (-1.0, 1.0, 1.0, -1.0), FULL),              # reflected views
    (301, 290, 211, (-1.0, 1.0, 1.0, -1.0), (0.2, 1.0, 2.9, -1.0)),   # half-turn pairs
    (256, 360, 240, (-0.9, 1.0, 1.0, -0.9), FULL)])             # four taps
def test_error_is_the_results_rounding(orc, n, r, a, ic, sc):
    rng = np.random.default_rng(n)
    t = np.linspace(-1.0, 1.0, r)[:, None]
    s = (2.0 * np.sqrt(np.maximum(0.5 - (t - 0.2 * np.cos(np.arange(a) * 0.02)) ** 2, 0.0)) +
         0.05 * rng.random((r, a))).astype(np.float32)
    g = rg.gpu_image(torch.from_numpy(s).cuda(), sc[:2], sc[2:])
    got = rg.backprojection(g, (DDA, (n, n), 0), top_left=ic[:2], bottom_right=ic[2:]).data
    ref = orc.backprojection_bresenham(s.astype(np.float64), (n, n), ic, sc)
    err = np.linalg.norm(got.cpu().numpy().astype(np.float64) - ref)
    assert err <= 1.002 * np.linalg.norm(ref.astype(np.float32).astype(np.float64) - ref)
