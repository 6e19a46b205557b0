"""A non-finite sample in the lowpass filter makes its view NaN and changes no other:
two views share a complex transform, for ray counts that are a power of two and
that are not, and in the FBP the paired backprojection's quads.  The other views
are what they are without it, but for the rounding that they take from the view
they share a transform with (1e-7 of the larger one, 1e-6 in the image)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pyraft_gb300 as rg  # noqa: E402

SLANT = rg.radon_method.SLANTSTACK


def _sino(s):
    return rg.gpu_image(torch.from_numpy(s).cuda(), (0.0, 1.0), (math.pi, -1.0))


@pytest.mark.parametrize("value", [math.nan, math.inf, -math.inf])
@pytest.mark.parametrize("r,a", [(2, 3), (33, 5), (64, 6), (367, 9), (512, 4), (1025, 3)])
def test_one_sample_spoils_one_view(r, a, value):
    s = (np.random.default_rng(r).random((r, a)) + 0.5).astype(np.float32)
    want = rg.lowpassino_fbp(_sino(s)).data.cpu().numpy()
    for j, k in ((0, 0), (a - 1, r - 1), (1, r // 2)):
        t = s.copy()
        t[k, j] = value
        got = rg.lowpassino_fbp(_sino(t)).data.cpu().numpy()
        assert np.isnan(got[:, j]).all()
        rest = [q for q in range(a) if q != j]
        assert np.abs(got[:, rest] - want[:, rest]).max() <= 3e-7 * np.abs(want).max()


@pytest.mark.parametrize("n,a", [(67, 40), (64, 512), (67, 512)])
def test_the_image_misses_one_view(monkeypatch, n, a):
    """Pixels outside the detector's range at the spoiled view stay finite, and are those
    of the filter and the backprojection one after the other."""
    s = (np.random.default_rng(n).random((n, a)) + 0.5).astype(np.float32)
    s[n // 2, a // 3] = math.nan
    run = lambda: rg.fbp(_sino(s), n).data.cpu().numpy()
    got = run()
    monkeypatch.setenv("RG_FBP_QUADS", "0")
    want = run()
    bad = np.isnan(want)
    assert bad.any() and not bad.all()
    assert np.array_equal(np.isnan(got), bad)
    assert np.abs(got - want)[~bad].max() <= 1e-6 * np.abs(want[~bad]).max()
