"""End samples of the slant stack.  The backprojection counts a sample of a view
only while its floor index is in [0, R - 2] and the Radon one of a line while it
is in [0, N - 2]; the value there does not go to zero, so a position within
rounding of an end puts or drops a whole sample in one element.  Inputs whose
end samples do not vanish, held element by element (no norm over the image
would see one of them).

An odd number of views has no quarter-turn pairs: every pixel takes every view
at its own position, the one-view gather's, whatever RG_GATHER_ROT says."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pyraft_gb300 as rg  # noqa: E402

SLANT = rg.radon_method.SLANTSTACK


def _sino(r, a, seed, layout="ray"):
    s = np.random.default_rng(seed).random((r, a)).astype(np.float32)
    t = torch.from_numpy(s).cuda()
    if layout == "view":
        t = t.t().contiguous().t()
    return s, rg.gpu_image(t, (0.0, 1.0), (math.pi, -1.0))


@pytest.mark.parametrize("n,a,kind,layout", [
    (384, 513, "ramlak", "ray"), (511, 409, "lowpass", "view"), (640, 401, "ramlak", "view"),
    (512, 513, "lowpass", "ray"), (991, 859, "lowpass", "ray")])
def test_fbp_of_odd_views_takes_one_view_at_a_time(monkeypatch, n, a, kind, layout):
    _, g = _sino(n, a, n + a, layout)
    run = lambda: rg.fbp(g, n, filter=kind).data.cpu().numpy()
    got = run()
    monkeypatch.setenv("RG_GATHER_ROT", "0")
    assert np.array_equal(got, run())


@pytest.mark.parametrize("rows", ["4", "8", "16"])
@pytest.mark.parametrize("n,r,a", [(384, 384, 61), (400, 551, 257), (417, 417, 96)])
def test_backprojection_element_by_element(orc, monkeypatch, n, r, a, rows):
    """Positions are stepped in units of 2^-23 of a sample from a tile's corner
    (127 rows, 31 columns): within 127 2^-24 + 31 2^-24 + 2^-23 = 9.6e-6 of the
    64-bit ones.  Samples in [0, 1): a view's value moves by at most that, pi / A
    of it counts, A views: 3.1e-5, and 1e-6 for the sums.  A pixel that meets
    views within 1e-5 of the detector's ends may gain or lose a sample of each."""
    s, g = _sino(r, a, r + a)
    monkeypatch.setenv("RG_GATHER_ROWS", rows)
    run = lambda: rg.backprojection(g, (SLANT, (n, n), 0)).data.cpu().numpy()
    got = run()
    ref = orc.backprojection_slantstack(s.astype(np.float64), n)
    x = np.linspace(-1.0, 1.0, n)
    near = np.zeros((n, n))
    for j in range(a):
        th = j * math.pi / a
        u = (x[None, :] * math.cos(th) + x[:, None] * math.sin(th) + 1.0) * ((r - 1) / 2.0)
        near += (np.abs(u) < 1e-5) | (np.abs(u - (r - 1)) < 1e-5)
    assert near.any()
    off = np.abs(got - ref)
    assert np.all(off <= 3.2e-5 + near * (math.pi / a))
    if a % 2:
        monkeypatch.setenv("RG_GATHER_ROT", "0")
        assert np.array_equal(got, run())
