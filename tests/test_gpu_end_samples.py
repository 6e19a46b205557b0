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


def _line_counts(n, r, a, e, j):
    """Samples of view j's rays that the Radon counts: on each strip of 16 lines
    positions start from the truncated Q32.32 one of the ray's first line in the
    strip and step in units of 2^-23."""
    d, dt = 2.0 * e / (n - 1), 2.0 / (r - 1)
    th = j * (math.pi / a)
    c, s, tn = math.cos(th), math.sin(th), math.tan(th)
    if abs(c) < 1.0 / math.sqrt(2.0):
        rk, ri, r0 = dt / (s * d), -d / (tn * d), (-1.0 / s + e / tn + e) / d
    else:
        rk, ri, r0 = dt / (c * d), -d * tn / d, (-1.0 / c + e * tn + e) / d
    rk, ri, r0 = (int(round(v * 4294967296.0)) for v in (rk, ri, r0))
    u0 = r0 + np.arange(r, dtype=np.int64)[:, None] * rk
    i = np.arange(n, dtype=np.int64)[None, :]
    # lines within [-0.5, n - 0.5], as estimated in FP32
    f = np.float32
    uf, qf = u0.astype(f) * f(2.0 ** -32), f(f(ri) * f(2.0 ** -32))
    t1, t2 = (f(-0.5) - uf) / qf, (f(n) - f(0.5) - uf) / qf
    lo = np.ceil(np.maximum(np.minimum(t1, t2), f(0))).astype(np.int64)
    hi = np.floor(np.minimum(np.maximum(t1, t2), f(n - 1))).astype(np.int64)
    first = np.maximum(lo, i & ~15)
    k = (((u0 + first * ri) >> 9) + (i - first) * ((ri + 256) >> 9)) >> 23
    return ((i >= lo) & (i <= hi) & (k >= 0) & (k <= n - 2)).sum(1), d / max(abs(c), abs(s))


@pytest.mark.parametrize("n,r,a,e,views", [
    (1205, 1450, 851, 1.0, [305, 40, 422, 700]), (1205, 1450, 851, 0.6, [29, 822, 60, 500]),
    (333, 401, 97, 0.75, range(1, 97, 5))])
def test_radon_counts_the_samples_of_truncated_positions(n, r, a, e, views):
    """Of an image of ones a ray's sum is its step times the samples it counts.
    Views 305 (ray 1205) and 29 and 822 (ray 248) meet a line's end so closely
    that positions rounded about the strip's middle count another number."""
    g = rg.gpu_image(torch.ones((n, n), device="cuda"), (-e, e), (e, -e))
    got = rg.radon(g, (r, a), SLANT).data.cpu().numpy().astype(np.float64)
    for j in views:
        want, step = _line_counts(n, r, a, e, j)
        assert np.array_equal(np.rint(got[:, j] / step), want)
        assert np.max(np.abs(got[:, j] / step - want)) < 0.01
