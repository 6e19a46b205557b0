"""DDA scans at the limits of the line sums, past which the walking kernels take them:
an image of more lines than a grid has rows of 32, and a scan of many axis-aligned
views, whose rays a plan would hold one by one."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pyraft_gb300 as rg  # noqa: E402

DDA = rg.radon_method.BRESENHAM


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("lines", [65535 * 32, 65535 * 32 + 1])
def test_radon_of_a_tall_image(orc, lines):
    """Sums of up to 2 lines steps, compensated, with one rounding of each step:
    4e-7 as for every DDA Radon."""
    x = (np.random.default_rng(1).random((lines, 2)) + 0.5).astype(np.float32)
    h = 0.5 * (lines - 1)
    ic, sc = (-0.5, h, 0.5, -h), (0.4, 1.0, 0.4 + math.pi, -1.0)
    g = rg.gpu_image(torch.from_numpy(x).cuda(), ic[:2], ic[2:])
    got = rg.radon(g, (5, 4), DDA, top_left=sc[:2], bottom_right=sc[2:]).data.cpu().numpy()
    assert rel(got, orc.radon_bresenham(x.astype(np.float64), 5, 4, ic, sc)) <= 4e-7


def test_scan_of_axis_aligned_views_keeps_no_ray_lists(orc):
    """2000 views at angle 0: their rays' lists would be 131 MB, as often as there are
    geometries."""
    n, r, a = 64, 2048, 2000
    sc = (0.0, 1.0, 0.0, -1.0)
    x = (np.random.default_rng(2).random((n, n)) + 0.5).astype(np.float32)
    g = rg.gpu_image(torch.from_numpy(x).cuda(), (-1.0, 1.0), (1.0, -1.0))
    run = lambda b: rg.radon(g, (r, a), DDA, top_left=sc[:2], bottom_right=b).data
    run((math.pi, -1.0))                              # context, kernels, caching allocator
    torch.cuda.synchronize()
    free, held = torch.cuda.mem_get_info()[0], torch.cuda.memory_reserved()
    got = run(sc[2:]).cpu().numpy()
    grown = free - torch.cuda.mem_get_info()[0] - (torch.cuda.memory_reserved() - held)
    assert grown < 32 << 20
    ref = orc.radon_bresenham(x.astype(np.float64), r, 2, (-1.0, 1.0, 1.0, -1.0), sc)
    assert rel(got[:, [0, 999, 1999]], ref[:, [0, 0, 0]]) <= 4e-7


def test_cached_plans_are_bounded_in_bytes():
    """24 scans of 400000 rays with three axis-aligned views, whose lists take 38 MB
    each: the cache of plans keeps 384 MB."""
    r, n = 400000, 16
    g = rg.gpu_image(torch.ones((n, n), device="cuda"), (-1.0, 1.0), (1.0, -1.0))
    run = lambda e: rg.radon(g, (r, 3), DDA, top_left=(0.0, e), bottom_right=(math.pi, -e)).data
    run(1.0)
    torch.cuda.synchronize()
    free, held = torch.cuda.mem_get_info()[0], torch.cuda.memory_reserved()
    for k in range(24):
        out = run(1.0 + 0.01 * k)
    torch.cuda.synchronize()
    grown = free - torch.cuda.mem_get_info()[0] - (torch.cuda.memory_reserved() - held)
    assert grown <= 400 << 20
    assert bool((out.sum(0) > 0).all())
