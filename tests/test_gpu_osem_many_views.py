"""OSEM subsets of so many views that the rows of two of them exceed a grid: the
tile-driven Radon's epilogue then leaves the next subset's rows to their own
clearing pass.  Against the direct walks 1e-5, as for every OSEM iteration."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pyraft_gb300 as rg  # noqa: E402


@pytest.mark.parametrize("a", [65534, 65538])
def test_osem_of_two_large_subsets(monkeypatch, a):
    n, r = 16, 14
    g = torch.Generator(device="cuda").manual_seed(a)
    s = rg.gpu_image(torch.rand((r, a), device="cuda", generator=g) + 0.5, (0.0, 1.0), (math.pi, -1.0))
    outs = []
    for kernel in ("tiles", "direct"):
        monkeypatch.setenv("RG_RADON_KERNEL", kernel)
        outs.append(rg.osem(s, (n, n), 1, 2).data.cpu().numpy().astype(np.float64))
    assert np.linalg.norm(outs[0] - outs[1]) <= 1e-5 * np.linalg.norm(outs[1])
    assert outs[1].any()
