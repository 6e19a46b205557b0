"""EM stays inside the workspace that its query asks for: the bytes after it keep
their values, for both slant-stack pairs and the DDA, over even and odd view
counts and subsets that do not divide them, on both sides of the 256 view pairs
from which the paired gathers stage through the workspace."""
import math

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pyraft_gb300 as rg  # noqa: E402
from pyraft_gb300 import _native  # noqa: E402
from pyraft_gb300.raftypes import rg_image, stream_ptr  # noqa: E402

GUARD = 1 << 20


@pytest.mark.parametrize("method", ["RG_SLANTSTACK", "RG_SLANTSTACK_BP", "RG_BRESENHAM"])
@pytest.mark.parametrize("n,r,a,subsets", [(384, 640, 513, 1), (416, 640, 601, 1), (384, 384, 514, 1),
                                           (385, 380, 513, 2), (64, 60, 45, 4)])
def test_em_keeps_to_its_workspace(method, n, r, a, subsets):
    m = getattr(_native, method)
    if method == "RG_SLANTSTACK":
        r = min(r, n)                                 # the matched adjoint's limit
    g = torch.Generator(device="cuda").manual_seed(n + a)
    s = rg.gpu_image(torch.rand((r, a), device="cuda", generator=g) + 0.5, (0.0, 1.0),
                     (math.pi, -1.0))
    x = rg.gpu_image(torch.ones((n, n), device="cuda"), (-1.0, 1.0), (1.0, -1.0))
    L = _native.load()
    A, B = rg_image(s), rg_image(x)
    need = L.rg_em_workspace(A, B, m, subsets)
    mem = torch.full((need + GUARD,), 0xA5, dtype=torch.uint8, device="cuda")
    _native.check(L.rg_em(A, B, m, 1, subsets, mem.data_ptr(), need, stream_ptr()))
    torch.cuda.synchronize()
    assert bool((mem[need:] == 0xA5).all())
    assert bool(torch.isfinite(x.data).all()) and bool((x.data > 0).any())
    _native.check(L.rg_device_status())
