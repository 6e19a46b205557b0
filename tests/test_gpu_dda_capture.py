"""DDA calls in a stream capture.  A geometry that a plain call has met replays its line
sums; one that none has, over views that one has, walks, since a capture admits
none of the allocations that a plan makes."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pyraft_gb300 import _native  # noqa: E402
from pyraft_gb300.raftypes import stream_ptr  # noqa: E402

SQ = (-1.0, 1.0, 1.0, -1.0)


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("call", ["radon", "radon_transpose", "backprojection", "em"])
def test_calls_in_a_capture(orc, call):
    L = _native.load()
    a = {"radon": 43, "radon_transpose": 44, "backprojection": 46, "em": 47}[call]
    rng = np.random.default_rng(a)

    def buffers(n, r):
        x = torch.from_numpy((rng.random((n, n)) + 0.5).astype(np.float32)).cuda()
        y = torch.from_numpy((rng.random((r, a)) + 0.5).astype(np.float32)).cuda()
        I = _native.RG_IMAGE(x.data_ptr(), n, 1, n, n, *SQ)
        S = _native.RG_IMAGE(y.data_ptr(), r, 1, a, a, 0.0, 1.0, math.pi, -1.0)
        if call == "em":
            need = L.rg_em_workspace(S, I, _native.RG_BRESENHAM, 1)
            run = lambda ws: L.rg_em(S, I, _native.RG_BRESENHAM, 2, 1, ws.data_ptr(), need, stream_ptr())
        else:
            args = (I, S) if call == "radon" else (S, I)
            need = getattr(L, f"rg_{call}_bresenham_workspace")(*args)
            fn = getattr(L, f"rg_{call}_bresenham")
            run = lambda ws: fn(*args, ws.data_ptr(), need, stream_ptr())
        return x, y, run, torch.empty(max(need, 1), dtype=torch.uint8, device="cuda")

    def captured(x, y, run, ws):
        x0, y0 = x.clone(), y.clone()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            rc = run(ws)
        _native.check(rc)
        x.copy_(x0)
        y.copy_(y0)
        g.replay()
        torch.cuda.synchronize()
        return (y if call == "radon" else x).cpu().numpy()

    x, y, run, ws = buffers(48, 50)
    x0 = x.clone()
    _native.check(run(ws))                            # the geometry's plan, the views' table
    torch.cuda.synchronize()
    want = (y if call == "radon" else x).cpu().numpy()
    x.copy_(x0)
    assert np.array_equal(captured(x, y, run, ws), want)

    n, r = 56, 60                                     # another geometry
    x, y, run, ws = buffers(n, r)
    x64, y64 = x.cpu().numpy().astype(np.float64), y.cpu().numpy().astype(np.float64)
    got = captured(x, y, run, ws)
    if call == "radon":
        ref = orc.radon_bresenham(x64, r, a)
    elif call == "radon_transpose":
        ref = orc.radon_transpose_bresenham(y64, (n, n))
    elif call == "backprojection":
        ref = orc.backprojection_bresenham(y64, (n, n))
    else:
        ref, sens = x64, orc.radon_transpose_bresenham(np.ones((r, a)), (n, n))
        for _ in range(2):
            p = orc.radon_bresenham(ref, r, a)
            ref = ref * orc.radon_transpose_bresenham(np.divide(y64, p, out=np.zeros_like(p), where=p != 0), (n, n))
            ref = np.divide(ref, sens, out=np.zeros_like(ref), where=sens != 0)
    assert rel(got, ref) <= 1e-5
