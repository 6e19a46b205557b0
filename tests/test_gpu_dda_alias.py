"""DDA calls whose output lies in their input's memory: the operators read all of it
before they write, so the output is that of separate memory, bit for bit.  The
scans have axis-aligned views, and the images a ray that the walk loses (the
diagonal of 3 pi / 4 on an even grid) and a non-finite pixel, whose rays are
walked after the others."""
import math

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from pyraft_gb300 import _native  # noqa: E402
from pyraft_gb300.raftypes import stream_ptr  # noqa: E402


def _image(t, offset, rows, cols, ld_row, ld_col, tl, br):
    return _native.RG_IMAGE(t.data_ptr() + 4 * offset, rows, ld_col, cols, ld_row, *tl, *br)


@pytest.mark.parametrize("shift", [0, 1000])
@pytest.mark.parametrize("layout", ["view", "ray"])
@pytest.mark.parametrize("call", ["radon", "radon_transpose", "backprojection"])
def test_output_in_the_inputs_memory(call, layout, shift):
    # (a normalised backprojection of a scan that loses a ray walks: not 3 pi / 4)
    n, r, a = 300, 301, 182 if call == "backprojection" else 185
    L = _native.load()
    fn = getattr(L, f"rg_{call}_bresenham")
    wsfn = getattr(L, f"rg_{call}_bresenham_workspace")
    g = torch.Generator(device="cuda").manual_seed(n)
    data = torch.rand(r * a + n * n + shift, device="cuda", generator=g) + 0.5
    sld = (1, r) if layout == "view" else (a, 1)      # strides of a ray, of a view

    def run(apart):
        inp = data.clone()
        out = torch.zeros_like(inp) if apart else inp
        im, sino = ((inp, out) if call == "radon" else (out, inp))
        io, so = (0, shift) if call == "radon" else (shift, 0)
        if call == "radon":
            inp[77 * n + 120] = math.nan
        I = _image(im, io, n, n, n, 1, (-1.0, 1.0), (1.0, -1.0))
        S = _image(sino, so, r, a, *sld, (0.0, 1.0), (math.pi, -1.0))
        args = (I, S) if call == "radon" else (S, I)
        need = wsfn(*args)
        ws = torch.empty(max(need, 1), dtype=torch.uint8, device="cuda")
        _native.check(fn(*args, ws.data_ptr(), need, stream_ptr()))
        torch.cuda.synchronize()
        n_out, o = (r * a, so) if call == "radon" else (n * n, io)
        return out[o:o + n_out].clone()

    want, got = run(True), run(False)
    assert bool(want.any())
    assert torch.equal(torch.nan_to_num(want, nan=-1.0), torch.nan_to_num(got, nan=-1.0))
