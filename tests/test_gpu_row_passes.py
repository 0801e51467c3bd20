"""The residual passes that hold a row in registers (csrc/hybrid_block.cu) against float64: widths on both sides of a part of the row a thread
more, of the general form (not a multiple of four, more than 4096), every norm and every operand there and not there."""
import ctypes as C

import pytest
import torch

import hyb_cabi as H

pytestmark = pytest.mark.gpu
F, L = C.c_float, C.c_longlong
RMS, DYT, LAYER, COPY = range(4)


def norm(x, kind, w, b):
    if kind == RMS:
        return x / (x.square().mean(-1, keepdim=True) + 1e-5).sqrt() * (0.5 + w)
    if kind == LAYER:
        d = x - x.mean(-1, keepdim=True)
        return d / (d.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w + b
    return torch.tanh(0.7 * x) * w + b if kind == DYT else x


@pytest.mark.parametrize("width", [4, 252, 256, 260, 1024, 1028, 1030, 2048, 2052, 4096, 4100])
@pytest.mark.parametrize("kind", [RMS, DYT, LAYER, COPY])
@pytest.mark.parametrize("there", [0, 1])
def test_row_passes(width, kind, there):
    """A thread sums up to 16 values, then come 13 levels of the block's tree: 29 roundings of 2^-24, 1.7e-6; as much again for the mean or the root and the
    products around them.  bf16 outputs: 2^-8."""
    lib = H.lib()
    R = 3
    g = torch.Generator("cuda").manual_seed(width + kind)
    t = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, a, c, e, tap = t(R, width), t(R, width), t(R, width), t(R, width), torch.zeros(R, width, device="cuda")
    ab, v, w, b, yw = t(width), t(width), t(width), t(width), t(width)
    n = H.Norm(kind=kind, w=H.ptr(w), b=H.ptr(b), w_offset=0.5, alpha=0.7)
    o = lambda p: C.c_void_p(H.ptr(p) if there else None)
    p = lambda q: C.c_void_p(H.ptr(q))
    for dtype, out_t, tol in ((H.F32, torch.float32, 4e-6), (H.BF16, torch.bfloat16, 2 ** -8)):
        x1, x2 = x.clone(), x.clone()
        ldo = 2 * width if width % 2 == 0 else width
        out = torch.zeros(R, ldo, device="cuda", dtype=out_t)
        lib.check(lib.c.tha_hyb_add_norm(None, dtype, p(x1), p(a), o(ab), F(0.8), o(c), F(-1.5), o(e), o(v), C.byref(n), F(1e-5), p(out), L(ldo), R, width))
        want = x.double() + 0.8 * (a.double() + there * ab.double()) + there * (-1.5 * c.double() + e.double() + v.double())
        check(x1, want, 4e-6)
        check(out[:, :width], norm(want, kind, w.double(), b.double()), tol)
        lib.check(lib.c.tha_hyb_block_finish(None, dtype, p(x2), p(a), o(ab), o(c), F(0.8), p(yw), F(1e-5), o(tap), o(e), o(v), C.byref(n), p(out), L(ldo), R, width))
        y = c.double()
        mid = x.double() + 0.8 * (a.double() + there * ab.double()) + there * 0.8 * y / (y.square().mean(-1, keepdim=True) + 1e-5).sqrt() * yw.double()
        want = mid + there * (e.double() + v.double())
        if there:
            check(tap, mid, 4e-6)
        check(x2, want, 4e-6)
        check(out[:, :width], norm(want, kind, w.double(), b.double()), tol)


def check(got, want, tol):
    torch.cuda.synchronize()
    assert float((got.double() - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))
