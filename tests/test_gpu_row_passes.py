"""The residual passes that hold a row in registers (csrc/hybrid_block.cu) against float64: widths on both sides of a part of the row a thread
more, of the general form (not a multiple of four, more than 4096), every norm and every operand there and not there."""
import ctypes as C

import pytest
import torch

import hyb_cabi as H
import test_gpu_logulix as TL

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


@pytest.mark.parametrize("width", [4, 252, 256, 260, 1024, 1028, 1030, 2052, 4096, 4100])
@pytest.mark.parametrize("top", [0, 3])
def test_norm_of_rows_and_post_norm(width, top):
    """Sums as above."""
    lib = H.lib()
    R = 3
    g = torch.Generator("cuda").manual_seed(width + top)
    t = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, d, w, down, wt = t(R, width), t(R, width), t(width), t(R * 3, width), t(R, 3)
    gate = t(R, 5)
    inv = torch.randperm(R * 3, device="cuda", generator=g).int()
    rows = torch.tensor([2, 0, 2], device="cuda", dtype=torch.int32)
    n = H.Norm(kind=RMS, w=H.ptr(w), w_offset=0.5)
    p = lambda q: C.c_void_p(H.ptr(q))
    for dtype, out_t, tol in ((H.F32, torch.float32, 4e-6), (H.BF16, torch.bfloat16, 2 ** -8)):
        out = torch.zeros(R, width, device="cuda", dtype=out_t)
        lib.check(lib.c.tha_hyb_norm(None, dtype, p(out), p(x), C.byref(n), F(1e-5), R, width, p(rows)))
        check(out, norm(x.double()[rows.long()], RMS, w.double(), None), tol)
        x1, tap = x.clone(), torch.zeros_like(x)
        lib.check(lib.c.tha_hyb_post_norm(None, dtype, p(x1), p(d), p(gate), L(5), top, p(wt) if top else None, p(inv) if top else None, p(down) if top else None, F(0.8),
                                          C.byref(n), F(1e-5), p(tap), p(out), R, width))
        y = d.double() * torch.sigmoid(gate.double()[:, :1])
        if top:
            y = y + (wt.double()[:, :, None] * down.double()[inv.long()].reshape(R, 3, width)).sum(1)
        want = x.double() + 0.8 * norm(y, RMS, w.double(), None)
        for got, lim in ((x1, 4e-6), (tap, 4e-6), (out, tol)):
            check(got, want, lim)


@pytest.mark.parametrize("E", [4, 12, 60, 64, 65, 128, 132, 256, 260, 512, 516])
@pytest.mark.parametrize("per_head,gated,act", [(0, 1, 0), (1, 1, 1), (1, 0, 0)])
def test_head_gate(E, per_head, gated, act):
    """Up to 16 values a lane and five levels: 21 roundings of 2^-24, three times that with the root, the sigmoid and the products."""
    lib = H.lib()
    R, heads = 5, 3
    g = torch.Generator("cuda").manual_seed(E)
    o, z = torch.randn(R, heads * E, device="cuda", generator=g), torch.randn(R, heads * E + 4 - heads * E % 4, device="cuda", generator=g)
    w = torch.randn(heads * E, device="cuda", generator=g)
    for dtype, out_t, tol in ((H.F32, torch.float32, 4e-6), (H.BF16, torch.bfloat16, 2 ** -8)):
        out = torch.zeros(R, heads * E, device="cuda", dtype=out_t)
        for do_norm in (0, 1):
            lib.check(lib.c.tha_hyb_head_gate(None, dtype, C.c_void_p(H.ptr(out)), C.c_void_p(H.ptr(o)), R, heads, E, do_norm, F(1e-5), C.c_void_p(H.ptr(w)), per_head,
                                              C.c_void_p(H.ptr(z) if gated else None), L(z.shape[1]), act))
            v = o.double().reshape(R, heads, E)
            if do_norm:
                v = v / (v.square().mean(-1, keepdim=True) + 1e-5).sqrt() * (w.double().reshape(heads, E) if per_head else w.double()[:E])
            if gated:
                zd = z.double()[:, :heads * E].reshape(R, heads, E)
                v = v * torch.sigmoid(zd) * (zd if act else 1)
            check(out, v.reshape(R, -1), tol)


@pytest.mark.parametrize("rank", [7, 8, 40, 72, 256, 264])
@pytest.mark.parametrize("rows", [1, 7, 8, 9])
def test_decay_of_few_rows(tmp_path, rank, rows):
    """Both sides of the rule: up to eight rows, ranks of up to 256 that are a multiple of eight; portions of `rows` tokens."""
    b = TL.Built(tmp_path, TL.model([TL.wkv(TL.dense(40), heads=3, dim=26)]), 7, rank=rank)
    toks = TL.tokens_for(b, 27, 2)
    assert TL.rel_err(TL.feed(b.engine(), "a", toks, [rows]), b.ref(toks)[0]) < TL.F32_TOL


def check(got, want, tol):
    torch.cuda.synchronize()
    assert float((got.double() - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))
