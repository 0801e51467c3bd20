"""The forms of the layer program's row passes that hold a row in registers (csrc/hybrid_block.cu, csrc/hybrid_ops.cu) against the general ones, which take operands that
do not start on 16 bytes: the same order of every sum, so the same bits."""
import ctypes as C

import pytest
import torch

import hyb_cabi as H

pytestmark = pytest.mark.gpu
F, L = C.c_float, C.c_longlong
RMS, DYT, LAYER, COPY = range(4)


def both(run, moved):
    """run(operands) with the operands `moved` on 16 bytes and one float behind; what it returns must be the same bits."""
    got = []
    for shift in (0, 1):
        copies = []
        for t in moved:
            room = torch.zeros(t.numel() + 1, device="cuda", dtype=t.dtype)
            room[shift:shift + t.numel()] = t.flatten()
            copies.append(room[shift:shift + t.numel()].view(t.shape))
        got.append(run(copies))
        torch.cuda.synchronize()
    for a, b in zip(*got):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)


def p(t):
    return C.c_void_p(H.ptr(t))


@pytest.mark.parametrize("dtype,out_t", [(H.F32, torch.float32), (H.BF16, torch.bfloat16)])
@pytest.mark.parametrize("width", [4, 100, 256, 260, 1024, 1500, 2048, 3000, 4096])
@pytest.mark.parametrize("kind", [RMS, DYT, LAYER, COPY])
@pytest.mark.parametrize("there", [0, 1])
def test_residual_passes(dtype, out_t, width, kind, there):
    lib, R = H.lib(), 3
    g = torch.Generator("cuda").manual_seed(width + kind)
    t = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a, c, e, ab, v, w, b, yw = t(R, width), t(R, width), t(R, width), t(width), t(width), t(width), t(width), t(width)
    n = H.Norm(kind=kind, w=H.ptr(w), b=H.ptr(b), w_offset=0.5, alpha=0.7)
    o = lambda q: p(q if there else None)

    def add_norm(m):
        out = torch.zeros(R, width, device="cuda", dtype=out_t)
        lib.check(lib.c.tha_hyb_add_norm(None, dtype, p(m[0]), p(a), o(ab), F(0.8), o(c), F(-1.5), o(e), o(v), C.byref(n), F(1e-5), p(out), L(0), R, width))
        return m[0], out

    def finish(m):
        out, tap = torch.zeros(R, width, device="cuda", dtype=out_t), torch.zeros(R, width, device="cuda")
        lib.check(lib.c.tha_hyb_block_finish(None, dtype, p(m[0]), p(a), o(ab), o(c), F(0.8), p(yw), F(1e-5), p(tap), o(e), o(v), C.byref(n), p(out), L(0), R, width))
        return m[0], tap, out

    x = t(R, width)
    both(add_norm, [x])
    both(finish, [x])


@pytest.mark.parametrize("dtype,out_t", [(H.F32, torch.float32), (H.BF16, torch.bfloat16)])
@pytest.mark.parametrize("width", [4, 100, 256, 260, 1024, 1500, 2048, 3000, 4096])
def test_norm(dtype, out_t, width):
    lib, R = H.lib(), 3
    g = torch.Generator("cuda").manual_seed(width)
    w = torch.randn(width, device="cuda", generator=g)

    def run(m):
        out = torch.zeros(R, width, device="cuda", dtype=out_t)
        lib.check(lib.c.tha_hyb_rmsnorm(None, dtype, H.ptr(out), H.ptr(m[0]), H.ptr(w), 0.5, 1e-5, R, width, None))
        return (out,)

    both(run, [torch.randn(R, width, device="cuda", generator=g)])


@pytest.mark.parametrize("dtype,out_t", [(H.F32, torch.float32), (H.BF16, torch.bfloat16)])
@pytest.mark.parametrize("E", [4, 36, 64, 128, 132, 200, 256, 260, 512])
@pytest.mark.parametrize("gated,act", [(0, 0), (1, 0), (1, 1)])
def test_head_gate(dtype, out_t, E, gated, act):
    lib, R, heads = H.lib(), 5, 3
    g = torch.Generator("cuda").manual_seed(E)
    z, w = torch.randn(R, heads * E, device="cuda", generator=g), torch.randn(heads * E, device="cuda", generator=g)

    def run(m):
        out = torch.zeros(R, heads * E, device="cuda", dtype=out_t)
        lib.check(lib.c.tha_hyb_head_gate(None, dtype, p(out), p(m[0]), R, heads, E, 1, F(1e-5), p(w), 1, p(z if gated else None), L(heads * E), act))
        return (out,)

    both(run, [torch.randn(R, heads * E, device="cuda", generator=g)])


Wkv = H._struct("tha_wkv_t", [("heads dim rank", H.I), ("eps", H.F), ("mu", H.P), ("o_r o_k o_v o_g o_w1", H.I), ("w_w2 w0 u norm w_o", H.P), ("state_off shift_state_off", H.L)])


@pytest.mark.parametrize("dtype,t", [(H.F32, torch.float32), (H.BF16, torch.bfloat16)])
@pytest.mark.parametrize("rank", [8, 56, 64, 72, 128, 200, 256])
@pytest.mark.parametrize("rows", [1, 3, 4, 5, 8])
def test_decay_of_few_rows(dtype, t, rank, rows):
    """Up to eight rows against the tiles, which take a W2 that does not start on 16 bytes."""
    lib, heads, dim = H.lib(), 3, 26
    HD = heads * dim
    g = torch.Generator("cuda").manual_seed(rank + rows)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    ldp = 4 * HD + rank
    proj, w0, u, norm = rnd(rows, ldp), rnd(HD), rnd(HD), rnd(HD)
    w2 = (rnd(HD, rank) / rank ** 0.5).to(t)
    r, keep = H.rows_of([(0, 0, rows)])
    lib.c.tha_hyb_scan_state_floats.restype = L
    floats = lib.c.tha_hyb_scan_state_floats(heads, dim, dim)

    def run(m):
        state = torch.zeros(1, floats, device="cuda")
        decay, raw, out = torch.zeros(rows, HD, device="cuda"), torch.zeros(rows, HD, device="cuda"), torch.zeros(rows, HD, device="cuda", dtype=t)
        k = Wkv(heads=heads, dim=dim, rank=rank, eps=1e-5, o_r=0, o_k=HD, o_v=2 * HD, o_g=3 * HD, o_w1=4 * HD, w_w2=H.ptr(m[0]), w0=H.ptr(w0), u=H.ptr(u), norm=H.ptr(norm))
        st = H.States(H.ptr(state), state.shape[1])
        lib.check(lib.c.tha_hyb_wkv_scan(None, dtype, C.byref(k), C.byref(r), C.byref(st), p(proj), L(ldp), p(decay), p(raw), p(out), None, C.c_size_t(0)))
        return decay, raw, out

    both(run, [w2])
