"""Prompt portions on tcgen05 (csrc/hybrid_attn_tc.cu) through tha_hyb_attn_gated: every form of scores, both head sizes, groups that fill a block evenly and not,
ragged ends of blocks, of key tiles and of halves of them, portions behind a context, several sequences with short ones among them, against a
float64 statement on inputs that are exact in bf16."""
import ctypes as C

import numpy as np
import pytest
import torch

import hyb_cabi as H
import test_gpu_gavodra as G
from test_gpu_attention_calls import Cache, rel

pytestmark = pytest.mark.gpu
LONG = [(0, 0, 1)], [(0, 0, 2065)], [(1, 0, 1300), (0, 77, 900), (2, 5, 1), (3, 0, 33)], [(0, 1000, 1100), (1, 31, 1025)]


def want(a, cache, q, seqs, t):
    out, at, group = [], 0, a.heads // a.kv_heads
    for slot, p0, n in seqs:
        K, V = (x[slot, :p0 + n].double().repeat_interleave(group, 1) for x in (cache.k, cache.v))
        s = torch.einsum("nhd,thd->hnt", q[at:at + n].double(), K) * a.scale
        if a.softcap:
            s = a.softcap * torch.tanh(s / a.softcap)
        k, p = torch.arange(p0 + n, device="cuda"), torch.arange(p0, p0 + n, device="cuda")[:, None]
        if "rel" in t:
            s = s + t["rel"].double()[:, (p - k).clamp(0, a.rel_n - 1)]
        hidden = k > p
        if a.window:
            hidden = hidden | ((p - k >= a.window) & (k >= a.keep_first))
        if a.chunk:
            hidden = hidden | (k < p // a.chunk * a.chunk)
        s = s.masked_fill(hidden, float("-inf"))
        if "sink" in t:
            s = torch.cat([s, t["sink"].double()[:, None, None].expand(-1, n, 1)], -1)
            V = torch.cat([V, torch.zeros_like(V[:1])])
        o = torch.einsum("hnt,the->nhe", torch.softmax(s, -1), V)
        if "gate" in t:
            o = o * torch.sigmoid(t["gate"][at:at + n].double())[:, :, None]
        out.append(o)
        at += n
    return torch.cat(out)


@pytest.mark.parametrize("seqs", LONG)
@pytest.mark.parametrize("heads,kv_heads,dim", [(16, 4, 128), (6, 2, 128), (16, 16, 64), (8, 1, 64)])
@pytest.mark.parametrize("form", [dict(), dict(fp32_scores=1), dict(softcap=7.0, window=300), dict(rel=2048), dict(rel=40, window=500, keep_first=70),
                                  dict(fp32_scores=1, chunk=333, sink=1), dict(window=50, keep_first=10, gate=1)])
def test_portions(heads, kv_heads, dim, seqs, form):
    a = H.Attn()
    a.heads, a.kv_heads, a.dim, a.vdim, a.rot, a.scale, a.out_f32 = heads, kv_heads, dim, dim, -1, dim ** -0.5, 1
    for k in ("fp32_scores", "softcap", "window", "keep_first", "chunk"):
        setattr(a, k, form.get(k, 0))
    g = torch.Generator(device="cuda").manual_seed(heads + dim)
    R, longest = sum(n for _, _, n in seqs), max(p + n for _, p, n in seqs)
    cache = Cache(max(s for s, _, _ in seqs) + 1, longest, kv_heads, dim, dim)
    cache.k, cache.v = cache.k.bfloat16().float(), cache.v.bfloat16().float()
    q = torch.randn(R, heads, dim, device="cuda", generator=g).bfloat16().float()
    t = {}
    if "rel" in form:
        t["rel"] = torch.randn(heads, form["rel"], device="cuda", generator=g)
        a.rel, a.rel_n = t["rel"].data_ptr(), form["rel"]
    if "sink" in form:
        t["sink"] = torch.randn(heads, device="cuda", generator=g)
        a.sink = t["sink"].data_ptr()
    if "gate" in form:
        t["gate"] = torch.randn(R, heads, device="cuda", generator=g)
        a.head_gate, a.o_g = 1, 0
    lib = H.lib()
    lib.c.tha_hyb_attn_gated.argtypes = [H.P, H.I, C.POINTER(H.Attn), C.POINTER(H.Rows), C.POINTER(H.Kv), H.P, H.P, H.P, C.c_size_t, H.P, H.L]
    rows, keep = H.rows_of(seqs)
    kv = cache.struct()
    out = torch.full((R + 1, heads, dim), 7.0, device="cuda")
    floats = len(seqs) * (longest + 32) * kv_heads * dim + 64
    scratch = torch.full((floats + 1024,), float("nan"), device="cuda")     # what is not staged may hold anything
    exact = want(a, cache, q, seqs, t)
    # weights as two bf16 (2^-17 of themselves) or one (2^-9), random over hundreds of keys; the scores' fp32 sums below that
    tol = 1e-5 if a.fp32_scores or a.softcap or "rel" in form else 3e-3
    for given in (floats, 0):       # without scratch the step takes the other kernel
        out.fill_(7.0)
        torch.cuda.synchronize()
        lib.check(lib.c.tha_hyb_attn_gated(None, H.BF16, a, rows, kv, H.ptr(q), H.ptr(out), H.ptr(scratch) if given else None, given, H.ptr(t.get("gate")), heads))
        torch.cuda.synchronize()
        assert bool(torch.isnan(scratch[floats:]).all()) and bool((out[R] == 7.0).all())
        assert rel(out[:R], exact) < tol
    assert lib.c.tha_gemm_check_error() == 0


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("sink", [False, True])
def test_large_common_scores(dim, sink):
    """Scores of 4096 or 8192 and a few units apart, exact in fp32: what is left of the error is the weights' (two bf16, 2^-17 of themselves, over hundreds of
    keys).  Rounded in other units, as powers of two, such scores would be off by 1e-4 each."""
    a = H.Attn()
    a.heads, a.kv_heads, a.dim, a.vdim, a.rot, a.scale, a.out_f32, a.fp32_scores = 16, 16 * 64 // dim, dim, dim, -1, 2.0 ** -5, 1, 1
    R, g = 1100, torch.Generator(device="cuda").manual_seed(dim)
    cache = Cache(1, R, a.kv_heads, dim, dim)
    cache.v = cache.v.bfloat16().float()
    q = torch.randint(-3, 4, (R, a.heads, dim), device="cuda", generator=g).float()
    cache.k.copy_(torch.randint(-3, 4, cache.k.shape, device="cuda", generator=g).float())
    q[..., :dim // 2] = cache.k[..., :dim // 2] = 64.0
    t = {}
    if sink:
        t["sink"] = 64.0 * dim + torch.randint(-2, 6, (a.heads,), device="cuda", generator=g).float()
        a.sink = t["sink"].data_ptr()
    seqs = [(0, 0, R)]
    rows, keep = H.rows_of(seqs)
    lib = H.lib()
    lib.c.tha_hyb_attn_gated.argtypes = [H.P, H.I, C.POINTER(H.Attn), C.POINTER(H.Rows), C.POINTER(H.Kv), H.P, H.P, H.P, C.c_size_t, H.P, H.L]
    out, scratch = torch.empty(R, a.heads, dim, device="cuda"), torch.empty((R + 32) * a.kv_heads * dim + 64, device="cuda")
    exact = want(a, cache, q, seqs, t)
    for given in (scratch.numel(), 0):
        torch.cuda.synchronize()
        lib.check(lib.c.tha_hyb_attn_gated(None, H.BF16, a, rows, cache.struct(), H.ptr(q), H.ptr(out), H.ptr(scratch) if given else None, given, None, 0))
        torch.cuda.synchronize()
        assert rel(out, exact) < 1e-5


def test_more_position_tiles_than_a_grid_holds():
    """256 query heads to a key head: a tile of one position; 66000 of them take the other kernel."""
    a = H.Attn()
    a.heads, a.kv_heads, a.dim, a.vdim, a.rot, a.scale, a.window = 256, 1, 64, 64, -1, 0.125, 40
    R, g = 66000, torch.Generator(device="cuda").manual_seed(1)
    cache = Cache(1, R, 1, 64, 64)
    cache.k, cache.v = cache.k.bfloat16().float(), cache.v.bfloat16().float()
    q = torch.randn(R, 256, 64, device="cuda", generator=g)
    rows, keep = H.rows_of([(0, 0, R)])
    lib = H.lib()
    lib.c.tha_hyb_attn_gated.argtypes = [H.P, H.I, C.POINTER(H.Attn), C.POINTER(H.Rows), C.POINTER(H.Kv), H.P, H.P, H.P, C.c_size_t, H.P, H.L]
    out, scratch = torch.empty(R, 256, 64, device="cuda", dtype=torch.bfloat16), torch.empty((R + 32) * 64 + 64, device="cuda")
    torch.cuda.synchronize()
    lib.check(lib.c.tha_hyb_attn_gated(None, H.BF16, a, rows, cache.struct(), H.ptr(q), H.ptr(out), H.ptr(scratch), scratch.numel(), None, 0))
    torch.cuda.synchronize()
    for p in (0, 39, 31000, R - 1):
        K, V = (c[0, max(0, p - 39):p + 1, 0].double() for c in (cache.k, cache.v))
        exact = torch.softmax(q[p].bfloat16().double() @ K.T * a.scale, -1) @ V
        assert rel(out[p].float(), exact) < 6e-3       # weights and results rounded to bf16: 2^-9 each


@pytest.mark.parametrize("out_f32", [0, 1])
def test_results_on_an_8_byte_boundary(out_f32):
    """Its stores are of 16 bytes: such a call takes the other kernel, whose are of 4 and 8."""
    a = H.Attn()
    a.heads, a.kv_heads, a.dim, a.vdim, a.rot, a.scale, a.out_f32 = 16, 4, 64, 64, -1, 0.125, out_f32
    R, g = 1100, torch.Generator(device="cuda").manual_seed(1)
    cache = Cache(1, R, a.kv_heads, a.dim, a.dim)
    cache.k, cache.v = cache.k.bfloat16().float(), cache.v.bfloat16().float()
    q = torch.randn(R, a.heads, a.dim, device="cuda", generator=g).bfloat16().float()
    seqs = [(0, 0, R)]
    rows, keep = H.rows_of(seqs)
    lib = H.lib()
    lib.c.tha_hyb_attn_gated.argtypes = [H.P, H.I, C.POINTER(H.Attn), C.POINTER(H.Rows), C.POINTER(H.Kv), H.P, H.P, H.P, C.c_size_t, H.P, H.L]
    scratch = torch.empty((R + 32) * a.kv_heads * a.dim + 64, device="cuda")
    exact, n = want(a, cache, q, seqs, {}), q.numel()
    buf = torch.full((n + 8,), 7.0, device="cuda", dtype=torch.float32 if out_f32 else torch.bfloat16)
    for skip in (0, 2 if out_f32 else 4):
        out = buf[skip:skip + n]
        torch.cuda.synchronize()
        lib.check(lib.c.tha_hyb_attn_gated(None, H.BF16, a, rows, cache.struct(), H.ptr(q), H.ptr(out), H.ptr(scratch), scratch.numel(), None, 0))
        torch.cuda.synchronize()
        assert rel(out.view(R, a.heads, a.dim).float(), exact) < (3e-3 if out_f32 else 4e-3)


@pytest.mark.parametrize("lengths", [[64], [100, 128, 64]])
def test_the_output_product_behind_it(tmp_path, lengths):
    """Whole steps with heads of 64: a block of the attention and one of the product behind it, both of which allocate TMEM, fit an SM side by side."""
    b = G.one_layer(tmp_path, G.attention(heads=64, kv_heads=8, dim=64, vdim=64, scale=0.125), width=4096)
    prompts = [G.tokens_for(b, n, n) for n in lengths]
    e = b.engine("bfloat16")
    for turn in range(3):
        names = ["%d.%d" % (turn, i) for i in range(len(lengths))]
        got = e.step([(r, t, list(range(len(t)))) for r, t in zip(names, prompts)])
        for r in names:
            e.finish(r)
        assert G.rel_err(got, np.concatenate([b.ref(t)[0] for t in prompts])) < G.BF16_TOL
