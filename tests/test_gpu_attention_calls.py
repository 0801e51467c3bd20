"""tha_hyb_attn called by itself (csrc/hybrid_ops.cu, csrc/hybrid_attn_row.cu) against a float64 statement of its definition: which form a row takes,
how many runs a context is cut into, and how the runs meet."""
import numpy as np
import pytest
import torch

import hyb_cabi as H

pytestmark = pytest.mark.gpu
BLOCK = 64


class Cache:
    """Random cache rows of a few slots in a fragmented pool, and the float64 attention over them."""

    def __init__(self, slots, longest, kv_heads, dim, vdim, seed=0):
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.per = -(-longest // BLOCK)
        self.kv_dim = kv_heads * max(dim, vdim)
        self.k = torch.randn(slots, self.per * BLOCK, kv_heads, dim, device="cuda", generator=g)
        self.v = torch.randn(slots, self.per * BLOCK, kv_heads, vdim, device="cuda", generator=g)
        self.slots = slots

    def struct(self):
        order = torch.from_numpy(np.random.default_rng(1).permutation(self.slots * self.per)).cuda()
        pools = []
        for rows in (self.k, self.v):
            pool = torch.zeros(self.slots * self.per, BLOCK, self.kv_dim, device="cuda")
            flat = rows.flatten(2)
            pool[order] = torch.nn.functional.pad(flat, (0, self.kv_dim - flat.shape[-1])).reshape(self.slots * self.per, BLOCK, self.kv_dim)
            pools.append(pool)
        table = order.to(torch.int32).reshape(self.slots, self.per).contiguous()
        self.keep = pools + [table]
        return H.Kv(H.ptr(pools[0]), H.ptr(pools[1]), H.ptr(table), self.per, BLOCK, 1, self.kv_dim)


def want(a, cache, q, seqs, sink=None):
    """[rows, heads, vdim] in float64."""
    out, at, group = [], 0, a.heads // a.kv_heads
    for slot, p0, n in seqs:
        K, V = (t[slot, :p0 + n].double().repeat_interleave(group, 1) for t in (cache.k, cache.v))
        s = torch.einsum("nhd,thd->hnt", q[at:at + n].double(), K) * a.scale
        t, p = torch.arange(p0 + n, device="cuda"), torch.arange(p0, p0 + n, device="cuda")[:, None]
        s = s.masked_fill((t > p) | ((p - t >= a.window) & (t >= a.keep_first) if a.window else t < 0), float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None, None].expand(-1, n, 1)], -1)
            V = torch.cat([V, torch.zeros_like(V[:1])])
        out.append(torch.einsum("hnt,the->nhe", torch.softmax(s, -1), V))
        at += n
    return torch.cat(out)


def run(dtype, a, cache, q, seqs, scratch_floats):
    lib = H.lib()
    r, keep = H.rows_of(seqs)
    kv = cache.struct()
    out = torch.full((r.n_rows, a.heads, a.vdim), float("nan"), device="cuda", dtype=torch.float32 if a.out_f32 or dtype == H.F32 else torch.bfloat16)
    # exactly as long as said: what lies behind it keeps its value
    scratch = torch.full((scratch_floats + 1024,), 3.25, device="cuda")
    torch.cuda.synchronize()
    lib.check(lib.c.tha_hyb_attn(None, dtype, a, r, kv, H.ptr(q), H.ptr(out), H.ptr(scratch) if scratch_floats else None, scratch_floats))
    torch.cuda.synchronize()
    assert bool((scratch[scratch_floats:] == 3.25).all())
    return out


def rel(got, exact):
    return float((got.double() - exact).norm() / exact.norm())


SINGLES = [(2, 5, 1), (1, 0, 300), (0, 700, 1), (3, 62, 2), (4, 0, 1)]


@pytest.mark.parametrize("dtype", [H.BF16, H.F32])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(8, 2, 64, 64), (8, 1, 128, 128), (6, 2, 32, 96)])
@pytest.mark.parametrize("seqs,scratch", [(SINGLES, 0), (SINGLES, 16), ([(0, 700, 1), (1, 0, 1100)], 16), ([(1, 3, 90), (0, 700, 1)], 2), ([(0, 700, 1), (2, 690, 1)], 16)])
def test_a_decoded_row_whatever_else_is_in_the_step(dtype, heads, kv_heads, dim, vdim, seqs, scratch):
    """A sequence with one row is computed in fp32 alone and beside prompt portions, which the tiled forms round to bf16 in that number format.
    fp32 sums of at most 701 products of order one: 1e-6; bf16 weights and values: 2^-9 each, less over the keys."""
    a = H.Attn(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, rot=-1, scale=dim ** -0.5, out_f32=1)
    cache = Cache(5, 1101, kv_heads, dim, vdim)
    n = sum(s[2] for s in seqs)
    q = torch.randn(n, heads, dim, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)) * 2
    got = run(dtype, a, cache, q, seqs, scratch * n * heads * (vdim + 2))
    exact = want(a, cache, q, seqs)
    at = 0
    for s in seqs:
        part = slice(at, at + s[2])
        at += s[2]
        assert rel(got[part], exact[part]) < (1e-6 if s[2] == 1 or dtype == H.F32 else 6e-3), s
        if s[2] == 1:
            alone = run(dtype, a, cache, q[part].contiguous(), [s], 32 * heads * (vdim + 2))
            assert rel(got[part], alone.double()) < 1e-6, s


# the runs of a single row's context: 66 tiles of 32 keys in 22 runs of three and ten that get none; 64 tiles in 32 runs of two; what fits the scratch
@pytest.mark.parametrize("pos,runs", [(2100, 32), (2047, 32), (2047, 7), (2047, 2), (2047, 1), (2047, 0), (130, 32)])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,window,keep_first", [(2, 1, 64, 128, 0, 0), (3, 1, 128, 32, 0, 0), (2, 2, 96, 96, 1500, 40)])
@pytest.mark.parametrize("dtype,out_f32", [(H.BF16, 1), (H.BF16, 0), (H.F32, 0)])
def test_runs_of_a_single_row(dtype, out_f32, heads, kv_heads, dim, vdim, window, keep_first, pos, runs):
    a = H.Attn(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, rot=-1, scale=dim ** -0.5, out_f32=out_f32, window=window, keep_first=keep_first)
    cache = Cache(2, 2101, kv_heads, dim, vdim)
    seqs = [(1, pos, 1)]
    q = torch.randn(1, heads, dim, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4)) * 2
    got = run(dtype, a, cache, q, seqs, runs * heads * (vdim + 2))
    # fp32 throughout; rounded to bf16 at the end where that is asked for: eight significant bits, so half a unit is up to 2^-8 of a value
    assert rel(got, want(a, cache, q, seqs)) < (2e-6 if dtype == H.F32 or out_f32 else 2.0 ** -8)


@pytest.mark.parametrize("form", ["runs", "sink"])
def test_large_scores(form):
    """Scores around 65536 that differ by whole 64ths, a different largest one in every run of keys: every score, weight exponent and value is
    exact, so the result carries the 16 bits of the weights (hi + lo) and fp32 sums.  An exponent's offset rounded per run (65536 log2(e)
    has a spacing of 2^-7) would move the runs, or the keys and the sink,
    against one another by up to 0.3 %."""
    heads, dim, p0 = 2, 64, 1023
    a = H.Attn(heads=heads, kv_heads=1, dim=dim, vdim=dim, rot=-1, scale=1.0, out_f32=1, fp32_scores=1)
    cache = Cache(1, p0 + 2, 1, dim, dim)
    rng = np.random.default_rng(7)
    t = np.arange(cache.k.shape[1])
    run_of = t // 96
    x = (rng.integers(0, 96, run_of.max() + 1)[run_of] + t * 37 % 32) / 64.0
    cache.k.zero_()
    cache.k[0, :, 0, 0] = 65536.0
    cache.k[0, :, 0, 1] = torch.from_numpy(x).cuda().float()
    cache.v[0, :, 0] = torch.from_numpy(rng.choice([-1.0, 1.0], (run_of.max() + 1, dim))[run_of]).cuda().float()
    q = torch.zeros(2, heads, dim, device="cuda")
    q[:, :, :2] = 1.0
    sink = torch.tensor([65543.5, 65544.0 + 5 / 64], device="cuda") if form == "sink" else None
    a.sink = H.ptr(sink)
    seqs = [(0, p0, 2)]                     # a portion of two rows: the tensor-core form
    got = run(H.BF16, a, cache, q, seqs, 0 if form == "sink" else 16 * 2 * heads * (dim + 2))
    assert rel(got, want(a, cache, q, seqs, sink)) < 5e-5
