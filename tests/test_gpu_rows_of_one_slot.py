"""Single rows of one layer-program step that see each other's keys: two sequences with the same slot, or slots whose block tables share blocks.  The attention of single rows
(csrc/hybrid_attn_row.cu) asks for cache rows ahead of the kernel that writes the step's own, so it has to know all of these; against the same rows in steps of their own."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import torch

import hyb_cabi as H

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LAYERS = """
#include <string.h>
#include "tha_hybrid.h"
static tha_hyb_layer_t L[2];
const void* layers(const void* w_in, const float* norm, const void* w_o, int heads, int kv_heads, int dim) {
  memset(L, 0, sizeof L);
  for (int i = 0; i < 2; i++) {
    L[i].mixer = THA_MIX_ATTN; L[i].block = THA_BLOCK_SEQUENTIAL; L[i].has_ff = THA_FF_NONE; L[i].res_mult = 1.0f;
    L[i].norm1.kind = THA_NORM_RMS; L[i].norm1.w = norm;
    L[i].w_in = w_in; L[i].n_in = (heads + 2 * kv_heads) * dim;
    tha_attn_t* a = &L[i].attn;
    a->heads = heads; a->kv_heads = kv_heads; a->dim = a->vdim = dim; a->rot = -1; a->eps = 1e-5f; a->scale = 0.3f; a->cache_layer = i;
    a->o_k = heads * dim; a->o_v = (heads + kv_heads) * dim; a->w_o = w_o;
  }
  return L;
}
"""


@pytest.fixture(scope="module")
def layers(tmp_path_factory):
    d = tmp_path_factory.mktemp("layers")
    (d / "a.c").write_text(LAYERS)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"), "-o", str(d / "a.so"), str(d / "a.c")])
    f = C.CDLL(str(d / "a.so")).layers
    f.restype, f.argtypes = H.P, [H.P, H.P, H.P, H.I, H.I, H.I]
    return f


@pytest.mark.parametrize("dtype,tol", [(H.F32, 1e-5), (H.BF16, 2e-2)])
@pytest.mark.parametrize("heads,kv_heads", [(16, 4), (8, 4), (4, 4)])
@pytest.mark.parametrize("shared", ["slot", "blocks"])
@pytest.mark.parametrize("first,n", [(0, 2), (31, 2), (95, 40), (300, 3)])
def test_rows_that_see_each_other(layers, dtype, tol, heads, kv_heads, shared, first, n):
    lib, width, vocab, dim, block = H.lib(), 256, 64, 64, 16
    t = torch.float32 if dtype == H.F32 else torch.bfloat16
    g = torch.Generator("cuda").manual_seed(first + n + heads)
    mat = lambda r, c: (torch.randn(r, c, device="cuda", generator=g) * c ** -0.5).to(t)
    embed, head, w_in, w_o = mat(vocab, width), mat(vocab, width), mat((heads + 2 * kv_heads) * dim, width), mat(width, heads * dim)
    one = torch.ones(width, device="cuda")
    m = H.Model(dtype=dtype, width=width, vocab=vocab, n_layers=2, eps=1e-6, embed=H.ptr(embed), final_norm=H.Norm(0, H.ptr(one), None, 0.0, 0.0), head=H.ptr(head),
                layers=layers(H.ptr(w_in), H.ptr(one), H.ptr(w_o), heads, kv_heads, dim))
    blocks = 32
    ids = np.random.default_rng(1).permutation(blocks).astype(np.int32)
    table = torch.from_numpy(np.tile(ids, (n, 1))).cuda()
    pools = [torch.randn(blocks, 2, block, kv_heads * dim, device="cuda", generator=g) for _ in range(2)]
    tokens = torch.randint(0, vocab, (n,), device="cuda", generator=g, dtype=torch.int32)
    stream = torch.cuda.Stream()

    def step(kv, seqs, toks, out):
        r, keep = H.rows_of(seqs)
        keep[0].copy_(toks)
        want = torch.arange(len(seqs), device="cuda", dtype=torch.int32)
        torch.cuda.synchronize()
        lib.check(lib.c.tha_hyb_step(stream.cuda_stream, m, r, kv, H.States(), len(seqs), H.ptr(want), H.ptr(out), None))
        torch.cuda.synchronize()

    seqs = [(i if shared == "blocks" else 0, first + i, 1) for i in range(n)]
    got, want = torch.zeros(n, vocab, device="cuda"), torch.zeros(n, vocab, device="cuda")
    caches = []
    for together in (True, False):
        k, v = (p.clone() for p in pools)
        kv = H.Kv(k.data_ptr(), v.data_ptr(), table.data_ptr(), blocks, block, 2, kv_heads * dim)
        if together:
            step(kv, seqs, tokens, got)
        else:
            # layer by layer the rows of one step see the keys that it writes: one row after the other does, too, as each is causal
            for i in range(n):
                step(kv, seqs[i:i + 1], tokens[i:i + 1], want[i:i + 1])
        caches.append((k, v))
    rel = lambda a, b: float((a.double() - b.double()).norm() / b.double().norm())
    assert torch.isfinite(got).all() and rel(got, want) < tol
    for a, b in zip(*caches):
        assert rel(a, b) < tol
