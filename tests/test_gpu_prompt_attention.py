"""fp32 prompt attention (csrc/attn_prefill.cu) inside tha_prefill_f32: prompts at the edges of query and key tiles, both tile heights,
every head size, grouped queries, portions behind a context, against a float64 statement."""
import numpy as np
import pytest
import torch

import llama64
from pkgload import load_pkg

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("heads,kv_heads,hs", [(8, 8, 16), (4, 2, 32), (2, 2, 64), (4, 1, 128), (2, 2, 128)])
@pytest.mark.parametrize("lens,start", [([1], 0), ([64, 63, 65], 0), ([127, 1, 129], 70), ([192], 0), ([193, 383], 0), ([500], 131), ([2, 640, 66], 1)])
def test_prompts(heads, kv_heads, hs, lens, start):
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, 96, 2, heads, kv_heads, 80, start + max(lens) + 3)
    if not load_pkg("cabi").lib().c.tha_prefill_supported(eng.c_config(cfg)):
        pytest.skip("the decode attention does not take this head layout")
    # queries and keys of order one: a score s of magnitude S carries the products' error (1e-6) times S into its weight, and 0.15 here (S up to 60
    # at 512 channels) gave 4e-5
    w = eng.device_random_weights(cfg, seed=3, std=cfg.dim ** -0.5)
    e = eng.Engine(w, len(lens), with_att=False)
    g = torch.Generator(device="cuda").manual_seed(5)
    e.state.key_cache.normal_(generator=g)
    e.state.value_cache.normal_(generator=g)
    rng = np.random.default_rng(7)
    seqs = [(i, start, rng.integers(0, cfg.vocab_size, n).astype(np.int32)) for i, n in enumerate(lens)]
    before = {"k": e.state.key_cache.clone(), "v": e.state.value_cache.clone()}
    logits = torch.empty(len(lens), cfg.vocab_size, device="cuda")
    torch.cuda.synchronize()
    e.prefill(seqs, logits)
    torch.cuda.synchronize()
    want, k, v = llama64.forward(cfg, w.t, lambda c, s, l, n: before[c][s, l, :n], seqs)
    # fp32 sums of up to 640 terms through two layers: a few 1e-6; 3xTF32 products the same
    assert rel(logits, want) < 3e-5
    at = 0
    for i, n in enumerate(lens):
        for which, got, exact in (("k", e.state.key_cache, k), ("v", e.state.value_cache, v)):
            assert rel(got[i, :, start:start + n], exact[at:at + n].transpose(0, 1)) < 3e-5
            other = torch.ones(cfg.seq_len, dtype=torch.bool)
            other[start:start + n] = False
            assert torch.equal(got[i][:, other], before[which][i][:, other])    # nothing else was written
        at += n


@pytest.mark.parametrize("heads,kv_heads,hs", [(8, 8, 16), (4, 2, 32), (2, 2, 64), (4, 1, 128)])
@pytest.mark.parametrize("lens,start,block", [([193, 383], 0, 16), ([500], 131, 16), ([700, 2], 5, 64), ([100, 90, 65], 70, 32)])
def test_paged_prompts(heads, kv_heads, hs, lens, start, block):
    """The same through a fragmented block table: several key tiles, so that the tile that is
    fetched ahead is looked up in the table too; blocks narrower than a key tile, and as wide."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, 96, 2, heads, kv_heads, 80, start + max(lens) + 3)
    if not load_pkg("cabi").lib().c.tha_prefill_supported(eng.c_config(cfg)):
        pytest.skip("the decode attention does not take this head layout")
    w = eng.device_random_weights(cfg, seed=3, std=cfg.dim ** -0.5)
    rng = np.random.default_rng(7)
    per = -(-cfg.seq_len // block)
    pages = eng.PagedKV(cfg, len(lens), len(lens) * per + 5, block)
    table = rng.permutation(pages.n_blocks)[:len(lens) * per].reshape(per, len(lens)).T.copy()
    pages.set_table(table)
    e = eng.Engine(w, len(lens), with_att=False, paged=pages)
    g = torch.Generator(device="cuda").manual_seed(5)
    pages.k.normal_(generator=g)
    pages.v.normal_(generator=g)
    seqs = [(i, start, rng.integers(0, cfg.vocab_size, n).astype(np.int32)) for i, n in enumerate(lens)]
    before = {"k": pages.k.clone(), "v": pages.v.clone()}
    at_table = torch.from_numpy(table).cuda()

    def rows(pool, s, n):
        """[layers, n, kv_dim]: rows 0 .. n - 1 of slot s"""
        return pool[at_table[s]].transpose(0, 1).flatten(1, 2)[:, :n]

    logits = torch.empty(len(lens), cfg.vocab_size, device="cuda")
    torch.cuda.synchronize()
    e.prefill(seqs, logits)
    torch.cuda.synchronize()
    want, k, v = llama64.forward(cfg, w.t, lambda c, s, l, n: rows(before[c], s, n)[l], seqs)
    assert rel(logits, want) < 3e-5             # as above
    at = 0
    for which, pool, exact in (("k", pages.k, k), ("v", pages.v, v)):
        at = 0
        for i, n in enumerate(lens):
            assert rel(rows(pool, i, start + n)[:, start:], exact[at:at + n].transpose(0, 1)) < 3e-5
            assert torch.equal(rows(pool, i, start), rows(before[which], i, start))
            at += n
        free = [b for b in range(pages.n_blocks) if b not in table]
        assert torch.equal(pool[free], before[which][free])
    pages.close()


TALL = [(64, 64, 16, [500], 3), (64, 8, 32, [193, 383], 0), (32, 32, 64, [1030], 5), (32, 8, 128, [700, 400], 70)]


@pytest.mark.parametrize("heads,kv_heads,hs,lens,start", TALL)
def test_tall_tiles(heads, kv_heads, hs, lens, start):
    """Many heads, which is where tiles of 128 rows are taken: ragged last tiles, a context in front."""
    test_prompts(heads, kv_heads, hs, lens, start)


@pytest.mark.parametrize("heads,kv_heads,hs,lens,start", TALL)
def test_tall_tiles_paged(heads, kv_heads, hs, lens, start):
    test_paged_prompts(heads, kv_heads, hs, lens, start, 16)
