"""Decode attention with RoPE inside (csrc/attention.cu) at the sizes that pick its forms -- persistent groups of 8, 4 and 2 warps in one round and in
several, the deep form of few CTAs with and without splits of the time axis -- with ragged, idle and first positions, dense and paged,
against a float64 statement; and the persistent form against the plain one: the same bits."""
import numpy as np
import pytest
import torch

import llama64
from pkgload import load_pkg

pytestmark = pytest.mark.gpu


def step(B, heads, kv_heads, hs, seq_len, positions, block=0):
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, 2304, 1, heads, kv_heads, 80, seq_len)      # too wide a feed-forward for the one-launch step of small models
    w = eng.device_random_weights(cfg, seed=3, std=cfg.dim ** -0.5)
    rng = np.random.default_rng(B)
    pages = None
    if block:
        per = -(-seq_len // block)
        pages = eng.PagedKV(cfg, B, B * per + 3, block)
        pages.set_table(rng.permutation(pages.n_blocks)[:B * per].reshape(per, B).T.copy())
    e = eng.Engine(w, B, with_att=False, paged=pages)
    g = torch.Generator(device="cuda").manual_seed(5)
    e.state.key_cache.normal_(generator=g)
    e.state.value_cache.normal_(generator=g)
    pos = np.asarray(positions, np.int32)
    tok = rng.integers(0, cfg.vocab_size, B).astype(np.int32)
    table = pages.table.long() if pages else None

    def before(cache, s, l, n):
        if table is None:
            return cache[s, l, :n]
        return cache[table[s, :-(-n // block)], l].reshape(-1, cache.shape[-1])[:n] if n else cache[0, l, :0]

    kc, vc = e.state.key_cache.clone(), e.state.value_cache.clone()
    live = [b for b in range(B) if pos[b] >= 0]
    want, k, v = llama64.forward(cfg, w.t, lambda c, s, l, n: before(kc if c == "k" else vc, s, l, n), [(b, int(pos[b]), [int(tok[b])]) for b in live])
    logits = torch.full((B, cfg.vocab_size), 7.0, device="cuda")
    nxt = torch.zeros(B, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):      # the second replays the captured step
        e.decode_step(torch.from_numpy(tok).cuda(), torch.from_numpy(pos).cuda(), logits, nxt)
        torch.cuda.synchronize()
    # contexts of up to 1300 rows summed in fp32 in groups of four, products in 3xTF32: a few 1e-6 of a row each; sixteen times that
    assert float(((logits[live].double() - want).norm(dim=1) / want.norm(dim=1)).max()) < 5e-5
    for i, b in enumerate(live):
        row = lambda c: before(c, b, 0, int(pos[b]) + 1)[-1]
        assert float((row(e.state.key_cache).double() - k[i, 0]).norm() / k[i, 0].norm()) < 3e-5
        assert float((row(e.state.value_cache).double() - v[i, 0]).norm() / v[i, 0].norm()) < 3e-5


def ragged(B, longest):
    p = np.random.default_rng(B + longest).integers(0, longest, B)
    p[: 6] = [longest - 1, 0, -1, 1, 31, 32]
    return p


@pytest.mark.parametrize("block", [0, 16])
@pytest.mark.parametrize("B,heads,kv_heads,hs,seq_len", [
    (80, 8, 8, 64, 200),        # groups of 8 warps, one round
    (130, 4, 4, 128, 1040),     # and two, taken by their contexts: the cache is long enough
    (40, 16, 4, 32, 300),       # four query heads to a key head within a segment
    (200, 8, 8, 64, 150),       # groups of 4
    (250, 6, 6, 128, 100),      # groups of 2
    (9, 8, 8, 64, 700),         # few CTAs, the time axis in eight
    (37, 8, 8, 64, 130),        # few CTAs, not split
])
def test_against_float64(B, heads, kv_heads, hs, seq_len, block):
    step(B, heads, kv_heads, hs, seq_len, ragged(B, seq_len), block)


@pytest.mark.parametrize("B,heads,hs", [(80, 8, 64), (200, 8, 64), (250, 6, 128)])
def test_all_at_one_position(B, heads, hs):
    for p in (0, 3, 64):
        step(B, heads, heads, hs, 80, [p] * B)
