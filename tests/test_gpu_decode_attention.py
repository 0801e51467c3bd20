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
    for _ in range(3):      # the second may take another form, by the contexts that the first found; the third replays it
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


FUSED, DEEP, PERSISTENT = 1, 2, 3


@pytest.mark.parametrize("block", [0, 16])
@pytest.mark.parametrize("weights", ["f32", "q8", "bf16"])
@pytest.mark.parametrize("B,heads,kv_heads,hs,plain", [
    (40, 8, 8, 64, DEEP),           # 160 pairs of slot and segment
    (80, 8, 8, 64, FUSED),          # 320, one round of groups of 8 warps
    (130, 4, 4, 128, FUSED),        # 520, a poor second round
    (100, 16, 4, 32, FUSED),        # 400, four query heads to a key head within a segment
    (200, 8, 8, 64, FUSED),         # 800, groups of 4
    (250, 6, 6, 128, FUSED),        # 1500, groups of 2
])
def test_forms_give_the_same_bits(B, heads, kv_heads, hs, plain, weights, block):
    """A step whose positions are on the device takes the form that the contexts of the step before it ask for: the same step behind short uniform contexts
    and behind long ragged ones.  Given host positions it goes by its own."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    seq_len = 720
    cfg = ck.Config(heads * hs, 2304, 1, heads, kv_heads, 80, seq_len)
    w = eng.DeviceWeightsBF16.random(cfg, seed=3) if weights == "bf16" else eng.device_random_weights(cfg, q8=weights == "q8", seed=3, gs=64)
    rng = np.random.default_rng(B)
    pages = None
    if block:
        per = seq_len // block
        pages = eng.PagedKV(cfg, B, B * per, block)
        pages.set_table(rng.permutation(B * per).reshape(B, per).astype(np.int32))
    e = eng.Engine(w, B, with_att=False, paged=pages)
    g = torch.Generator(device="cuda").manual_seed(5)
    caches = e.state.key_cache, e.state.value_cache
    for c in caches:
        c.normal_(generator=g)
    kept = [c.clone() for c in caches]
    tok = rng.integers(0, cfg.vocab_size, B).astype(np.int32)
    pos = ragged(B, seq_len).astype(np.int32)
    short, long = np.zeros(B, np.int32), np.where(np.arange(B) % 5 == 0, seq_len - 1, 3).astype(np.int32)
    tok_d = torch.from_numpy(tok).cuda()
    nxt = torch.zeros(B, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()

    def step(p):
        for c, k in zip(caches, kept):
            c.copy_(k)
        logits = torch.full((B, cfg.vocab_size), 7.0, device="cuda")
        p = torch.from_numpy(p).cuda()
        torch.cuda.synchronize()
        e.decode_step(tok_d, p, logits, nxt, stream=stream)
        form = e.last_step_attention()
        torch.cuda.synchronize()
        return form, [logits[torch.from_numpy(pos >= 0).cuda()]] + [c.clone() for c in caches]

    seen = []
    for before, form in ((short, plain), (long, PERSISTENT), (long, PERSISTENT), (short, plain)):
        step(before)
        took, out = step(pos)
        assert took == form
        seen.append(out)
    for out in seen[1:]:
        assert all(torch.equal(a, b) for a, b in zip(out, seen[0]))
    host = torch.empty(B, cfg.vocab_size).pin_memory()
    for p, form in ((short, plain), (long, PERSISTENT), (short, plain)):
        e.forward_batch(tok, p, host, stream=stream)
        assert e.last_step_attention() == form
    if pages:
        pages.close()
