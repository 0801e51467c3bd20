"""The decode step of a few slots as one kernel (csrc/megastep.cu), whose phases hand each other tagged words: steps of models of different shapes in turn (they share
the words' memory), contexts around the splits of its attention, idle slots, CTAs without a share of a phase; against float64."""
import numpy as np
import pytest
import torch

import llama64
from pkgload import load_pkg

pytestmark = pytest.mark.gpu


def model(heads, hs, kv_heads, hidden, layers, slots, seed):
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, hidden, layers, heads, kv_heads, 130, 1024)
    w = eng.device_random_weights(cfg, seed=seed, std=cfg.dim ** -0.5)
    e = eng.Engine(w, slots, with_att=False)
    g = torch.Generator(device="cuda").manual_seed(seed)
    e.state.key_cache.normal_(0.0, 1.0, generator=g)
    e.state.value_cache.normal_(0.0, 1.0, generator=g)
    return cfg, w, e


def step(cfg, w, e, pos, rng):
    toks = rng.integers(0, cfg.vocab_size, len(pos)).astype(np.int32)
    keys, values = e.state.key_cache.clone(), e.state.value_cache.clone()
    got = torch.as_tensor(e.forward_batch(toks, np.array(pos, np.int32)))
    assert e.last_step_launches() == 1
    live = [b for b, t in enumerate(pos) if t >= 0]
    seqs = [(b, pos[b], toks[b:b + 1]) for b in live]
    want, k, v = llama64.forward(cfg, w.t, lambda c, s, l, n: (keys if c == "k" else values)[s, l, :n], seqs)
    rel = lambda a, b: float((a.double() - b.double()).norm() / b.double().norm())
    # fp32 sums of 32 to 2048 terms in warps of 32 lanes: below 1e-6 each, through a few layers; and the angles of the rotation, fp32 products of the position: off by up to
    # position 2^-24, which rotates a key by as much
    tol = 1e-5 + max(pos) * 2.0 ** -24
    assert rel(got[live].cuda(), want) < tol
    for i, b in enumerate(live):
        assert rel(e.state.key_cache[b, :, pos[b]], k[i]) < tol and rel(e.state.value_cache[b, :, pos[b]], v[i]) < tol
        keys[b, :, pos[b]], values[b, :, pos[b]] = e.state.key_cache[b, :, pos[b]], e.state.value_cache[b, :, pos[b]]
    assert torch.equal(keys, e.state.key_cache) and torch.equal(values, e.state.value_cache)


@pytest.mark.parametrize("slots", [1, 2, 3, 4])
def test_models_in_turn(slots):
    shapes = [(12, 64, 12, 2048, 2), (2, 32, 1, 36, 3), (8, 128, 2, 1376, 2), (9, 32, 9, 768, 2)]
    models = [model(*s, slots, i + 1) for i, s in enumerate(shapes)]
    rng = np.random.default_rng(slots)
    for turn, at in enumerate([0, 1, 63, 64, 127, 128, 255, 256, 257, 700, 1023]):
        for m in models:
            pos = [max(at - 37 * b, 0) for b in range(slots)]
            if slots > 2 and turn % 3 == 1:
                pos[1] = -1
            step(*m, pos, rng)


@pytest.mark.parametrize("slots", [5, 6, 7, 8])
def test_models_in_turn_of_up_to_eight_slots(slots):
    """Two warps a staged row in place of four to sixteen; with the row pipeline, which takes these sizes from five slots on, switched off."""
    lib = load_pkg("cabi").lib()
    lib.check(lib.c.tha_set_option(b"tc", 0))
    try:
        test_models_in_turn(slots)
    finally:
        lib.check(lib.c.tha_set_option(b"tc", -1))


def test_graph_replays_and_steps_in_a_row():
    cfg, w, e = model(12, 64, 12, 2048, 2, 2, 9)
    rng = np.random.default_rng(5)
    for t in range(120, 140):
        step(cfg, w, e, [t, t + 130], rng)
