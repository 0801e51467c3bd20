"""The row kernels of a step (csrc/step_tc.cu) from 512 prompt rows on: widths around a block's share."""
import numpy as np
import pytest
import torch

import llama64
from pkgload import load_pkg

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def prefill(e, seqs, vocab):
    out = torch.empty(len(seqs), vocab, device="cuda")
    torch.cuda.synchronize()
    e.prefill(seqs, out)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("heads,hs,hidden", [(8, 16, 36), (16, 64, 2052), (18, 64, 100), (33, 128, 4196)])
@pytest.mark.parametrize("lens", [[512], [400, 111, 2]])
def test_fp32_rows(heads, hs, hidden, lens):
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, hidden, 1, heads, heads, 96, 520)
    w = eng.device_random_weights(cfg, seed=2, std=cfg.dim ** -0.5)
    e = eng.Engine(w, len(lens), with_att=False)
    rng = np.random.default_rng(3)
    seqs = [(i, 0, rng.integers(0, 96, n).astype(np.int32)) for i, n in enumerate(lens)]
    got = prefill(e, seqs, 96)
    want, k, v = llama64.forward(cfg, w.t, lambda c, s, l, n: e.state.key_cache[s, l, :n], seqs)
    # 3xTF32 sums of 32 to 4224 terms: 1e-6 to 1e-5 (accumulation in the tensor core), through three products one after the other
    assert rel(got, want) < 5e-5
    at = 0
    for i, n in enumerate(lens):
        assert rel(e.state.key_cache[i, :, :n], k[at:at + n].transpose(0, 1)) < 3e-5 and rel(e.state.value_cache[i, :, :n], v[at:at + n].transpose(0, 1)) < 3e-5
        at += n


@pytest.mark.parametrize("heads,hs,hidden", [(8, 32, 128), (18, 64, 2112), (33, 128, 4160)])
def test_q8_rows(heads, hs, hidden):
    """One call of 512 + 1 rows against calls of 171: the first layer's key rows (rmsnorm, quantiser, product, rotation) differ by the order
    of partial sums at most, later values by quantiser steps that fall the other way."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, hidden, 2, heads, heads, 96, 520)
    w = eng.device_random_weights(cfg, q8=True, seed=4, gs=32)
    toks = np.random.default_rng(5).integers(0, 96, 513).astype(np.int32)
    a, b = eng.Engine(w, 1, with_att=False), eng.Engine(w, 1, with_att=False)
    got = prefill(a, [(0, 0, toks)], 96)
    for i in range(0, 513, 171):
        want = prefill(b, [(0, i, toks[i:i + 171])], 96)
    assert rel(a.state.key_cache[0, 0, :513], b.state.key_cache[0, 0, :513]) < 2e-6
    assert rel(got, want) < 5e-2


@pytest.mark.parametrize("rows", [2, 511, 512])
@pytest.mark.parametrize("hidden", [128, 1024, 1056, 2080])
def test_quantiser_on_both_sides_of_its_line(rows, hidden):
    """The SwiGLU quantiser takes one float4 a thread below 512 rows of this width and two from there on, the same bits either way: the rows of one call
    against calls of their own (each value differs by the order of partial sums ahead of the quantiser at most)."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(1152, hidden, 2, 18, 18, 96, 520)
    w = eng.device_random_weights(cfg, q8=True, seed=6, gs=32)
    toks = np.random.default_rng(8).integers(0, 96, rows).astype(np.int32)
    a, b = eng.Engine(w, 1, with_att=False), eng.Engine(w, 1, with_att=False)
    prefill(a, [(0, 0, toks)], 96)
    half = rows // 2
    prefill(b, [(0, 0, toks[:half])], 96)
    prefill(b, [(0, half, toks[half:])], 96)
    # the second layer's rows have gone through the first one's SwiGLU and its quantiser: a value in a thousand may fall the other way
    for cache in (lambda e: e.state.key_cache, lambda e: e.state.value_cache):
        assert rel(cache(a)[0, 1, :rows], cache(b)[0, 1, :rows]) < 1e-2


@pytest.mark.parametrize("heads,hs,hidden", [(18, 64, 2112), (9, 128, 1024), (32, 128, 512)])
def test_q8_rows_are_the_same_bits_in_both_forms(heads, hs, hidden):
    """A prompt of 512 rows against its first 511: the same products and attention tiles, rmsnorm and quantiser in their prompt form and in the other.
    Both add in the same order, so that no value falls on the other side of a quantiser step."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, hidden, 3, heads, heads, 96, 520)
    w = eng.device_random_weights(cfg, q8=True, seed=9, gs=32)
    toks = np.random.default_rng(10).integers(0, 96, 512).astype(np.int32)
    a, b = eng.Engine(w, 1, with_att=False), eng.Engine(w, 1, with_att=False)
    prefill(a, [(0, 0, toks)], 96)
    prefill(b, [(0, 0, toks[:511])], 96)
    assert torch.equal(a.state.key_cache[0, :, :511], b.state.key_cache[0, :, :511])
    assert torch.equal(a.state.value_cache[0, :, :511], b.state.value_cache[0, :, :511])


@pytest.mark.parametrize("heads,hs,hidden,lens", [(8, 16, 36, [4700]), (16, 64, 2052, [300, 280])])
def test_fp32_rows_of_narrow_models(heads, hs, hidden, lens):
    """Narrow models reach the prompt form of the row kernels with more rows."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, hidden, 1, heads, heads, 96, max(lens) + 4)
    w = eng.device_random_weights(cfg, seed=2, std=cfg.dim ** -0.5)
    e = eng.Engine(w, len(lens), with_att=False)
    rng = np.random.default_rng(3)
    seqs = [(i, 0, rng.integers(0, 96, n).astype(np.int32)) for i, n in enumerate(lens)]
    got = prefill(e, seqs, 96)
    want, k, v = llama64.forward(cfg, w.t, lambda c, s, l, n: e.state.key_cache[s, l, :n], seqs)
    assert rel(got, want) < 5e-5        # as test_fp32_rows
    at = 0
    for i, n in enumerate(lens):
        assert rel(e.state.key_cache[i, :, :n], k[at:at + n].transpose(0, 1)) < 3e-5 and rel(e.state.value_cache[i, :, :n], v[at:at + n].transpose(0, 1)) < 3e-5
        at += n
