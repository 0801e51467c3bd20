"""Prompt calls of the fp32 path in which one portion's context is another portion of the same call: consecutive portions of one slot, in either order, and slots whose block
tables share the blocks that the call fills.  Against float64 of the whole sequence, on both sides of the sizes that take the tensor cores (csrc/step_tc.cu: rows_f16x3)."""
import numpy as np
import pytest
import torch

import llama64
from pkgload import load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[20, 12], [65, 16, 30], [128, 128], [200, 57]])
@pytest.mark.parametrize("how", ["in order", "reversed", "shared blocks"])
@pytest.mark.parametrize("heads,hs,kv_heads", [(16, 128, 16), (32, 64, 8), (6, 64, 6)])
def test_portions_of_one_sequence(heads, hs, kv_heads, lens, how):
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, 264, 2, heads, kv_heads, 96, 512)
    w = eng.device_random_weights(cfg, seed=2, std=cfg.dim ** -0.5)
    toks = np.random.default_rng(3).integers(0, 96, sum(lens)).astype(np.int32)
    at = np.cumsum([0] + lens)
    pages, slots = None, 1
    if how == "shared blocks":                      # a table row a portion, all of them the same blocks
        slots, per = len(lens), 512 // 16
        pages = eng.PagedKV(cfg, slots, per, 16)
        pages.set_table(np.tile(np.random.default_rng(6).permutation(per).astype(np.int32), (slots, 1)))
    e = eng.Engine(w, slots, with_att=False, paged=pages)
    e.state.key_cache.normal_(0.0, 1.0)
    e.state.value_cache.normal_(0.0, 1.0)
    seqs = [(i % slots, int(at[i]), toks[at[i]:at[i + 1]]) for i in range(len(lens))]
    order = list(range(len(lens)))[::-1] if how == "reversed" else list(range(len(lens)))
    got = torch.empty(len(lens), 96, device="cuda")
    torch.cuda.synchronize()
    e.prefill([seqs[i] for i in order], got)
    torch.cuda.synchronize()
    for row, i in enumerate(order):
        want, _, _ = llama64.forward(cfg, w.t, lambda c, s, l, n: e.state.key_cache[:0].reshape(-1, kv_heads * hs)[:0], [(0, 0, toks[:at[i + 1]])])
        # products of up to 2048 terms at 1e-6 to 1e-5 each (test_gpu_prompt_rows.py), through two layers
        assert float((got[row].double() - want[0]).norm() / want.norm()) < 5e-5


@pytest.mark.parametrize("kind", ["q8", "bf16"])
@pytest.mark.parametrize("lens", [[20, 12], [200, 57], [300, 400]])
@pytest.mark.parametrize("reverse", [False, True])
def test_portions_of_the_other_formats(kind, lens, reverse):
    """Against the whole sequence as one portion: the second layer's cache rows, a value in some hundred of which may fall on the other side of a quantiser's or a bf16 step."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(1024, 1024, 2, 8, 8, 96, 768)
    w = eng.DeviceWeightsBF16.random(cfg, seed=2) if kind == "bf16" else eng.device_random_weights(cfg, q8=True, seed=2, gs=64)
    toks = np.random.default_rng(3).integers(0, 96, sum(lens)).astype(np.int32)
    at = np.cumsum([0] + lens)
    parts = [(0, int(at[i]), toks[at[i]:at[i + 1]]) for i in range(len(lens))]
    rows = []
    for seqs in (parts[::-1] if reverse else parts, [(0, 0, toks)]):
        e = eng.Engine(w, 1, with_att=False)
        e.state.key_cache.normal_(0.0, 1.0)
        e.state.value_cache.normal_(0.0, 1.0)
        out = torch.empty(len(seqs), 96, device="cuda")
        torch.cuda.synchronize()
        e.prefill(seqs, out)
        torch.cuda.synchronize()
        rows.append(torch.stack([e.state.key_cache[0, 1, :sum(lens)], e.state.value_cache[0, 1, :sum(lens)]]).double())
    assert float((rows[0] - rows[1]).norm() / rows[1].norm()) < 2e-2
