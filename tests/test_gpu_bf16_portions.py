"""Prompts of the bf16 model in portions (csrc/attn_prefill_tc.cu; the rows ahead of a portion by bf_kv_context_kernel): cuts and ends on both sides of the
groups of 16 keys and the tiles of 128, plain and paged caches, with NaN in scratch from a call before.  Same statement and bound as
tests/test_gpu_bf16.py: a rounding that falls on the other side moves a logit by a few 1e-3 of the largest, three such steps are allowed."""
import os
import subprocess
import sys

import numpy as np
import pytest

from gpu_util import assert_close_scaled
from pkgload import load_pkg
from test_gpu_bf16 import BF16_EPS, MODELS, bf16_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,cuts,lens", [("hs64", (16, 127, 1), (33, 128, 17)), ("hs64", (128, 15, 100), (129, 16, 190)),
                                            ("hs128", (127, 129, 255), (130, 257, 257)), ("hs128", (17, 128, 383), (400, 144, 385))])
def test_portions_vs_oracle(oracle, tmp_path, name, cuts, lens):
    import torch
    eng = load_pkg("engine")
    cfg, wb, path = bf16_model(tmp_path, name, MODELS[name])
    m = oracle.open(path, bf16=True)
    m.set_bf16_attention(True)
    rng = np.random.default_rng(lens[0])
    prompts = [rng.integers(0, cfg.vocab_size, n).astype(np.int32) for n in lens]
    want = []
    for b in range(3):
        seq = m.new_seq()
        for i, t in enumerate(prompts[b]):
            lg = seq.forward(int(t), i)
        want.append(lg.copy())
    w = eng.DeviceWeightsBF16(cfg, wb)
    per = -(-cfg.seq_len // 16)
    pages = eng.PagedKV(cfg, 4, 4 * per, 16)
    pages.set_table(rng.permutation(4 * per).reshape(4, per).astype(np.int32))
    bits = []
    for e in (eng.Engine(w, 4), eng.Engine(w, 4, paged=pages)):
        logits, nxt = torch.empty(3, cfg.vocab_size, device="cuda"), torch.empty(3, dtype=torch.int32, device="cuda")
        e.state.key_cache.fill_(float("nan"))
        e.state.value_cache.fill_(float("nan"))
        e.prefill([(3, cfg.seq_len - 7, prompts[0][:5])] * 3, logits, nxt)     # a context of NaN: staged rows of it stay in scratch
        e.prefill([(b, 0, prompts[b][:cuts[b]]) for b in range(3)])
        e.prefill([(b, cuts[b], prompts[b][cuts[b]:]) for b in range(3)], logits, nxt)
        torch.cuda.synchronize()
        assert load_pkg("cabi").lib().c.tha_gemm_check_error() == 0
        for b in range(3):
            assert_close_scaled(logits[b].cpu().numpy(), want[b], BF16_EPS, f"slot {b}, {cuts[b]} + {lens[b] - cuts[b]}")
        bits.append(logits.clone())
    pages.close()
    assert torch.equal(bits[0], bits[1])


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def engine(slots, seq_len, layers):
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    w = eng.DeviceWeightsBF16.random(ck.Config(512, 768, layers, 4, 4, 96, seq_len), seed=3)
    e = eng.Engine(w, slots)
    e.state.key_cache.normal_()
    e.state.value_cache.normal_()
    return e


def test_scratch_of_many_short_portions_behind_long_contexts_is_bounded():
    """160 contexts of about 2000 rows are 670 MB of staged rows: they are taken in groups, with the results of calls of 40, which are one group each."""
    import torch
    e = engine(160, 2064, 2)
    rng = np.random.default_rng(0)
    seqs = [(i, int(rng.integers(1900, 2040)), rng.integers(0, 96, int(rng.integers(1, 20))).astype(np.int32)) for i in range(160)]
    before = e.state.key_cache.clone(), e.state.value_cache.clone()
    want, nxt = torch.empty(160, 96, device="cuda"), torch.empty(160, dtype=torch.int32, device="cuda")
    for i in range(0, 160, 40):
        e.prefill(seqs[i:i + 40], want[i:i + 40], nxt[i:i + 40])
    rows = [c.clone() for c in (e.state.key_cache, e.state.value_cache)]
    e.state.key_cache.copy_(before[0])
    e.state.value_cache.copy_(before[1])
    got, had = torch.empty_like(want), free()
    e.prefill(seqs, got, nxt)
    assert had - free() < 300 << 20
    assert load_pkg("cabi").lib().c.tha_gemm_check_error() == 0
    for i in range(160):
        assert_close_scaled(got[i].cpu().numpy(), want[i].cpu().numpy(), BF16_EPS, f"sequence {i}")
    for a, b in zip(rows, (e.state.key_cache, e.state.value_cache)):
        assert float((a - b).abs().max()) <= BF16_EPS * float(a.abs().max())


def test_contexts_that_do_not_fit_side_by_side_are_taken_one_by_one():
    """With room for one context of them, not for 256 MB: the results of the call that had it, to the bit.  In a process of its own, whose scratch is
    not there yet."""
    code = "import test_gpu_bf16_portions as t; t.one_by_one()"
    r = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.abspath(__file__)), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "one by one: the same" in r.stdout, r.stdout + r.stderr


def one_by_one():
    import torch
    rng = np.random.default_rng(4)
    seqs = [(i, int(rng.integers(1900, 2040)), rng.integers(0, 96, int(rng.integers(1, 20))).astype(np.int32)) for i in range(100)]
    big = engine(100, 2064, 2)              # its cache is what the second call holds the memory with
    before = big.state.key_cache.clone(), big.state.value_cache.clone()
    got = []
    cabi = load_pkg("cabi").lib()
    for tight in (True, False):
        big.state.key_cache.copy_(before[0])
        big.state.value_cache.copy_(before[1])
        held = None
        logits, nxt = torch.empty(100, 96, device="cuda"), torch.empty(100, dtype=torch.int32, device="cuda")
        if tight:
            big.prefill([(0, 0, np.zeros(1200, np.int32))])       # the scratch of the rows themselves
            big.state.key_cache.copy_(before[0])
            big.state.value_cache.copy_(before[1])
            held = torch.empty(max(0, free() - (120 << 20)), dtype=torch.uint8, device="cuda")
        big.prefill(seqs, logits, nxt)
        torch.cuda.synchronize()
        assert cabi.c.tha_gemm_check_error() == 0
        got.append(logits)
        del held
        torch.cuda.empty_cache()
    assert torch.equal(got[0], got[1])
    print("one by one: the same")


def test_portions_of_a_prompt_grow_the_scratch_once():
    """Growing frees, allocates and drops the workspace's graphs."""
    e = engine(1, 32768, 1)
    rng = np.random.default_rng(1)
    left = []
    for at in range(0, 32768, 4096):
        e.prefill([(0, at, rng.integers(0, 96, 4096).astype(np.int32))])
        left.append(free())
    assert len(set(left[1:])) == 1


def test_a_call_that_finds_no_room_leaves_the_workspace_usable():
    """Scratch that cannot grow: an error, and the calls behind it allocate again instead of using what was given back."""
    import torch
    e = engine(2, 40000, 2)
    rng = np.random.default_rng(2)
    small = [(0, 0, rng.integers(0, 96, 40).astype(np.int32)), (1, 3, rng.integers(0, 96, 9).astype(np.int32))]
    tok, pos = torch.tensor([5, 6], dtype=torch.int32, device="cuda"), torch.tensor([41, 12], dtype=torch.int32, device="cuda")

    def calls():
        logits, nxt = torch.empty(2, 96, device="cuda"), torch.empty(2, dtype=torch.int32, device="cuda")
        e.prefill(small, logits, nxt)
        step = torch.empty(2, 96, device="cuda")
        e.decode_step(tok, pos, step, nxt, stream=stream)
        e.decode_step(tok, pos, step, nxt, stream=stream)
        torch.cuda.synchronize()
        return torch.stack([logits, step])

    stream = torch.cuda.Stream()
    want = calls()
    held = []
    try:
        for leave in (600 << 20, 100 << 20):      # some of its arrays fit, then none
            held.append(torch.empty(max(0, free() - leave), dtype=torch.uint8, device="cuda"))
            with pytest.raises(Exception):
                e.prefill([(0, 0, rng.integers(0, 96, 39990).astype(np.int32))] * 4, torch.empty(4, 96, device="cuda"), torch.empty(4, dtype=torch.int32, device="cuda"))
            torch.cuda.synchronize()
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert torch.equal(calls(), want)
