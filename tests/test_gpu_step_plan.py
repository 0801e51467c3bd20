"""Decode steps through a plan (tha_hyb_step_planned: executable graphs, csrc/hybrid_step.cu) against the same steps without one (a step that
asks for the layers' taps is issued kernel by kernel): the same launches, so the same bits, and steps that do run as graphs."""
import ctypes as C
import os

import numpy as np
import pytest

import logulix_oracle as LO
import hyb_cabi as H
from pkgload import load_pkg
from test_gpu_logulix import attention, dense, model, retention, wkv

pytestmark = pytest.mark.gpu
OFTEN = 16      # more times than a form is issued before it is captured


def folder(tmp, cfg, seed):
    os.makedirs(tmp, exist_ok=True)
    load_pkg("serving").save_model_folder(str(tmp), cfg, LO.random_weights(cfg, seed, 6))
    return str(tmp)


class Pair:
    """An engine whose steps are planned and one whose steps are issued."""

    def __init__(self, f, dtype, max_tokens, max_seqs):
        S = load_pkg("serving").ServingEngine
        self.planned, self.issued = S(f, dtype, max_tokens, max_seqs), S(f, dtype, max_tokens, max_seqs)

    def step(self, entries):
        assert np.array_equal(self.planned.step(entries), self.issued.step(entries, taps=True)[0])

    def finish(self, name):
        self.planned.finish(name)
        self.issued.finish(name)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_planned_steps_equal_issued_ones(tmp_path, dtype):
    """Requests that join, decode past multiples of 64 positions (where the attention is cut into more runs), wait for one another's prompts (which
    grow the scratch of all engines) and leave."""
    cfg = model([attention(dense(), heads=4, kv_heads=2, dim=32), retention(dense()), wkv(dense())], loop=(0, 1, 2))
    e = Pair(folder(tmp_path / "m", cfg, 3), dtype, 4096, 12)
    rng = np.random.default_rng(1)

    def tokens(names):
        return [(n, [int(rng.integers(0, cfg["vocab"]))], [0]) for n in names]

    def prompt(name, n, want):
        return (name, rng.integers(0, 130, n).tolist(), [n - 1] if want else [])

    def replays(steps):
        had = e.planned.replayed_steps()
        for s in steps:
            e.step(s)
        return e.planned.replayed_steps() - had

    e.step([prompt("a", 235, True), prompt("b", 7, True)])
    assert replays(tokens("ab") for _ in range(2 * OFTEN)) >= 3          # position 256 in the middle
    e.step([prompt("c", 300, False)] + tokens("a"))
    assert replays(t for _ in range(OFTEN) for t in (tokens("abc"), [(n, x, []) for n, x, _ in tokens("a")] + tokens("c"))) >= 6   # two forms in turn
    e.finish("b")
    e.step([prompt("d", 900, True)])                                     # scratch of all engines grows
    assert replays(tokens("acd") for _ in range(OFTEN)) >= 3
    names = "acd"
    for n in "efghijkl":
        names += n
        e.step([prompt(n, 3, True)])
        assert replays(tokens(names) for _ in range(OFTEN)) >= 3
    assert replays(tokens("ac") for _ in range(OFTEN)) >= 3
    assert e.issued.replayed_steps() == 0


def test_two_engines_in_turn(tmp_path):
    """Plans of two models over the one scratch."""
    cfgs = [model([attention(dense())]), model([retention(dense()), wkv(None)], width=96)]
    pairs = [Pair(folder(tmp_path / str(i), c, i), "float32", 512, 2) for i, c in enumerate(cfgs)]
    rng = np.random.default_rng(2)
    for k in range(2 * OFTEN):
        for e in pairs:
            t = rng.integers(0, 130, 5 if k == 0 else 1).tolist()
            e.step([("r", t, [len(t) - 1])])
    assert all(e.planned.replayed_steps() >= OFTEN for e in pairs)


def test_a_step_that_cannot_be_captured_is_issued(tmp_path, monkeypatch):
    """Many rows of a mixture whose group sizes come back to the host."""
    import gavodra_oracle as GO
    import test_gpu_gavodra as G
    monkeypatch.setenv("THA_HYB_EXPERT_ROWS", "1")
    cfg = G.model([G.attention(G.moe(ff=64, shared=None), heads=2, kv_heads=1, dim=16, vdim=16)], width=64, vocab=60)
    f = str(tmp_path / "m")
    os.makedirs(f)
    load_pkg("serving").save_model_folder(f, cfg, {k: np.asarray(v, np.float32) for k, v in GO.random_weights(cfg, 1, 12).items()})
    e = Pair(f, "bfloat16", 1100 * 64, 1100)
    rng = np.random.default_rng(3)
    for _ in range(OFTEN):
        e.step([("r%d" % i, [int(rng.integers(0, 60))], [0] if i % 100 == 0 else []) for i in range(1100)])
    assert e.planned.replayed_steps() == 0


def test_forms_of_a_plan():
    """Through the C entry: a model without layers, more batch sizes than a plan keeps, the switches that a launch reads, and a capture of the caller's."""
    import torch
    lib, vocab, width, most = H.lib(), 64, 64, 70
    lib.c.tha_hyb_step_planned.argtypes = [H.P, H.P, C.POINTER(H.Model), C.POINTER(H.Rows), C.POINTER(H.Kv), C.POINTER(H.States), H.I, H.P, H.P]
    lib.c.tha_hyb_plan_create.argtypes = [C.POINTER(H.P)]
    lib.c.tha_hyb_plan_destroy.argtypes, lib.c.tha_hyb_plan_destroy.restype = [H.P], None
    lib.c.tha_hyb_plan_counts.argtypes, lib.c.tha_hyb_plan_counts.restype = [H.P, C.POINTER(C.c_longlong), C.POINTER(C.c_longlong)], None
    g = torch.Generator(device="cuda").manual_seed(1)
    embed, head = (torch.randn(vocab, width, device="cuda", generator=g).bfloat16() for _ in range(2))
    one = torch.ones(width, device="cuda")
    m = H.Model(dtype=H.BF16, width=width, vocab=vocab, eps=1e-6, embed=H.ptr(embed), final_norm=H.Norm(0, H.ptr(one), None, 0.0, 0.0), head=H.ptr(head))
    plan, stream = H.P(), torch.cuda.Stream()
    lib.check(lib.c.tha_hyb_plan_create(C.byref(plan)))
    forms, kv, st = {}, H.Kv(), H.States()

    def step(n, planned=True, on=None):
        if n not in forms:
            r, keep = H.rows_of([(i, 3, 1) for i in range(n)])
            keep[0].copy_(torch.randint(0, vocab, (n,), device="cuda", generator=g))
            forms[n] = r, keep, torch.arange(n, device="cuda", dtype=torch.int32), torch.zeros(n, vocab, device="cuda")
            torch.cuda.synchronize()
        r, _, want, logits = forms[n]
        args = (m, r, kv, st, n, H.ptr(want), H.ptr(logits))
        s = (on or stream).cuda_stream
        lib.check(lib.c.tha_hyb_step_planned(s, plan, *args) if planned else lib.c.tha_hyb_step(s, *args, None))
        return logits

    def counts():
        a, b = C.c_longlong(), C.c_longlong()
        lib.c.tha_hyb_plan_counts(plan, C.byref(a), C.byref(b))
        return a.value, b.value

    def same(n):
        torch.cuda.synchronize()
        logits = forms[n][3]
        got = logits.clone()
        logits.zero_()
        torch.cuda.synchronize()
        step(n, planned=False)
        torch.cuda.synchronize()
        assert torch.equal(got, logits) and float(got.abs().max()) > 0.5

    step(most)                                       # scratch for all of them
    for n in range(1, most):
        for _ in range(OFTEN):
            step(n)
        same(n)
    captured, replayed = counts()
    assert captured == most - 1 and replayed >= 3 * (most - 1)
    for _ in range(OFTEN):                           # the first form has gone, and comes again
        step(1)
    same(1)
    assert counts()[0] == captured + 1
    for name, value in (("THA_HYB_SCAN", "shared"), ("THA_HYB_EXPERT_ROWS", "7")):
        os.environ[name] = value
        try:
            had = counts()[1]
            step(1)
            assert counts()[1] == had                # another form
        finally:
            del os.environ[name]
    had = counts()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        step(1)
    forms[1][3].zero_()
    graph.replay()
    same(1)
    assert counts() == had
    lib.c.tha_hyb_plan_destroy(plan)
