"""The fp32 matmul of prompts (csrc/gemm_f16x3.cu): three fp16 products of split operands, against float64."""
import numpy as np
import pytest
import torch

import llama64
from gpu_util import P, stream_ptr
from pkgload import load_pkg

pytestmark = pytest.mark.gpu
RUN = 16 * 64      # values of K that the tensor core sums up before they leave it


def product(W, X, splits=1, ldo=None):
    lib = load_pkg("cabi").lib()
    (M, K), (N, ldx) = W.shape, X.shape
    ldo = ldo or M
    out = torch.full((splits, N, ldo), float("nan"), device="cuda")
    planes = [torch.empty(N, K, dtype=torch.int16, device="cuda") for _ in range(2)]
    scale = torch.empty(N, device="cuda")
    lib.check(lib.c.tha_gemm_f16x3(stream_ptr(), P(out), ldo, P(W), M, K, P(X), N, ldx, splits, P(planes[0]), P(planes[1]), P(scale)), "tha_gemm_f16x3")
    torch.cuda.synchronize()
    assert lib.c.tha_gemm_check_error() == 0
    return out


def check(W, X, splits=1, ldo=None):
    (M, K) = W.shape
    out = product(W, X, splits, ldo)
    if ldo:
        assert torch.isnan(out[:, :, M:]).all()
    got = out[:, :, :M].double().sum(0)
    w, x = W.double(), X[:, :K].double()
    want, size = x @ w.T, x.abs() @ w.abs().T
    # hi + lo holds 22 bits and lo.lo is left out: 3 2^-22 of a product; an addition in the tensor core drops less than 2^-23 of the running sum, K / 16 of them a run
    # (and two for the corrections), then a rounding for each run and three to scale
    bound = 3 * 2.0 ** -22 + (min(K, RUN) / 16 + 4 + K / RUN + 3) * 2.0 ** -23
    assert ((got - want).abs() <= bound * size).all()
    return got, want


@pytest.mark.parametrize("M,K,N,splits", [(1, 64, 1, 1), (127, 72, 63, 1), (128, 128, 64, 1), (129, 136, 65, 1), (256, 1024, 127, 1), (257, 1032, 128, 1),
                                          (600, 2056, 129, 2), (513, 4096, 200, 5), (19072, 192, 257, 1), (300, 16384, 3, 1),
                                          (32000, 64, 300, 1), (9000, 256, 300, 4), (20000, 72, 600, 1), (20000, 72, 600, 2)])
def test_product(M, K, N, splits):
    """Among them shares of one k-block, and more than four items a pair of CTAs: a ring of four scales of weight rows is used again and again."""
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    W, X = (torch.randn(s, device="cuda", generator=g) for s in ((M, K), (N, K + 8)))
    check(W, X, splits, ldo=M + 5)


@pytest.mark.parametrize("splits", [1, 2])
def test_rows_beyond_their_first_values(splits):
    """Weight rows whose first values say nothing of the others: the pair of CTAs that has one goes over its items again."""
    g = torch.Generator(device="cuda").manual_seed(3)
    W, X = torch.randn(700, 1024, device="cuda", generator=g) * 0.02, torch.randn(200, 1024, device="cuda", generator=g)
    W[3, 200:] *= 1e4
    W[5, :128] = 0
    W[130, :1000] = 0
    W[300] = 0
    W[301, 700] = 1e7
    W[302] *= 1e-20
    W[303] *= 1e20
    W[600, :128] *= 1e-30
    X[7] *= 1e-15
    X[8, 5] = 1e6
    X[9] = 0
    X[199] *= 1e15
    check(W, X, splits)                             # every output against the sizes of its own row and column


@pytest.mark.parametrize("splits", [1, 3])
def test_second_pass_over_many_items(splits):
    """Five and more items a pair of CTAs, gone over twice by the pairs that have a row beyond its first values."""
    g = torch.Generator(device="cuda").manual_seed(6)
    W, X = torch.randn(40000, 576, device="cuda", generator=g), torch.randn(300, 576, device="cuda", generator=g)
    W[torch.arange(7, 40000, 3000, device="cuda"), 191] = 1e6
    check(W, X, splits)


@pytest.mark.parametrize("down", [2.0 ** -12, 2.0 ** -20, 1e-6])
@pytest.mark.parametrize("splits", [1, 2])
def test_rows_that_shrink_behind_their_first_values(splits, down):
    """Weight rows (and activation rows) of whose values all but a few large ones are small, where only the small ones meet anything but zeros: they keep their 22 bits."""
    g = torch.Generator(device="cuda").manual_seed(5)
    W, X = torch.randn(300, 1024, device="cuda", generator=g), torch.randn(130, 1024, device="cuda", generator=g)
    large = torch.zeros(1024, dtype=torch.bool, device="cuda")
    large[:128] = True
    large[512:640] = True                            # ahead in each share of K
    W[:, ~large] *= down
    X[:100, large] = 0                               # the other rows meet the large values
    check(W, X, splits)
    check(X, W, splits)


def test_values_that_are_not_finite_stay_in_their_rows():
    g = torch.Generator(device="cuda").manual_seed(4)
    W, X = torch.randn(300, 256, device="cuda", generator=g), torch.randn(70, 256, device="cuda", generator=g)
    W[20, 50], W[21, 200], X[30, 3], X[31, 3] = float("inf"), float("nan"), float("-inf"), float("nan")
    bad = ~torch.isfinite(product(W, X)[0])
    want = torch.zeros_like(bad)
    want[30:32] = True
    want[:, 20:22] = True
    assert torch.equal(bad, want)


@pytest.mark.parametrize("heads,hs,kv_heads,hidden,lens", [(16, 128, 16, 4104, [64]), (16, 128, 4, 4104, [65]), (16, 128, 16, 5000, [100, 1, 28]), (32, 64, 32, 264, [129]), (16, 128, 16, 264, [128]), (32, 128, 8, 264, [64]), (32, 128, 8, 264, [40, 25]),
                                                           (8, 64, 8, 1376, [511]), (8, 64, 2, 1376, [500, 12])])
def test_prompts(heads, hs, kv_heads, hidden, lens):
    """Both sides of the rule by rows and width, two layers, behind a context."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, hidden, 2, heads, kv_heads, 96, 540)
    w = eng.device_random_weights(cfg, seed=2, std=cfg.dim ** -0.5)
    e = eng.Engine(w, len(lens), with_att=False)
    rng = np.random.default_rng(3)
    g = torch.Generator(device="cuda").manual_seed(5)
    e.state.key_cache.normal_(0.0, 1.0, generator=g)
    e.state.value_cache.normal_(0.0, 1.0, generator=g)
    seqs = [(i, 7, rng.integers(0, 96, n).astype(np.int32)) for i, n in enumerate(lens)]
    keys = e.state.key_cache.clone()
    values = e.state.value_cache.clone()
    got = torch.empty(len(seqs), 96, device="cuda")
    torch.cuda.synchronize()
    e.prefill(seqs, got)
    torch.cuda.synchronize()
    want, k, v = llama64.forward(cfg, w.t, lambda c, s, l, n: (keys if c == "k" else values)[s, l, :n], seqs)
    rel = lambda a, b: float((a.double() - b.double()).norm() / b.double().norm())
    assert rel(got, want) < 5e-5                    # as test_fp32_rows
    at = 0
    for i, n in enumerate(lens):
        assert rel(e.state.key_cache[i, :, 7:7 + n], k[at:at + n].transpose(0, 1)) < 3e-5
        assert rel(e.state.value_cache[i, :, 7:7 + n], v[at:at + n].transpose(0, 1)) < 3e-5
        at += n


@pytest.mark.parametrize("heads,hs,kv_heads", [(16, 128, 16), (16, 128, 4), (32, 64, 32), (32, 64, 8)])
@pytest.mark.parametrize("pos0,lens,paged", [(0, [128, 1, 100], False), (1, [127, 129], False), (127, [130], True), (128, [16, 64, 60], True), (0, [257, 15], True), (300, [20, 130], False)])
def test_prompt_attention(heads, hs, kv_heads, pos0, lens, paged):
    """Prompt attention on the tensor cores (csrc/attn_prefill_x3.cu): tiles of 128 rows and keys, portions behind contexts, block tables; keys and values of very
    different sizes, so that each has a scale of its own."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, 264, 1, heads, kv_heads, 96, 512)
    w = eng.device_random_weights(cfg, seed=2, std=cfg.dim ** -0.5)
    pages = None
    if paged:
        per = 512 // 16
        pages = eng.PagedKV(cfg, len(lens), per * len(lens), 16)
        pages.set_table(np.random.default_rng(6).permutation(per * len(lens)).astype(np.int32).reshape(len(lens), per))
    e = eng.Engine(w, len(lens), with_att=False, paged=pages)
    g = torch.Generator(device="cuda").manual_seed(5)
    for cache in (e.state.key_cache, e.state.value_cache):
        cache.normal_(0.0, 1.0, generator=g)
        cache.mul_(torch.exp2(torch.randint(-12, 2, cache.shape[:-1], device="cuda", generator=g).float())[..., None])
    rng = np.random.default_rng(3)
    seqs = [(i, pos0, rng.integers(0, 96, n).astype(np.int32)) for i, n in enumerate(lens)]
    kept = {"k": e.state.key_cache.clone(), "v": e.state.value_cache.clone()}

    def rows(c, s, l, n):
        if not paged:
            return kept[c][s, l, :n]
        return kept[c][pages.table[s].long(), l].reshape(-1, kept[c].shape[-1])[:n]

    got = torch.empty(len(seqs), 96, device="cuda")
    torch.cuda.synchronize()
    e.prefill(seqs, got)
    torch.cuda.synchronize()
    want, _, _ = llama64.forward(cfg, w.t, rows, seqs)
    # sums of 32 to 2048 terms at 1e-6 to 2e-6 each (test_product), through three products and the attention one after the other
    assert float((got.double() - want).norm() / want.norm()) < 1e-5


@pytest.mark.parametrize("heads,hs,kv_heads", [(16, 128, 16), (32, 64, 8)])
@pytest.mark.parametrize("size", [20, 40, 60])
@pytest.mark.parametrize("at", [45, 100, 200])
def test_prompt_attention_ahead_of_a_large_value(heads, hs, kv_heads, at, size):
    """Rows that do not see a key are as exact as without it, whatever the size of its values (2^size times the others'): the weights of a row are scaled by the keys that it sees.
    The token at `at` is the only one with the channel whose gain is 2^size."""
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    cfg = ck.Config(heads * hs, 264, 2, heads, kv_heads, 96, 512)
    w = eng.device_random_weights(cfg, seed=2, std=cfg.dim ** -0.5)
    w.t["tok_emb"][:, 0] = 0
    w.t["tok_emb"][95] = 0
    w.t["tok_emb"][95, 0] = 1
    w.t["rms_att"][0, 0] = 2.0 ** (size - 0.5 * np.log2(cfg.dim))
    w.t["wq"][0, :, 0] = 0
    w.t["wk"][0, :, 0] = 0
    e = eng.Engine(w, 1, with_att=False)
    toks = np.random.default_rng(3).integers(0, 95, 230).astype(np.int32)
    toks[at] = 95
    got = torch.empty(1, 96, device="cuda")
    torch.cuda.synchronize()
    e.prefill([(0, 0, toks)], got)
    torch.cuda.synchronize()
    _, k, v = llama64.forward(cfg, w.t, lambda c, s, l, n: e.state.key_cache[0, l, :0], [(0, 0, toks[:at])])
    assert float(v[:, 0].abs().max()) < 100
    for cache, want in ((e.state.key_cache, k), (e.state.value_cache, v)):
        # the second layer's rows: through the attention and four products, as test_prompt_attention
        assert float((cache[0, 1, :at].double() - want[:, 1]).norm() / want[:, 1].norm()) < 1e-5
    assert float(e.state.value_cache[0, 0, at].abs().max()) > 2.0 ** (size - 6)
