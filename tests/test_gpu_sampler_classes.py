"""The sampler's selection by classes of keys (csrc/sampler.cu, smp_select_class): whatever the distribution, the token of the form that keeps the row in memory, which
accumulates the same integer masses level by level."""
import ctypes as C

import numpy as np
import pytest
import torch

from gpu_util import P, stream_ptr
from pkgload import load_pkg

pytestmark = pytest.mark.gpu


def rows(kind, B, V, rng):
    if kind == "flat":
        return rng.standard_normal((B, V)) * 0.02
    if kind == "steep":
        return rng.standard_normal((B, V)) * 6.0
    if kind == "equal":                       # one class of all elements, and of a few values
        return np.repeat(rng.integers(0, 1 + np.arange(B)[:, None] % 3, (B, V)) * 0.5, 1, 1)
    if kind == "halves":                      # probabilities 1/2, 1/4, ...: prefix masses on the edges of classes
        return np.tile(-np.arange(V) * np.log(2.0), (B, 1))
    x = rng.standard_normal((B, V))           # a class of a few hundred neighbours around the target, and one far ahead
    x[:, : V // 2] = 2.0 + rng.standard_normal((B, V // 2)) * 1e-3
    x[:, V // 2] = 8.0
    return x


@pytest.mark.parametrize("kind", ["flat", "steep", "equal", "halves", "crowd"])
@pytest.mark.parametrize("V", [2, 3, 40, 511, 513, 4097, 32000])
@pytest.mark.parametrize("topp", [0.02, 0.5, 0.75, 0.9, 0.999])
def test_classes_pick_the_tokens_of_the_levels(kind, V, topp):
    lib = load_pkg("cabi").lib()
    B = 24
    logits = torch.from_numpy(rows(kind, B, V, np.random.default_rng(V)).astype(np.float32)).cuda()
    seeds = torch.arange(1, B + 1, dtype=torch.int64, device="cuda") * 2654435761
    pos = torch.zeros(B, dtype=torch.int32, device="cuda")
    got = {}
    try:
        for resident in (1, 0):
            lib.check(lib.c.tha_set_option(b"sample_resident", resident))
            state, nxt, toks = seeds.clone(), torch.zeros(B, dtype=torch.int32, device="cuda"), []
            for _ in range(3):
                t = logits.clone()
                torch.cuda.synchronize()
                lib.check(lib.c.tha_sample(stream_ptr(), B, P(t), V, C.c_float(1.0), C.c_float(topp), P(state), None, None, P(pos), P(nxt)))
                torch.cuda.synchronize()
                toks.append(nxt.clone())
            got[resident] = torch.stack(toks), t, state
    finally:
        lib.check(lib.c.tha_set_option(b"sample_resident", 1))
    for a, b in zip(got[1], got[0]):
        assert torch.equal(a, b)
