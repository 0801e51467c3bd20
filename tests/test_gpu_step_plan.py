"""Decode steps through a plan (tha_hyb_step_planned: executable graphs, csrc/hybrid_step.cu) against the same steps without one: a step that
asks for the layers' taps is issued kernel by kernel."""
import os

import numpy as np
import pytest

import logulix_oracle as LO
from pkgload import load_pkg
from test_gpu_logulix import attention, dense, model, retention, wkv

pytestmark = pytest.mark.gpu


def folder(tmp, cfg, seed):
    os.makedirs(tmp, exist_ok=True)
    load_pkg("serving").save_model_folder(str(tmp), cfg, LO.random_weights(cfg, seed, 6))
    return str(tmp)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_planned_steps_equal_issued_ones(tmp_path, dtype):
    """Requests that join, decode past a multiple of 256 positions, wait for one another's prompts (which grow the scratch of all engines)
    and leave; eleven batch sizes and want lists, more forms than a plan keeps."""
    S = load_pkg("serving").ServingEngine
    cfg = model([attention(dense(), heads=4, kv_heads=2, dim=32), retention(dense()), wkv(dense())], loop=(0, 1, 2))
    f = folder(tmp_path / "m", cfg, 3)
    planned, issued = S(f, dtype, 4096, 12), S(f, dtype, 4096, 12)
    rng = np.random.default_rng(1)

    def both(entries, repeat=1):
        for _ in range(repeat):
            a = planned.step(entries)
            b, _ = issued.step(entries, taps=True)
            # the same kernels on the same numbers; the longest context, by which a key range is cut into runs, is rounded up in a plan:
            # fp32 sums of up to 280 terms in another order, a handful of roundings (2^-24 each) through three layers
            tol = 2e-5 if dtype == "float32" else 2e-2
            assert np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max())

    def token(names):
        return [(n, [int(rng.integers(0, cfg["vocab"]))], [0]) for n in names]

    both([("a", rng.integers(0, 130, 250).tolist(), [249]), ("b", rng.integers(0, 130, 7).tolist(), [6])])
    for _ in range(9):
        both(token("ab"))                                   # position 256 in the middle
    both([("c", rng.integers(0, 130, 300).tolist(), [])] + token("a"))
    for _ in range(4):
        both(token("abc"))
        both([(n, t, []) for n, t, _ in token("a")] + token("c"))   # another form in turn: neither twice running
    for e in (planned, issued):
        e.finish("b")
    both([("d", rng.integers(0, 130, 900).tolist(), [899])])        # scratch of all engines grows
    for _ in range(4):
        both(token("acd"))
    names = "acd"
    for n in "efghijkl":
        names += n
        both([(n, rng.integers(0, 130, 3).tolist(), [2])])
        for _ in range(3):
            both(token(names))
    for _ in range(3):
        both(token("ac"))                                   # a form that the plan may have dropped


def test_two_engines_in_turn(tmp_path):
    """Plans of two models over the one scratch."""
    S = load_pkg("serving").ServingEngine
    cfgs = [model([attention(dense())]), model([retention(dense()), wkv(None)], width=96)]
    fs = [folder(tmp_path / str(i), c, i) for i, c in enumerate(cfgs)]
    engines, plain = [S(f, "float32", 512, 2) for f in fs], [S(f, "float32", 512, 2) for f in fs]
    rng = np.random.default_rng(2)
    for k in range(12):
        for e, p in zip(engines, plain):
            t = rng.integers(0, 130, 5 if k == 0 else 1).tolist()
            a, (b, _) = e.step([("r", t, [len(t) - 1])]), p.step([("r", t, [len(t) - 1])], taps=True)
            assert np.abs(a - b).max() <= 2e-5 * max(1.0, np.abs(b).max())
