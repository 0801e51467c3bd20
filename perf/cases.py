"""What this framework's speed is measured on: calls that a user's program makes, through the Python binding of the public
entry points, over the range of sizes, number formats and options that are served in earnest.

Three kinds of case:

  decode   one step of the batched llama2 decoder (thaDNN_s_forward_batch and its resident / sampling forms): every slot one
           token at its own position, behind a context that is already in the cache
  prefill  prompt ingestion: all prompt positions of one or several sequences in one call
  layered  requests through a layer-program model folder (ServingEngine): prompts in one step, then decoded tokens

`llama` models have random weights of the named architecture's shape.  The wide model (Llama-2-7B's layer) is cut to a few of its
32 equal layers so that a plain 64-bit statement of the whole call stays cheap.
"""
import functools
import importlib
import importlib.util
import json
import math
import os
import shutil
import struct
import sys
import tempfile
from fractions import Fraction

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package(sub):
    """A module of the package, whose folder name is not an identifier."""
    name, folder = "hip_llama_cpp_b200", os.path.join(ROOT, "hip_llama.cpp_b200")
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"), submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return importlib.import_module(name + "." + sub)


@functools.lru_cache(maxsize=None)
def _stream():
    """The one stream a serving loop runs on (the library replays a decode step as a graph on any stream but the default one)."""
    return torch.cuda.Stream()


# ---- sizes ----------------------------------------------------------------------------------------------------------------
STORIES42M = dict(dim=512, hidden=1376, layers=8, heads=8, kv_heads=8, vocab=32000)
STORIES110M = dict(dim=768, hidden=2048, layers=12, heads=12, kv_heads=12, vocab=32000)
WIDE = dict(dim=4096, hidden=11008, layers=2, heads=32, kv_heads=32, vocab=32000)     # Llama-2-7B, 2 of its 32 layers


def listed():
    return [
        # a single user's chat loop on the small model, through the reference's own call (host tokens in, host logits out)
        dict(STORIES110M, name="decode stories110M f32 1 slot", kind="decode", weights="f32", seq_len=1024, slots=1, first=211, stride=0, call="logits", paged=False),
        # the batching driver's default step at its benchmark's batch: tokens in, sampled tokens out (temperature 1, top-p 0.9)
        dict(STORIES110M, name="decode stories110M f32 256 slots", kind="decode", weights="f32", seq_len=512, slots=256, first=0, stride=1, call="sample", paged=False),
        # a handful of users on the large model in full precision
        dict(WIDE, name="decode 7B f32 6 slots", kind="decode", weights="f32", seq_len=1024, slots=6, first=17, stride=131, call="resident", paged=False),
        # one user on the quantised large model, well into a conversation
        dict(WIDE, name="decode 7B q8 1 slot", kind="decode", weights="q8", seq_len=2048, slots=1, first=1003, stride=0, call="resident", paged=False),
        # a full batch on the quantised large model behind the paged cache
        dict(WIDE, name="decode 7B q8 64 slots paged", kind="decode", weights="q8", seq_len=2048, slots=64, first=3, stride=9, call="resident", paged=True),
        # a medium batch of long contexts on the bf16 model
        dict(WIDE, name="decode 7B bf16 24 slots", kind="decode", weights="bf16", seq_len=2048, slots=24, first=100, stride=61, call="resident", paged=False),
        # many short prompts of the small model at once
        dict(STORIES110M, name="prefill stories110M f32 16 prompts", kind="prefill", weights="f32", seq_len=512, seqs=16, shortest=9, longest=201, start=0),
        # one long prompt in full precision
        dict(WIDE, name="prefill 7B f32 1024", kind="prefill", weights="f32", seq_len=1024, seqs=1, shortest=1024, longest=1024, start=0),
        # a few prompts on the quantised model
        dict(WIDE, name="prefill 7B q8 3 prompts", kind="prefill", weights="q8", seq_len=1024, seqs=3, shortest=37, longest=700, start=0),
        # long prompts on the bf16 model: what decides the time to the first token of long documents
        dict(WIDE, name="prefill 7B bf16 2 prompts", kind="prefill", weights="bf16", seq_len=2048, seqs=2, shortest=777, longest=2048, start=0),
        # a softmax-attention design in serving: two prompts enter, then both decode
        dict(name="layered attention 2 requests", kind="layered", design="gavodra", width=2048, heads=16, kv_heads=4, dim=128, ff=6144, layers=2, vocab=32000,
             dtype="bfloat16", seqs=2, shortest=1100, longest=2900, new=8),
        # a recurrent design (retention, windowed attention, key-value memory) in serving
        dict(name="layered recurrent 3 requests", kind="layered", design="logulix", width=1024, heads=8, kv_heads=2, dim=128, ff=4608, layers=4, vocab=32000,
             dtype="bfloat16", seqs=3, shortest=150, longest=1300, new=8),
    ]


def _log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "layered"])
    if kind == "layered":
        design = rng.choice(["gavodra", "logulix"])
        width = rng.choice([1024, 2048])
        seqs = rng.choice([1, 2, 3, 5])
        longest = _log_between(rng, 40, 2900 if design == "gavodra" else 1300)
        longest = min(longest, 6000 // seqs) if design == "gavodra" else min(longest, 2600 // seqs)
        return dict(kind=kind, design=design, width=width, heads=width // 128, kv_heads=width // 512, dim=128, ff=3 * width + 8 * rng.randrange(0, 96),
                    layers=rng.choice([1, 2]) if design == "gavodra" else rng.choice([3, 4]), vocab=32000,
                    dtype="float32" if longest * seqs <= 600 and rng.random() < 0.25 else "bfloat16", seqs=seqs, shortest=max(1, int(longest * rng.uniform(0.2, 1.0))), longest=longest, new=rng.randint(1, 8))
    weights = rng.choice(["f32", "q8", "bf16"])
    wide = rng.random() < 0.6
    m = dict(WIDE) if wide else dict(rng.choice([STORIES42M, STORIES110M] if weights != "q8" else [STORIES110M]))
    if wide and rng.random() < 0.25:
        m["kv_heads"] = 8     # grouped queries
    if kind == "prefill":
        start = rng.choice([0, 0, 0, rng.randint(1, 200)])
        seqs = _log_between(rng, 1, 16)
        most = {"f32": 1024, "q8": 1100, "bf16": 2800}[weights]
        longest = max(2, min(_log_between(rng, 8, most), most // seqs))
        return dict(m, kind=kind, weights=weights, seq_len=start + longest + rng.randint(1, 64), seqs=seqs, shortest=max(1, int(longest * rng.uniform(0.1, 1.0))),
                    longest=longest, start=start)
    slots = _log_between(rng, 1, 64 if wide else 256)
    seq_len = _log_between(rng, 128, 2048 if wide else 1024)
    while m["layers"] * seq_len * slots * m["dim"] > 1.3e9:
        seq_len = seq_len * 3 // 4
    last = rng.randint(seq_len // 8, seq_len - 1)      # the longest context of the batch
    stride = rng.randint(0, last // max(1, slots - 1)) if slots > 1 else 0
    return dict(m, kind=kind, weights=weights, seq_len=seq_len, slots=slots, first=last - stride * (slots - 1), stride=stride,
                call=rng.choice(["logits", "sample", "resident", "resident"]), paged=rng.random() < 0.25)


# ---- the llama2 path ------------------------------------------------------------------------------------------------------
def _config(case):
    ck = _package("checkpoint")
    return ck.Config(case["dim"], case["hidden"], case["layers"], case["heads"], case["kv_heads"], case["vocab"], case["seq_len"])


def _group(case):
    return 64 if case["dim"] % 64 == 0 and case["hidden"] % 64 == 0 else 32


def _llama_weights(case, seed):
    eng, cfg = _package("engine"), _config(case)
    if case["weights"] == "bf16":
        w = eng.DeviceWeightsBF16.random(cfg, seed=seed)
    else:
        w = eng.device_random_weights(cfg, q8=case["weights"] == "q8", seed=seed, gs=_group(case))
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    for n in ("rms_att", "rms_ffn", "rms_final"):
        w.t[n].uniform_(0.6, 1.4, generator=g)
    return w, g


def _lengths(case, rng):
    """Prompt lengths from the shortest to the longest, in a random order."""
    n, lo, hi = case["seqs"], case["shortest"], case["longest"]
    lens = [hi] + ([lo] if n > 1 else []) + [int(x) for x in rng.integers(lo, hi + 1, max(0, n - 2))]
    return [lens[i] for i in np.random.default_rng(n).permutation(n)]


def _prepare_llama(case, seed):
    eng = _package("engine")
    cfg = _config(case)
    w, g = _llama_weights(case, seed)
    rng = np.random.default_rng(seed)
    # the lengths are the case's own: inputs of another seed are other values, not other sizes
    lens = _lengths(case, np.random.default_rng(case["longest"])) if case["kind"] == "prefill" else None
    slots = case["slots"] if case["kind"] == "decode" else case["seqs"]
    pages = None
    if case.get("paged"):
        per = -(-case["seq_len"] // 16)
        used = [-(-(case["first"] + case["stride"] * b + 1) // 16) for b in range(slots)]
        pages = eng.PagedKV(cfg, slots, sum(used), 16)
        ids = np.random.default_rng(slots).permutation(sum(used))
        table, at = np.zeros((slots, per), np.int32), 0
        for b, n in enumerate(used):
            table[b, :n] = ids[at:at + n]
            at += n
        pages.set_table(table)
    e = eng.Engine(w, slots, with_att=False, paged=pages)
    st = e.state
    st.key_cache.normal_(0.0, 1.0, generator=g)       # the context that earlier steps left in the cache
    st.value_cache.normal_(0.0, 1.0, generator=g)
    s = dict(case=case, w=w, e=e, pages=pages)
    if case["kind"] == "prefill":
        s["seqs"] = [(i, case["start"], rng.integers(0, cfg.vocab_size, n).astype(np.int32)) for i, n in enumerate(lens)]
        s["logits"] = torch.empty(slots, cfg.vocab_size, device="cuda")
        s["next"] = torch.zeros(slots, dtype=torch.int32, device="cuda")
        return s
    s["tokens"] = rng.integers(0, cfg.vocab_size, slots).astype(np.int32)
    s["pos"] = (case["first"] + case["stride"] * np.arange(slots)).astype(np.int32)
    if case["call"] == "logits":
        s["logits"] = torch.empty(slots, cfg.vocab_size).pin_memory()
    elif case["call"] == "sample":
        s["reseed"] = rng.integers(1, 1 << 62, slots).astype(np.uint64)
        s["next"] = np.zeros(slots, np.int32)
    else:
        s["tokens_d"], s["pos_d"] = torch.from_numpy(s["tokens"]).cuda(), torch.from_numpy(s["pos"]).cuda()
        s["logits"] = torch.empty(slots, cfg.vocab_size, device="cuda")
        s["next"] = torch.zeros(slots, dtype=torch.int32, device="cuda")
    return s


def _new_rows(s, cache):
    """The cache rows that the pass writes, as views of the cache (the whole pool where it is paged)."""
    case = s["case"]
    if case["kind"] == "prefill":
        return [cache[i, :, p0:p0 + len(t)] for i, p0, t in s["seqs"]]
    if case["paged"]:
        return cache
    B, L, S, kvd = cache.shape
    return cache.as_strided((B, L, kvd), (L * S * kvd + case["stride"] * kvd, S * kvd, 1), cache.storage_offset() + case["first"] * kvd)


def _run_llama(s):
    case, e, st = s["case"], s["e"], s["e"].state
    if case["kind"] == "prefill":
        e.prefill(s["seqs"], s["logits"], s["next"], stream=_stream())
        out = {"logits": s["logits"], "next": s["next"]}
    elif case["call"] == "logits":
        out = {"logits": e.forward_batch(s["tokens"], s["pos"], s["logits"], stream=_stream())}
    elif case["call"] == "sample":
        e.forward_sample(s["tokens"], s["pos"], None, s["reseed"], 1.0, 0.9, s["next"], stream=_stream())
        out = {"probabilities": st.logits, "next": s["next"]}
    else:
        e.decode_step(s["tokens_d"], s["pos_d"], s["logits"], s["next"], stream=_stream())
        out = {"logits": s["logits"], "next": s["next"]}
    out["keys"], out["values"] = _new_rows(s, st.key_cache), _new_rows(s, st.value_cache)
    return out


def _rows64(x):
    return x.to(torch.float64)


class _Matrices:
    """The case's matrices one layer at a time in 64 bits."""

    def __init__(self, case, w):
        self.kind, self.w, self.gs = case["weights"], w, _group(case)

    def of(self, name, layer):
        t = self.w.t
        if self.kind != "q8":
            return _rows64(t[name][layer] if layer is not None else t[name])
        q, sc = (t[name + ".q"], t[name + ".s"]) if layer is None else (t[name + ".q"][layer], t[name + ".s"][layer])
        q = q.reshape(q.shape[-2], -1, self.gs) if q.dim() == 2 else q
        return (_rows64(q) * _rows64(sc).reshape(q.shape[0], -1, 1)).reshape(q.shape[0], -1)


def _rms(x, gain):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * gain


def _exact_llama(case, seed):
    s = _prepare_llama(case, seed)
    w, st, cfg = s["w"], s["e"].state, _config(case)
    M = _Matrices(case, w)
    d, H, G, hs = cfg.dim, cfg.n_heads, cfg.n_kv_heads, cfg.dim // cfg.n_heads
    seqs = s["seqs"] if case["kind"] == "prefill" else [(b, int(p), [int(t)]) for b, (p, t) in enumerate(zip(s["pos"], s["tokens"]))]
    toks = torch.tensor([int(t) for _, _, ts in seqs for t in ts], device="cuda")
    pos = torch.tensor([p0 + j for _, p0, ts in seqs for j in range(len(ts))], device="cuda", dtype=torch.float64)
    last = torch.tensor(np.cumsum([len(ts) for _, _, ts in seqs]) - 1, device="cuda")
    ang = pos[:, None] * (10000.0 ** (-torch.arange(0, hs, 2, device="cuda", dtype=torch.float64) / hs))[None, :]
    cos, sin = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    table = s["pages"].table.long() if s["pages"] else None

    def rotate(x):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).flatten(-2)

    def before(cache, slot, layer, n):
        if table is None:
            return _rows64(cache[slot, layer, :n])
        return _rows64(cache[table[slot, :-(-n // 16)], layer].reshape(-1, cache.shape[-1])[:n]) if n else _rows64(cache[0, layer, :0])

    x = _rows64(w.t["tok_emb"][toks])
    keys, values = [], []
    for l in range(cfg.n_layers):
        h = _rms(x, _rows64(w.t["rms_att"][l]))
        q = rotate((h @ M.of("wq", l).T).view(-1, H, hs))
        k = rotate((h @ M.of("wk", l).T).view(-1, G, hs))
        v = (h @ M.of("wv", l).T).view(-1, G, hs)
        keys.append(k.flatten(1))
        values.append(v.flatten(1))
        o, at = torch.empty_like(x), 0
        for slot, p0, ts in seqs:
            n = len(ts)
            K = torch.cat([before(st.key_cache, slot, l, p0).view(p0, G, hs), k[at:at + n]])
            V = torch.cat([before(st.value_cache, slot, l, p0).view(p0, G, hs), v[at:at + n]])
            qq = q[at:at + n].view(n, G, H // G, hs)
            sc = torch.einsum("ngmd,tgd->gmnt", qq, K) / math.sqrt(hs)
            if n > 1:
                sc.masked_fill_(torch.ones(n, p0 + n, device="cuda", dtype=torch.bool).triu(p0 + 1), float("-inf"))
            o[at:at + n] = torch.einsum("gmnt,tgd->ngmd", torch.softmax(sc, -1), V).reshape(n, d)
            at += n
        x = x + o @ M.of("wo", l).T
        h = _rms(x, _rows64(w.t["rms_ffn"][l]))
        x = x + (torch.nn.functional.silu(h @ M.of("w1", l).T) * (h @ M.of("w3", l).T)) @ M.of("w2", l).T
    z = _rms(x[last], _rows64(w.t["rms_final"])) @ M.of("wcls", None).T
    keys, values = torch.stack(keys, 1), torch.stack(values, 1)      # [rows, layers, kv_dim]
    if case["kind"] == "prefill":
        cut = [len(ts) for _, _, ts in seqs]
        return {"logits": z, "next": None, "keys": [t.transpose(0, 1) for t in keys.split(cut)], "values": [t.transpose(0, 1) for t in values.split(cut)]}
    if case["paged"]:
        pools = []
        for pool, rows in ((st.key_cache, keys), (st.value_cache, values)):
            full = _rows64(pool)
            for b, p0, _ in seqs:
                full[table[b, p0 // 16], :, p0 % 16] = rows[b]
            pools.append(full)
        keys, values = pools
    if case["call"] == "logits":
        return {"logits": z.cpu(), "keys": keys, "values": values}
    if case["call"] == "sample":
        return {"probabilities": torch.softmax(z, -1), "next": None, "keys": keys, "values": values}
    return {"logits": z, "next": None, "keys": keys, "values": values}


def _work_llama(case):
    d, hd, L, V, kvd = case["dim"], case["hidden"], case["layers"], case["vocab"], case["dim"] // case["heads"] * case["kv_heads"]
    per = {"f32": 4.0, "bf16": 2.0, "q8": 1.0 + 4.0 / _group(case)}[case["weights"]]
    layer, head = 2 * d * d + 2 * d * kvd + 3 * d * hd, V * d
    if case["kind"] == "prefill":
        lens = _lengths(case, np.random.default_rng(case["longest"]))
        rows, outs = sum(lens), len(lens)
        seen = sum(sum(case["start"] + j + 1 for j in range(n)) for n in lens)
        cached = sum(case["start"] for _ in lens)
    else:
        rows = outs = case["slots"]
        seen = sum(case["first"] + case["stride"] * b + 1 for b in range(rows))
        cached = seen - rows
    return {"bytes": per * (layer * L + head) + 8.0 * L * kvd * (cached + rows) + 4.0 * V * outs + per * d * rows,
            "flops": 2.0 * layer * L * rows + 2.0 * head * outs + 4.0 * L * d * seen}


# ---- layer-program models -------------------------------------------------------------------------------------------------
def _layered_config(case):
    W, D = case["width"], case["dim"]
    if case["design"] == "gavodra":
        att = {"heads": case["heads"], "kv_heads": case["kv_heads"], "dim": D, "vdim": D, "scale": D ** -0.5, "bias_max": 2048, "v_mix": True}
        return {"architecture": "Gavodra", "layers": [{"type": "attention", "mixer": att, "mlp": {"kind": "dense", "ff": case["ff"], "limit": 7.0}}] * case["layers"],
                "norm": {"eps": 1e-6}, "vocab": case["vocab"], "width": W, "embedding": {"scale": W ** 0.5}, "residual_mult": 0.8, "logit_scale": 1.0,
                "logit_softcap": 30.0}
    att = {"heads": case["heads"], "kv_heads": case["kv_heads"], "dim": D, "vdim": D, "conv": 4, "scale": D ** -0.5, "softcap": 50.0, "mask": {"size": 1024},
           "rot": {"base": 500000.0, "dims": D, "scaling": {"factor": 2.0}}}
    n = W // 256
    ret = {"heads": n, "dim": 128, "vdim": 256, "rot": {"base": 500000.0, "dims": 128}, "decay": [1.0 - 2.0 ** -(5 + i) for i in range(n)]}
    kinds = [("retention", ret), ("attention", att), ("wkv", {"heads": W // 64, "dim": 64}), ("retention", ret)]
    return {"architecture": "Logulix", "layers": [{"type": kinds[i][0], "mixer": kinds[i][1], "mlp": {"kind": "dense", "ff": case["ff"]}} for i in range(case["layers"])],
            "norm": {"eps": 1e-6}, "vocab": case["vocab"], "width": W, "embedding": {"scale": 1.0}, "logit_scale": 0.5, "loop": {"start": 1, "stop": 3, "times": 1}}


def _layered_tensors(case, cfg, seed):
    """Random weights of the kinds that the folder's writers give: matrices N(0, 1 / in), norm weights around one, ..."""
    serving = _package("serving")
    shapes = serving.gavodra_tensor_shapes(cfg) if case["design"] == "gavodra" else serving.logulix_tensor_shapes(cfg, 64)
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(shape, std, mean=0.0):
        return torch.empty(shape, device="cuda").normal_(mean, std, generator=g)

    def uniform(shape, lo, hi):
        return torch.empty(shape, device="cuda").uniform_(lo, hi, generator=g)

    out = {}
    for name, shape in shapes.items():
        last = name.rsplit(".", 1)[-1]
        if last in ("rel", "conv", "u"):
            a = normal(shape, 0.5)
        elif last == "vmix":
            a = uniform(shape, 0.2, 0.8)
        elif last == "b":
            a = normal(shape, 0.1)
        elif ".mu." in name:
            a = uniform(shape, 0.0, 1.0)
        elif last == "w0":
            a = uniform(shape, -6.0, 0.0)
        elif len(shape) == 2:
            a = normal(shape, 1.0 if name == "embed" and case["design"] == "logulix" else shape[1] ** -0.5)
        else:
            a = normal(shape, 0.2, 1.0)
        out[name] = a.to(torch.bfloat16)
    return out


def _save(folder, cfg, tensors):
    """config.json and model.safetensors (bfloat16)."""
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(cfg, f)
    head, off = {}, 0
    for name, a in tensors.items():
        head[name] = {"dtype": "BF16", "shape": list(a.shape), "data_offsets": [off, off + 2 * a.numel()]}
        off += 2 * a.numel()
    hj = json.dumps(head).encode()
    hj += b" " * (-len(hj) % 8)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(hj)) + hj)
        for a in tensors.values():
            f.write(a.reshape(-1).view(torch.int16).cpu().numpy().tobytes())


def _layered_tokens(case, seed):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, case["vocab"], n + case["new"]).tolist() for n in _lengths(case, np.random.default_rng(case["longest"]))]


def _prepare_layered(case, seed):
    cfg = _layered_config(case)
    folder = tempfile.mkdtemp(prefix="layered_")
    try:
        _save(folder, cfg, _layered_tensors(case, cfg, seed))
        tokens = _layered_tokens(case, seed)
        room = sum(len(t) + 64 for t in tokens)
        eng = _package("serving").ServingEngine(folder, case["dtype"], max_tokens=room, max_seqs=case["seqs"])
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    return dict(case=case, eng=eng, tokens=tokens)


def _run_layered(s):
    """The life of a few requests: all prompts in one step, then `new` steps of one token each (the tokens are given)."""
    eng, new = s["eng"], s["case"]["new"]
    ids = ["r%d" % i for i in range(len(s["tokens"]))]
    out = [eng.step([(r, t[:len(t) - new], [len(t) - new - 1]) for r, t in zip(ids, s["tokens"])])]
    for k in range(new):
        out.append(eng.step([(r, [t[len(t) - new + k]], [0]) for r, t in zip(ids, s["tokens"])]))
    for r in ids:
        eng.finish(r)
    return out


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


@functools.lru_cache(maxsize=None)
def _bucket(n, rows, far):
    """Row of the distance table: its own below rows / 2, then logarithmically wider steps that end at `far`."""
    half = rows // 2
    if n < half:
        return n
    steps, k = rows - half, 0
    while k + 1 < steps and n ** steps * half ** (k + 1) >= Fraction(far) ** (k + 1) * half ** steps:
        k += 1
    return half + k


def _exact_gavodra(case, cfg, T, tokens):
    eps, mult = cfg["norm"]["eps"], cfg["residual_mult"]
    m = cfg["layers"][0]["mixer"]
    H, G, D, limit, n = m["heads"], m["kv_heads"], m["dim"], cfg["layers"][0]["mlp"]["limit"], len(tokens)
    x = T["embed"][tokens] * cfg["embedding"]["scale"]
    idx = torch.arange(n, device="cuda")
    dist = (idx[:, None] - idx[None, :]).clamp_min(0)
    rows = torch.tensor([_bucket(i, 32, 2048) for i in range(n)], device="cuda")[dist]
    hidden = torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1)
    first = None
    for i in range(len(cfg["layers"])):
        p = "l%d.mix." % i
        q = _unit((x @ T[p + "q"].T).view(n, H, D), eps) * T[p + "q.norm"]
        k = _unit((x @ T[p + "k"].T).view(n, G, D), eps) * T[p + "k.norm"]
        v = x @ T[p + "v"].T
        if first is None:
            first = v
        else:
            v = (1 - T[p + "vmix"]) * v + T[p + "vmix"] * first
        v, o = v.view(n, G, D), torch.empty(n, H, D, device="cuda", dtype=torch.float64)
        for h in range(H):
            s = q[:, h] @ k[:, h // (H // G)].T * m["scale"] + T[p + "rel"][rows, h]
            o[:, h] = torch.softmax(s.masked_fill_(hidden, float("-inf")), -1) @ v[:, h // (H // G)]
        o = o * torch.sigmoid(x @ T[p + "g"].T)[:, :, None]
        x = x + mult * _unit(o.reshape(n, H * D) @ T[p + "o"].T, eps) * T["l%d.norm1" % i]
        f = "l%d.mlp." % i
        g, u = (x @ T[f + "gate"].T).clamp_max(limit), (x @ T[f + "up"].T).clamp(-limit, limit)
        x = x + mult * _unit((g * torch.sigmoid(1.702 * g) * (u + 1)) @ T[f + "down"].T, eps) * T["l%d.norm2" % i]
    x = x[n - case["new"] - 1:]
    z = (_unit(x, eps) * T["final.norm"]) @ T["embed"].T * cfg["logit_scale"]
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


def _rotated(x, rot, halves):
    n, dims = x.shape[0], rot["dims"]
    f = float(rot["base"]) ** (-torch.arange(0, dims, 2, device="cuda", dtype=torch.float64) / dims) / rot.get("scaling", {}).get("factor", 1.0)
    ang = (torch.arange(n, device="cuda", dtype=torch.float64)[:, None] * f)[:, None]
    c, s = torch.cos(ang), torch.sin(ang)
    if halves:
        a, b = x[..., :dims // 2], x[..., dims // 2:dims]
        return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)
    a, b = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2), x[..., dims:]], -1)


def _exact_logulix(case, cfg, T, tokens):
    eps, n = cfg["norm"]["eps"], len(tokens)
    e = T["embed"][tokens] * cfg["embedding"]["scale"]
    x = e
    idx = torch.arange(n, device="cuda")
    dist = idx[:, None] - idx[None, :]

    def conv(u, w):
        full = torch.cat([u.new_zeros(w.shape[1] - 1, u.shape[1]), u])
        return sum(w[:, j] * full[j:j + n] for j in range(w.shape[1]))

    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], "l%d.mix." % i
        if i == cfg["loop"]["start"]:
            x = torch.cat([x, e], 1) @ T["loop.in"].T
        h = _unit(x, eps) * T["l%d.norm1" % i]
        if layer["type"] == "attention":
            H, G, D = m["heads"], m["kv_heads"], m["dim"]
            q = conv(h @ T[p + "q"].T + T[p + "q.b"], T[p + "q.conv"])
            k = conv(h @ T[p + "k"].T + T[p + "k.b"], T[p + "k.conv"])
            v = k.view(n, G, D)
            q = _rotated((_unit(q, eps) * T[p + "q.norm"]).view(n, H, D), m["rot"], False)
            k = _rotated((_unit(k, eps) * T[p + "k.norm"]).view(n, G, D), m["rot"], False)
            o = torch.empty(n, H, D, device="cuda", dtype=torch.float64)
            for hh in range(H):
                s = q[:, hh] @ k[:, hh // (H // G)].T * m["scale"]
                s = m["softcap"] * torch.tanh(s / m["softcap"])
                s.masked_fill_((dist < 0) | (dist >= m["mask"]["size"]), float("-inf"))
                o[:, hh] = torch.softmax(s, -1) @ v[:, hh // (H // G)]
            y = o.reshape(n, H * D) @ T[p + "o"].T + T[p + "o.b"]
        elif layer["type"] == "retention":
            H, D, E = m["heads"], m["dim"], m["vdim"]
            q = _rotated((h @ T[p + "q"].T).view(n, H, D), m["rot"], True)
            k = _rotated((h @ T[p + "k"].T).view(n, H, D), m["rot"], True) / math.sqrt(D)
            v = (h @ T[p + "v"].T).view(n, H, E)
            decay = torch.tensor(m["decay"], device="cuda", dtype=torch.float64)
            weight = torch.where(dist >= 0, decay[:, None, None] ** dist.clamp_min(0), torch.zeros((), device="cuda", dtype=torch.float64))
            o = torch.einsum("hts,she->the", torch.einsum("thd,shd->hts", q, k) * weight, v)
            y = (_unit(o, eps).reshape(n, H * E) * torch.nn.functional.silu(h @ T[p + "g"].T)) @ T[p + "o"].T
        else:
            H, D = m["heads"], m["dim"]
            prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
            mixed = {c: h + (prev - h) * T[p + "mu." + c] for c in "rkvgw"}
            r, k, v = ((mixed[c] @ T[p + c].T).view(n, H, D) for c in "rkv")
            w = torch.exp(-torch.exp(torch.tanh(mixed["w"] @ T[p + "w1"].T) @ T[p + "w2"].T + T[p + "w0"])).view(n, H, D)
            S, o = torch.zeros(H, D, D, device="cuda", dtype=torch.float64), torch.empty(n, H, D, device="cuda", dtype=torch.float64)
            for t in range(n):
                kv = k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.einsum("hde,hd->he", torch.addcmul(S, T[p + "u"][:, :, None], kv), r[t])
                S = torch.addcmul(kv, w[t][:, :, None], S)
            y = (_unit(o, eps).reshape(n, H * D) * T[p + "norm"] * torch.nn.functional.silu(mixed["g"] @ T[p + "g"].T)) @ T[p + "o"].T
        x = x + y
        f = "l%d.mlp." % i
        x = x + torch.relu((_unit(x, eps) * T["l%d.norm2" % i]) @ T[f + "up"].T) ** 2 @ T[f + "down"].T
    x = x[n - case["new"] - 1:]
    return (_unit(x, eps) * T["final.norm"]) @ T["head"].T * cfg["logit_scale"]


def _exact_layered(case, seed):
    cfg = _layered_config(case)
    T = {k: _rows64(v) for k, v in _layered_tensors(case, cfg, seed).items()}
    f = _exact_gavodra if case["design"] == "gavodra" else _exact_logulix
    z = torch.stack([f(case, cfg, T, t) for t in _layered_tokens(case, seed)])       # [requests, 1 + new, vocab]
    return [z[:, k].contiguous().cpu() for k in range(z.shape[1])]


def _work_layered(case):
    cfg = _layered_config(case)
    serving = _package("serving")
    shapes = serving.gavodra_tensor_shapes(cfg) if case["design"] == "gavodra" else serving.logulix_tensor_shapes(cfg, 64)
    per = 2.0 if case["dtype"] == "bfloat16" else 4.0
    weights = sum(int(np.prod(s)) for n, s in shapes.items() if n != "embed") + (case["vocab"] * case["width"] if case["design"] == "gavodra" else 0)
    head = case["vocab"] * case["width"]
    lens = _lengths(case, np.random.default_rng(case["longest"]))
    rows, wanted = sum(lens) + case["new"] * len(lens), (1 + case["new"]) * len(lens)
    bytes_, flops = per * weights * (1 + case["new"]) + 4.0 * case["vocab"] * wanted, 2.0 * (weights - head) * rows + 2.0 * head * wanted
    for layer in cfg["layers"]:
        m = layer["mixer"]
        if layer["type"] == "attention":
            window = m.get("mask", {}).get("size", 1 << 30)
            flops += sum(4.0 * m["heads"] * m["dim"] * min(j + 1, window) for n in lens for j in range(n + case["new"]))
            row = 4.0 * 2 * m["kv_heads"] * m["dim"]
            bytes_ += row * rows + row * sum(min(n + j, window) for n in lens for j in range(case["new"]))
        else:
            state = m["heads"] * m["dim"] * m.get("vdim", m["dim"])
            flops += 4.0 * state * rows
            bytes_ += 8.0 * state * len(lens) * (1 + case["new"])
    return {"bytes": bytes_, "flops": flops}


# ---- what is asked for ----------------------------------------------------------------------------------------------------
def prepare(case, seed):
    return _prepare_layered(case, seed) if case["kind"] == "layered" else _prepare_llama(case, seed)


def run(state):
    return _run_layered(state) if state["case"]["kind"] == "layered" else _run_llama(state)


def work(case):
    return _work_layered(case) if case["kind"] == "layered" else _work_llama(case)


def exact(case, seed):
    return _exact_layered(case, seed) if case["kind"] == "layered" else _exact_llama(case, seed)


def tolerance(case):
    """Measured against the 64-bit statement, which rounds nothing.  f32: sums in another order, 3e-5 at most.  q8 and bf16: every
    product's input is rounded to its format (one part in 127 of a group's largest value; one part in 256 of itself).  An input that
    two implementations compute a rounding apart may fall on either side of a step, each such step moves later inputs over theirs,
    and after a few products the two are as far apart as either is from the statement.  Whole values are next tokens: ties, and coins
    at a boundary."""
    if case["kind"] == "layered":
        return {"rel": 0.02, "max": 0.3} if case["dtype"] == "bfloat16" else {"rel": 2e-5, "max": 1e-3}
    return {"f32": {"rel": 1e-4, "max": 1e-3, "differ": 0.01}, "q8": {"rel": 0.03, "max": 0.3, "differ": 0.01},
            "bf16": {"rel": 0.02, "max": 0.3, "differ": 0.01}}[case["weights"]]
