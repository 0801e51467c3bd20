"""A plain float64 statement (torch, on the device) of one call of the fp32 llama2 path: rows of several sequences behind contexts that
are already in the cache.  Used where the C oracle, which computes every earlier position too, would take minutes."""
import math

import torch


def forward(cfg, w, cache, seqs):
    """w: DeviceWeights.t; cache(which, slot, layer, n) -> its first n rows [n, kv_dim]; seqs: [(slot, pos0, tokens)].
    Returns (logits of each sequence's last row [len(seqs), vocab], new key rows, new value rows: [rows, layers, kv_dim])."""
    d, H, G, hs = cfg.dim, cfg.n_heads, cfg.n_kv_heads, cfg.dim // cfg.n_heads
    f = {k: v.double() for k, v in w.items()}
    rows = [(s, p0 + j, int(t)) for s, p0, ts in seqs for j, t in enumerate(ts)]
    pos = torch.tensor([r[1] for r in rows], device="cuda", dtype=torch.float64)
    ang = pos[:, None] * (10000.0 ** (-torch.arange(0, hs, 2, device="cuda", dtype=torch.float64) / hs))[None]
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]

    def rot(x):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)

    def rms(x, g):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * g

    x = f["tok_emb"][torch.tensor([r[2] for r in rows], device="cuda")]
    keys, values = [], []
    for l in range(cfg.n_layers):
        h = rms(x, f["rms_att"][l])
        q, k, v = rot((h @ f["wq"][l].T).view(-1, H, hs)), rot((h @ f["wk"][l].T).view(-1, G, hs)), (h @ f["wv"][l].T).view(-1, G, hs)
        keys.append(k.flatten(1))
        values.append(v.flatten(1))
        o, at = torch.empty_like(x), 0
        for slot, p0, ts in seqs:
            n = len(ts)
            K = torch.cat([cache("k", slot, l, p0).double().view(p0, G, hs), k[at:at + n]])
            V = torch.cat([cache("v", slot, l, p0).double().view(p0, G, hs), v[at:at + n]])
            sc = torch.einsum("ngmd,tgd->gmnt", q[at:at + n].view(n, G, H // G, hs), K) / math.sqrt(hs)
            sc = sc.masked_fill(torch.ones(n, p0 + n, device="cuda", dtype=torch.bool).triu(p0 + 1), float("-inf"))
            o[at:at + n] = torch.einsum("gmnt,tgd->ngmd", torch.softmax(sc, -1), V).reshape(n, d)
            at += n
        x = x + o @ f["wo"][l].T
        h = rms(x, f["rms_ffn"][l])
        x = x + (torch.nn.functional.silu(h @ f["w1"][l].T) * (h @ f["w3"][l].T)) @ f["w2"][l].T
    last = torch.tensor([len(ts) for _, _, ts in seqs], device="cuda").cumsum(0) - 1
    return rms(x[last], f["rms_final"]) @ f["wcls"].T, torch.stack(keys, 1), torch.stack(values, 1)
