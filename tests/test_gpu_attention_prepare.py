"""Rows to queries and cache rows (csrc/hybrid_ops.cu): the kernel of four channels a lane against the general one, which takes projections that do not start on 16 bytes."""
import ctypes as C

import numpy as np
import pytest
import torch

import hyb_cabi as H

pytestmark = pytest.mark.gpu
FORMS = {
    "plain": dict(),
    "interleaved": dict(rot=1, turn=1.0),
    "interleaved part, unit": dict(rot=1, turn=0.5, unit_rms=1),
    "halves": dict(rot=1, turn=1.0, rot_layout=1),
    "halves part, unit": dict(rot=1, turn=0.5, rot_layout=1, unit_rms=1),
    "head norms": dict(rot=1, turn=1.0, norms=1, head_norm=1),
    "row norms, halves": dict(rot=1, turn=1.0, rot_layout=1, norms=1),
    "mixed values": dict(v_mix=1, v_mix_layer=0, v_mix_lambda=0.3, unit_rms=1),
    "shared values, growing queries": dict(v_share=2, q_temp_every=16, q_temp_coef=0.4),
    "queries only": dict(rot=1, turn=1.0, kv_shared=1),
    "values are keys": dict(v_is_k=1),
}


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(16, 4, 128, 128), (6, 2, 64, 32), (4, 4, 16, 128), (40, 2, 48, 48)])
@pytest.mark.parametrize("seqs", [[(0, 33, 1), (1, 0, 1)], [(1, 5, 200), (0, 0, 3)]])
def test_forms(form, heads, kv_heads, dim, vdim, seqs):
    f = dict(FORMS[form])
    if f.get("v_is_k"):
        vdim = dim
    turn, norms = f.pop("turn", 0.0), f.pop("norms", 0)
    f.pop("rot", None)
    lib = H.lib()
    rows, keep = H.rows_of(seqs)
    g = torch.Generator(device="cuda").manual_seed(dim + heads)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    R, layers, block, per = rows.n_rows, 2, 16, 16
    kv_dim = kv_heads * max(dim, vdim)
    o_k, o_v = heads * dim, heads * dim + kv_heads * dim
    ldp = o_v + kv_heads * vdim + 4
    proj = rnd(R, ldp)
    table = torch.from_numpy(np.random.default_rng(3).permutation(2 * per).astype(np.int32).reshape(2, per)).cuda()
    rot_dims = int(dim * turn) // 8 * 8
    cos, sin = rnd(R, max(1, rot_dims // 2)), rnd(R, max(1, rot_dims // 2))
    qn = rnd(dim if f.get("head_norm") else heads * dim) if norms else None
    kn = rnd(dim if f.get("head_norm") else kv_heads * dim) if norms else None
    if f.get("v_is_k"):
        f["o_v"] = o_k
    a = H.Attn(**{**dict(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, rot=-1, eps=1e-5, scale=1.0, cache_layer=1, o_q=0, o_k=o_k, o_v=o_v, q_norm=H.ptr(qn), k_norm=H.ptr(kn)),
                  **f})
    pools = [rnd(2 * per, layers, block, kv_dim) for _ in range(2)]
    got = []
    for shift in (0, 1):
        p = torch.empty(R * ldp + 1, device="cuda")
        p[shift:shift + R * ldp] = proj.flatten()
        k, v, q = pools[0].clone(), pools[1].clone(), torch.full((R, heads * dim), float("nan"), device="cuda")
        kv = H.Kv(k.data_ptr(), v.data_ptr(), table.data_ptr(), per, block, layers, kv_dim)
        torch.cuda.synchronize()
        lib.c.tha_hyb_attn_prepare.argtypes = [H.P, C.POINTER(H.Attn), C.POINTER(H.Rows), C.POINTER(H.Kv), H.P, H.L, H.P, H.P, H.I, H.P]
        lib.check(lib.c.tha_hyb_attn_prepare(None, C.byref(a), C.byref(rows), C.byref(kv), p.data_ptr() + 4 * shift, ldp, cos.data_ptr(), sin.data_ptr(), rot_dims, q.data_ptr()))
        torch.cuda.synchronize()
        got.append((q, k, v))
    for x, y in zip(*got):
        assert torch.isfinite(x).all() and torch.equal(x, y)     # the same order of every sum

