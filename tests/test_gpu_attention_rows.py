"""Attention of single rows (csrc/hybrid_attn_row.cu): decoded tokens of every attention form with heads of 32 to 128 channels, against
the plain float64 statements of the designs.  Two requests decode together, one with a context that is cut into runs of key tiles
(and crosses the end of a tile and of a cache block on the way), one from its first token on."""
import pytest

import test_gpu_bozovik as TB
import test_gpu_gavodra as TG
import test_gpu_logulix as TL
import test_gpu_mozetar as TM
import test_gpu_timerax as TT

pytestmark = pytest.mark.gpu


def gavodra(tmp, heads, kv_heads, dim, vdim):
    return TG.Built(tmp, TG.model([TG.attention(None, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, bias_max=150, v_mix=False),
                                   TG.attention(None, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, bias_max=35)]), 3)


def bozovik(tmp, heads, kv_heads, dim, vdim):
    return TB.Built(tmp, TB.model([TB.attention(None, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim),
                                   TB.parallel(None, left=TB.attn(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, mask=(90, 5)))]), 4)


def logulix(tmp, heads, kv_heads, dim, vdim):
    return TL.Built(tmp, TL.model([TL.attention(heads=heads, kv_heads=kv_heads, dim=dim, window=130)]), 5)


def mozetar(tmp, heads, kv_heads, dim, vdim):
    return TM.Built(tmp, TM.model([TM.windowed(None, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, window=70),
                                   TM.differential(None, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim),
                                   TM.windowed(None, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, window=70, kv_from=0)]), 6)


def timerax(tmp, heads, kv_heads, dim, vdim):
    return TT.Built(tmp, TT.model_cfg([TT.parallel_cfg(None, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, chunk=300)]), 7)


def logits_of(b, toks):
    z = b.ref(toks)
    return z[0] if isinstance(z, tuple) else z


@pytest.mark.parametrize("design", [gavodra, bozovik, logulix, mozetar, timerax])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(2, 2, 32, 32), (4, 2, 64, 96), (6, 2, 96, 64), (8, 2, 128, 128), (6, 1, 32, 128), (8, 1, 64, 64)])
def test_decoded_tokens(tmp_path, design, heads, kv_heads, dim, vdim):
    b = design(tmp_path, heads, kv_heads, dim, vdim)
    long, short, new = TG.tokens_for(b, 309 + 12, 1), TG.tokens_for(b, 1 + 12, 2), 12
    want = [logits_of(b, long)[-new - 1:], logits_of(b, short)[-new - 1:]]
    for dtype, tol in (("float32", 2e-4), ("bfloat16", 6e-2)):
        e = b.engine(dtype)
        got = [e.step([("l", long[:-new], [len(long) - new - 1]), ("s", short[:1], [0])])]
        for k in range(new):
            got.append(e.step([("l", [long[len(long) - new + k]], [0]), ("s", [short[1 + k]], [0])]))
        for i in range(2):
            for k in range(new + 1):
                assert TG.rel_err(got[k][i], want[i][k]) < tol, (dtype, i, k)
