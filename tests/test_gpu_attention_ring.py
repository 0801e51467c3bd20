"""Single rows whose run of key tiles goes around the kernel's ring of tiles in flight (csrc/hybrid_attn_row.cu), one run a context: with as many
sequences as fill the GPU without cuts."""
import pytest
import torch

import hyb_cabi as H
import test_gpu_attention_calls as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [H.BF16, H.F32])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,window,keep", [(8, 8, 32, 32, 0, 0), (16, 8, 64, 128, 0, 0), (32, 8, 128, 96, 0, 0), (24, 8, 96, 64, 150, 7)])
def test_long_runs(dtype, heads, kv_heads, dim, vdim, window, keep):
    """Contexts of 1 to 12 tiles that end on, before and behind the end of a tile; fp32 sums of at most 385 products of order one: 1e-6."""
    last = [0, 31, 32, 95, 96, 97, 127, 128, 129, 300, 383, 384] * 7
    a = H.Attn(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, rot=-1, scale=dim ** -0.5, out_f32=1, window=window, keep_first=keep)
    cache = A.Cache(len(last), 385, kv_heads, dim, vdim)
    q = torch.randn(len(last), heads, dim, device="cuda")
    seqs = [(i, p, 1) for i, p in enumerate(last)]
    assert A.rel(A.run(dtype, a, cache, q, seqs, 0), A.want(a, cache, q, seqs)) < 1e-6
