"""A feed-forward's first product with its activation in the read-out against the product and the activation as two kernels: the same
accumulators through the same function, so the same bits."""
import ctypes as C

import pytest

import hyb_cabi as H

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# sides of the rule's lines (128 and 256 rows), ragged rows, ragged and odd widths, offsets, a stack with rows of no part of it
@pytest.mark.parametrize("rows,ff,K,gap", [(128, 256, 128, 0), (129, 128, 64, 0), (256, 300, 192, 0), (257, 131, 72, 0), (300, 1000, 512, 5), (511, 129, 1024, 8),
                                           (2049, 640, 256, 0), (1025, 6144, 128, 3)])
@pytest.mark.parametrize("act", [0, 1, 2, 3, 4])
def test_same_bits_as_two_kernels(rows, ff, K, gap, act):
    lib = H.lib().c
    gated = act not in (1, 3)
    g = torch.Generator("cuda").manual_seed(rows + ff + act)
    N = (2 if gated else 1) * ff + gap
    ldg = (N + 3) // 4 * 4 + 4
    A = (torch.randn(rows, K, device="cuda", generator=g) * 3).bfloat16()
    W = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    A[rows // 2] = float("inf")
    A[rows - 1, 0] = float("nan")
    gu = torch.empty(rows, ldg, device="cuda")
    want, got = (torch.full((rows + 1, ff), -7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    col_u, col_g = (N - ff, gap // 2) if gated else (gap, -1)
    limit, alpha = (1.5, 1.702) if act == 0 else (0.8, 0.3)
    ptr = lambda t: C.c_void_p(t.data_ptr())
    ll, f = C.c_longlong, C.c_float
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.tha_hyb_linear(s, 0, ptr(gu), ll(ldg), ptr(A), ll(K), 0, None, ptr(W), ll(0), rows, N, K, None, 0) == 0
    assert lib.tha_hyb_ff_act(s, 0, act, ptr(want), ptr(gu), ll(ldg), col_g, col_u, rows, ff, f(limit), f(alpha)) == 0
    gu.fill_(0)
    assert lib.tha_hyb_linear_act(s, 0, act, ptr(got), ptr(gu), ll(ldg), ptr(A), ptr(W), rows, N, K, col_g, col_u, ff, f(limit), f(alpha)) == 0
    torch.cuda.synchronize()
    assert torch.equal(want.view(torch.int16), got.view(torch.int16))
