"""bf16 products (csrc/gemm_bf16.cu): few rows, whose tiles are dealt to clusters of CTAs along K, with ragged tiles, ragged and empty shares of
K, every column-tile width and the sizes on both sides of the rule that picks the cluster; and more rows, with every output tile."""
import ctypes as C

import pytest
import torch

from pkgload import load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 16, 17, 33, 64, 65, 128, 129, 384, 700, 1100])
@pytest.mark.parametrize("M,K", [(128, 64), (133, 128), (1024, 256), (1024, 1160), (2048, 1096), (3205, 512), (3208, 1024), (4608, 520), (6401, 256), (12900, 256)])
def test_rows(rows, M, K):
    lib = load_pkg("cabi").lib()
    g = torch.Generator(device="cuda").manual_seed(rows * 1000 + K)
    W = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    X = torch.randn(rows, K + 8, device="cuda", generator=g).to(torch.bfloat16)      # rows a pitch apart
    out = torch.full((rows + 1, M + 3), 7.0, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        lib.check(lib.c.tha_gemm_bf16(None, C.c_void_p(out.data_ptr()), M + 3, C.c_void_p(W.data_ptr()), M, K, C.c_void_p(X.data_ptr()), rows, K + 8))
    torch.cuda.synchronize()
    want = X[:, :K].double() @ W.double().T
    # every product is exact in fp32; K additions of fp32 partial sums: at most K * 2^-24 of the sum of magnitudes
    bound = K * 2.0 ** -24 * (X[:, :K].double().abs() @ W.double().abs().T) + 1e-30
    assert bool(((out[:rows, :M].double() - want).abs() <= bound).all())
    assert bool((out[rows] == 7.0).all()) and bool((out[:, M:] == 7.0).all())       # nothing outside the product
    assert lib.c.tha_gemm_check_error() == 0


@pytest.mark.parametrize("rows", [129, 384, 512])
@pytest.mark.parametrize("M,K", [(1024, 4096), (1024, 4032), (2048, 6144), (1000, 4680)])
def test_prompt_rows_on_both_sides_of_the_line(rows, M, K):
    """More than 128 rows: clusters of four and eight from K = 4096 on, a CTA a tile below."""
    test_rows(rows, M, K)
