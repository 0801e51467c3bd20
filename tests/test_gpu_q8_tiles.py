"""Q8_0 products (csrc/gemm_q8i.cu): every column tile that a launch can take, ragged rows, columns and last slots of K, every group size, against the
reference's loop (sums of a group exact, each of the two products and the addition rounded by itself, groups ascending): the same bits."""
import ctypes as C

import pytest
import torch

from pkgload import load_pkg

pytestmark = pytest.mark.gpu


def product(N, M, K, gs):
    lib = load_pkg("cabi").lib()
    g = torch.Generator(device="cuda").manual_seed(N * 1000 + K + gs)
    W = torch.randint(-127, 128, (M, K), device="cuda", dtype=torch.int8, generator=g)
    X = torch.randint(-127, 128, (N, K), device="cuda", dtype=torch.int8, generator=g)
    G = K // gs
    S = torch.rand(M, G, device="cuda", generator=g) * 0.01
    tile = min(16 if N <= 16 else 32 if N <= 32 else 64, gs)
    ld = -(-N // tile) * tile                                        # the fewest columns of scales that are accepted
    XS = torch.rand(G, ld, device="cuda", generator=g) * 0.01
    out = torch.full((N + 1, M + 3), 7.0, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())
    lib.check(lib.c.tha_matmul_q8_tc(None, p(out), M + 3, p(W), p(S), gs, M, K, p(X), p(XS), ld, N))
    torch.cuda.synchronize()
    assert lib.c.tha_gemm_check_error() == 0
    want = torch.zeros(N, M, device="cuda")
    for i in range(G):
        s = (X[:, i * gs:(i + 1) * gs].double() @ W[:, i * gs:(i + 1) * gs].double().T).float()      # integers below 2^22: exact
        s = s * S[:, i][None]
        s = s * XS[i, :N][:, None]
        want = want + s
    assert torch.equal(out[:N, :M].view(torch.int32), want.view(torch.int32))
    assert bool((out[N] == 7.0).all()) and bool((out[:, M:] == 7.0).all())                           # nothing outside the product


@pytest.mark.parametrize("gs", [32, 64, 128])
@pytest.mark.parametrize("N", [1, 16, 17, 32, 33, 64, 65, 96, 97, 128, 129, 192, 200, 385])
def test_column_tiles(N, gs):
    product(N, 300, 1152, gs)


@pytest.mark.parametrize("N,M,K,gs", [(5, 128, 128, 32), (5, 129, 160, 32), (40, 127, 192, 64), (200, 131, 1088, 64), (70, 260, 416, 32), (130, 5000, 320, 64)])
def test_ragged_k_and_rows(N, M, K, gs):
    product(N, M, K, gs)


@pytest.mark.parametrize("gs", [64, 128])
@pytest.mark.parametrize("N,M", [(900, 1536), (1000, 4100), (2000, 700), (300, 12288), (512, 2048)])
def test_wide_tiles(N, M, gs):
    """Enough columns for tiles of 64, 96 and 128, with several items to a CTA."""
    product(N, M, 768, gs)
