"""A layer-program step among other work of its stream: it sees what the kernels ahead of it wrote, its weights included."""
import pytest
import torch

import hyb_cabi as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 40])
def test_weights_written_just_ahead_of_the_step(rows):
    """The output matrix is the result of a call of this library, every block of which has started (and so let its successor launch) long before
    the matrix is complete; the step's product asks for its first weights ahead of its dependency wait."""
    lib, vocab, width = H.lib(), 256, 16384
    g = torch.Generator(device="cuda").manual_seed(1)
    embed = torch.randn(vocab, width, device="cuda", generator=g).to(torch.bfloat16)
    src, gain = torch.randn(vocab, width, device="cuda", generator=g), torch.rand(width, device="cuda", generator=g)
    one = torch.ones(width, device="cuda")
    r, keep = H.rows_of([(0, 0, rows)])
    want_rows = torch.arange(rows, device="cuda", dtype=torch.int32)
    head, logits = torch.zeros(vocab, width, device="cuda", dtype=torch.bfloat16), torch.zeros(rows, vocab, device="cuda")
    stream = torch.cuda.Stream()
    m = H.Model(dtype=H.BF16, width=width, vocab=vocab, eps=1e-6, embed=H.ptr(embed), final_norm=H.Norm(0, H.ptr(one), None, 0.0, 0.0), head=H.ptr(head))

    def write():
        lib.check(lib.c.tha_hyb_rmsnorm(stream.cuda_stream, H.BF16, H.ptr(head), H.ptr(src), H.ptr(gain), 0.0, 1e-6, vocab, width, None))

    def step():
        lib.check(lib.c.tha_hyb_step(stream.cuda_stream, m, r, H.Kv(), H.States(), rows, H.ptr(want_rows), H.ptr(logits), None))

    torch.cuda.synchronize()
    write()
    torch.cuda.synchronize()
    step()
    torch.cuda.synchronize()
    want = logits.clone()
    assert float(want.abs().max()) > 1.0
    for _ in range(20):
        head.zero_()
        logits.zero_()
        torch.cuda.synchronize()
        write()
        step()
        torch.cuda.synchronize()
        assert torch.equal(logits, want)
