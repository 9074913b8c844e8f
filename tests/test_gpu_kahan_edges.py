"""Compensated rows with a bf16 buffer, sixteen elements at a time, where that has edges: a head that ends inside a warp's 32
rows, features that fill part of a box of 128 (one-kernel step) or of a tile of 256 (update kernel, batch 160), and a weight
that is not a number, which sends its sixteen elements the careful way.  One step from the same weights and buffer on
both sides: where the updated weights agree the residuals do too, but for the accumulator's last bits, which
move about one bf16 rounding in 10 000."""
import pytest
import torch

from tests._util import frac_equal_bits
from tests.test_gpu_step import _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rounding", ["rn", "sr"])
@pytest.mark.parametrize("B", [24, 48, 128, 160])
@pytest.mark.parametrize("L,d,head", [(200, 320, 37), (130, 64, 130), (400, 576, 129)])
def test_kahan_rows(L, d, head, B, rounding):
    from elmo_b200.handle import XmcHandle
    from oracle import xmc_oracle as O
    w, x, lab = _inputs(L, d, B, 4 * B, seed=L + B)
    w.view(torch.uint8)[5, 17] = 0x7F
    kah = (torch.randn(head, d, generator=torch.Generator().manual_seed(B)) * 0.01).to(torch.bfloat16)
    h = XmcHandle(torch.device("cuda", 0), d, B, "fp8")
    wc, kc = w.clone().cuda(), kah.clone().cuda()
    h.bind([wc])
    h.bind_kahan(kc)
    g = torch.zeros(B, d, dtype=torch.float32, device="cuda")
    h.step(x.cuda(), lab.cuda(), 0.3, seed=5, step=1, stochastic=(rounding == "sr"), grad_f32=g)
    h.check()
    h.close()
    # a weight that is not a number makes its row's logits, and with them everything of that row, not a number
    finite = torch.ones(L, dtype=torch.bool)
    finite[5] = False
    w2 = w.clone()
    w2.view(torch.uint8)[5, 17] = 0
    (want,), _, _ = O.fp8_chunked_step([w2], x, lab, 0.3, rounding=rounding, seed=5, step=1, kahan=kah)
    got, got_k = wc.cpu(), kc.cpu()
    assert frac_equal_bits(got[finite], want[finite]) >= 0.999
    assert torch.isnan(got[5].float()).all() and torch.isnan(got_k[5].float()).all()
    rows = finite[:head]
    same = got[:head][rows].view(torch.uint8) == want[:head][rows].view(torch.uint8)
    bits = got_k[rows].view(torch.int16) == kah[rows].view(torch.int16)
    assert bits[same].float().mean() >= 0.995


@pytest.mark.parametrize("rounding", ["rn", "sr"])
@pytest.mark.parametrize("B", [24, 128, 160])
@pytest.mark.parametrize("L,d,head", [(200, 320, 37), (130, 64, 130)])
def test_e5m2_rows(L, d, head, B, rounding):
    """The same with an e5m2 buffer, and a feature whose residuals leave e5m2's range: they become infinite, as a conversion that
    does not saturate makes them, and so does not one of the fifteen beside it."""
    from elmo_b200.handle import XmcHandle
    from oracle import xmc_oracle as O
    w, x, lab = _inputs(L, d, B, 4 * B, seed=L + B)
    w[:, 3] = 0.0                                             # so that the feature leaves the logits alone
    x[:, 3] = 16384.0
    kah = (torch.randn(head, d, generator=torch.Generator().manual_seed(B)) * 0.01).to(torch.float8_e5m2)
    h = XmcHandle(torch.device("cuda", 0), d, B, "fp8")
    wc, kc = w.clone().cuda(), kah.clone().cuda()
    h.bind([wc])
    h.bind_kahan(kc)
    h.step(x.cuda(), lab.cuda(), 4.0, seed=5, step=1, stochastic=(rounding == "sr"), grad_f32=torch.zeros(B, d, device="cuda"))
    h.check()
    h.close()
    (want,), _, _ = O.fp8_chunked_step([w], x, lab, 4.0, rounding=rounding, seed=5, step=1, kahan=kah)
    got, got_k = wc.cpu(), kc.cpu()
    assert frac_equal_bits(got, want) >= 0.999
    assert bool(torch.isinf(got_k[:, 3].float()).all()) and int(torch.isinf(got_k.float()).sum()) == head
    assert torch.equal(torch.isinf(got_k.float()), torch.isinf(kah.float()))
    same = got[:head].view(torch.uint8) == want[:head].view(torch.uint8)
    assert (got_k.view(torch.uint8) == kah.view(torch.uint8))[same].float().mean() >= 0.995
