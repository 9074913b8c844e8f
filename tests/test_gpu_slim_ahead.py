"""The one-kernel step of e4m3 weights with stochastic rounding, three boxes of 128 features and more: CTAs of a cluster with unequal
numbers of boxes, one among them; one tile, clusters with one and two tiles, and with three and four, so that G's buffers and
every barrier come round again; the same with compensated rows.  Against the CPU oracle."""
import pytest
import torch

from tests._util import frac_equal_bits, rel_inf
from tests.test_gpu_step import _check_weights, _inputs, _run_gpu

pytestmark = pytest.mark.gpu


def _labels(rounds, more):
    """Label rows of `rounds` tiles of 128 for every cluster and `more` tiles on top, the last one ragged."""
    clusters = torch.cuda.get_device_properties(0).multi_processor_count // 2
    tiles = rounds * clusters + more
    return 128 * tiles - 7 * (tiles > 1)


@pytest.mark.parametrize("B", [3, 40, 64])
@pytest.mark.parametrize("d", [320, 384, 512, 576, 768])
@pytest.mark.parametrize("rounds,more", [(0, 1), (1, 0), (1, 1), (3, 8)])
def test_two_boxes_ahead(rounds, more, d, B):
    if rounds == 3 and (B, d) not in ((3, 320), (40, 576), (64, 320), (64, 768)):
        pytest.skip("the CPU oracle takes the largest size at four shapes only")
    from oracle import xmc_oracle as O
    L = _labels(rounds, more)
    w, x, lab = _inputs(L, d, B, 3 * B, seed=L + d)
    (want,), want_gx, want_loss = O.fp8_chunked_step([w], x, lab, 0.5, rounding="sr", seed=5, step=1, compute_loss=True)
    (got,), gx, _, loss = _run_gpu("fp8", [w], x, lab, 0.5, stochastic=True, step=1, loss=True)
    _check_weights([got], [want])
    assert rel_inf(gx, want_gx) < 1e-2
    assert abs(loss - want_loss) < 1e-3 * abs(want_loss)


@pytest.mark.parametrize("loss", [False, True])
@pytest.mark.parametrize("terms", [torch.bfloat16, torch.float8_e5m2])
@pytest.mark.parametrize("rounds,more,d,B", [(1, 1, 320, 40), (3, 8, 576, 40), (3, 8, 768, 17), (3, 8, 1024, 60), (2, 1, 128, 60),
                                             (2, 1, 576, 100)])
def test_compensated_rows(rounds, more, d, B, terms, loss):
    """Compensated rows in several tiles of a cluster, the last of them in part: bf16 terms and e5m2 ones, up to batch 64 and
    beyond.  Where the updated weights agree with
    the oracle's the terms do too, but for the accumulator's last bits, which move about one bf16 rounding in 10 000."""
    from elmo_b200.handle import XmcHandle
    from oracle import xmc_oracle as O
    L = _labels(rounds, more)
    head = L * 3 // 5 // 128 * 128 + 37
    w, x, lab = _inputs(L, d, B, 4 * B, seed=L + B)
    kah = (torch.randn(head, d, generator=torch.Generator().manual_seed(B)) * 0.01).to(terms)
    h = XmcHandle(torch.device("cuda", 0), d, B, "fp8")
    wc, kc = w.clone().cuda(), kah.clone().cuda()
    h.bind([wc])
    h.bind_kahan(kc)
    g = torch.zeros(B, d, dtype=torch.float32, device="cuda")
    lo = torch.zeros(1, dtype=torch.float64, device="cuda")
    h.step(x.cuda(), lab.cuda(), 0.3, seed=5, step=1, stochastic=True, compute_loss=loss, grad_f32=g, loss_out=lo)
    h.check()
    h.close()
    (want,), want_gx, want_loss = O.fp8_chunked_step([w], x, lab, 0.3, rounding="sr", seed=5, step=1, kahan=kah, compute_loss=loss)
    got, got_k = wc.cpu(), kc.cpu()
    assert frac_equal_bits(got, want) >= 0.999
    assert rel_inf(g.cpu(), want_gx) < 1e-2
    bits = torch.int16 if terms == torch.bfloat16 else torch.uint8
    same = got[:head].view(torch.uint8) == want[:head].view(torch.uint8)
    assert (got_k.view(bits) == kah.view(bits))[same].float().mean() >= 0.995
    if loss:
        assert abs(float(lo) - want_loss) < 1e-3 * abs(want_loss)
