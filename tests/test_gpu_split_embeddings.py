"""Simulated FP8 (bf16 embeddings, e4m3 weights) on the FP8 tensor cores: the embeddings in two parts whose sum they are.  Rows of
any magnitude, with numbers far below the row's largest, zeros, infinities and NaNs; on either side of the line up to which
inference converts the weights instead; embeddings that start at an odd address; many and few positives (the two preparations
of a step).  Against 64-bit products."""
import pytest
import torch

from tests._util import rel_inf

pytestmark = pytest.mark.gpu
E4M3 = torch.float8_e4m3fn


def _handle(L, d, B, seed):
    from elmo_b200.handle import XmcHandle
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(L, d, generator=g, device="cuda").mul_(0.25).to(E4M3)
    h = XmcHandle(torch.device("cuda", 0), d, B, "simfp8")
    h.bind([w])
    x = (torch.randn(B, d, generator=g, device="cuda") / d ** 0.5).to(torch.bfloat16)
    return h, w, x


def _logits(h, x, L):
    out = torch.empty(x.shape[0], (L + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
    h.forward_logits(x, out, L)
    h.check()
    return out[:, :L]


# labels x 256: 16 rounds of k-steps of 64 features are 4 rounds of tiles, on 148 SMs or on 74 pairs with two batch tiles
@pytest.mark.parametrize("L,d,B", [(256 * 148 * 3 + 9, 256, 2), (256 * 148 * 3, 256, 2), (256 * 148 * 3 + 9, 256, 300), (3000, 1088, 150),
                                   (40000, 768, 5), (40000, 320, 129)])
def test_rows_of_every_kind(L, d, B):
    h, w, x = _handle(L, d, max(B, 8), L + B)
    x = x[:B]
    if B > 100:
        x[3] *= 2.0 ** -100
        x[4] *= 2.0 ** 60
        x[5] = 0
        x[6, 1:] *= 2.0 ** -13                       # most of it below 2^-13 of the row's largest
        x[7] = (x[7].float() * torch.exp2(-torch.arange(d, device="cuda") * 20.0 / d)).to(torch.bfloat16)
    z = _logits(h, x, L)
    want = x.double() @ w.double().t()
    size = x.double().abs() @ w.double().abs().t()
    # one bf16 rounding of the logit and, generously, fp32 sums; numbers below 2^-13 of a row's largest come within 2^-21 of it
    rest = 2.0 ** -21 * x.double().abs().amax(1, keepdim=True) * w.double().abs().sum(1)
    assert bool(((z.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * size + rest + 2.0 ** -126).all())
    h.close()


def test_infinities_and_nan():
    L, d, B = 60000, 512, 140
    h, w, x = _handle(L, d, B, 3)
    x[1, 7] = float("inf")
    x[2, 9] = float("-inf")
    x[3, 100] = float("nan")
    x[4, 11], x[4, 12] = float("inf"), float("-inf")
    z = _logits(h, x, L).float()
    want = x.float() @ w.float().t()
    assert torch.equal(torch.isnan(z), torch.isnan(want)) and torch.equal(torch.isinf(z), torch.isinf(want))
    inf = torch.isinf(want)
    assert torch.equal(z[inf], want[inf])
    fin = torch.isfinite(want)
    assert rel_inf(z[fin], want[fin]) < 1e-2
    h.close()


def test_embeddings_at_an_odd_address():
    L, d, B = 60000, 512, 140
    h, w, x = _handle(L, d, B, 4)
    odd = torch.empty(B * d + 1, dtype=torch.bfloat16, device="cuda")[1:].view(B, d)
    odd.copy_(x)
    assert torch.equal(_logits(h, odd, L), _logits(h, x, L))
    h.close()


@pytest.mark.parametrize("nnz", [300, 3000, 9000])
@pytest.mark.parametrize("d,B", [(64, 40), (192, 140), (1088, 300)])
def test_steps(d, B, nnz):
    from oracle import xmc_oracle as O
    from tests.test_gpu_step import _check_weights, _inputs, _run_gpu
    w, x, lab = _inputs(5000, d, B, nnz, seed=d + nnz)
    x[1] *= 2.0 ** -9
    (want,), want_gx, want_loss = O.fp8_chunked_step([w], x, lab, 0.5, rounding="rn", seed=5, step=3, compute_loss=True, simulated=True)
    (got,), gx, _, loss = _run_gpu("simfp8", [w], x, lab, 0.5, stochastic=False, step=3, loss=True)
    _check_weights([got], [want])
    assert rel_inf(gx, want_gx) < 1e-2
    assert abs(loss - want_loss) < 1e-3 * abs(want_loss)
