"""The updates (of the one-kernel step up to batch 128, else the update kernel) where their tiling and their random stream have edges, against the CPU oracle: bf16 weights
pass through shared memory in two parts of 128 columns (part wholly, partly or not beyond the features; more
tiles than CTAs), and the Philox counter's high word changes in the middle of a launch."""
import pytest
import torch

from tests.test_gpu_step import _check_weights, _inputs, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rounding", ["rn", "sr"])
@pytest.mark.parametrize("L,d,B", [(129, 64, 1), (1023, 192, 65), (700, 320, 300), (128 * 301 + 3, 256, 40),
                                   (129, 64, 130), (1023, 192, 165), (128 * 301 + 3, 256, 140)])
def test_bf16_update_parts(L, d, B, rounding):
    from oracle import xmc_oracle as O
    w, x, lab = _inputs(L, d, B, 3 * B, seed=L, w_std=0.05, w_dtype=torch.bfloat16)
    want_w, _, _ = O.chunked_step(w, x, lab, 0.5, num_chunks=1, rounding=rounding, seed=5, step=2 ** 33 + 7)
    got_w, _, _, _ = _run_gpu("bf16", [w], x, lab, 0.5, stochastic=(rounding == "sr"), step=2 ** 33 + 7, round_dw=True)
    # dW is rounded to bf16 first: a sum of B products that the two sides add in different orders lands on the
    # other side of a bf16 step for about B * 2^-24 * 2^8 of the elements (B 300: 0.5 %)
    _check_weights(got_w, [want_w], min_equal=0.995)


@pytest.mark.parametrize("B", [37, 200])
@pytest.mark.parametrize("mode", ["fp8", "bf16"])
def test_random_stream_across_the_high_counter_word(mode, B):
    from oracle import xmc_oracle as O
    L, d = 300, 64
    off = 2 ** 35 // d - 150            # element 2^35 (counter 2^32) is the first one of row 150
    w, x, lab = _inputs(L, d, B, 60, seed=3, w_std=0.05, w_dtype=torch.bfloat16 if mode == "bf16" else torch.float8_e4m3fn)
    lab[:, 1] += off
    if mode == "fp8":
        (want,), _, _ = O.fp8_chunked_step([w], x, lab, 0.5, rounding="sr", seed=2 ** 40 + 9, step=3, label_offset=off)
    else:
        want, _, _ = O.chunked_step(w, x, lab, 0.5, num_chunks=1, rounding="sr", seed=2 ** 40 + 9, step=3, label_offset=off)
    got, _, _, _ = _run_gpu(mode, [w], x, lab, 0.5, stochastic=True, seed=2 ** 40 + 9, step=3, label_offset=off,
                            round_dw=(mode == "bf16"))
    _check_weights(got, [want], min_equal=0.995)


@pytest.mark.parametrize("B", [16, 160])
def test_bf16_weights_at_the_end_of_their_range(B):
    """Stochastic rounding of bf16 weights: what rounds up past the largest becomes infinite, as the reference's addition of
    random bits makes it, bit for bit; infinite updates stay infinite; a row with something that is not a number, or with an
    infinity that meets a zero in its logits, is not a number afterwards (the addition would leave -0)."""
    from oracle import xmc_oracle as O
    L, d = 512, 128
    largest = torch.finfo(torch.bfloat16).max
    w = torch.zeros(L, d, dtype=torch.bfloat16)
    w[:128, 1], w[128:256, 1] = largest, -largest
    x = torch.zeros(B, d, dtype=torch.bfloat16)
    x[0, 1] = 2.0 ** 100
    lab = torch.tensor([[0, i] for i in range(128, 256)], dtype=torch.int32)      # logits of -inf: G = -1
    # every update is +-(largest + 2^119), half a unit in the last place past the largest, or W - lr dW with dW = 2^99
    want, _, _ = O.chunked_step(w, x, lab, -2.0 ** 19, num_chunks=1, rounding="sr", seed=5, step=2)
    (got,), _, _, _ = _run_gpu("bf16", [w], x, lab, -2.0 ** 19, stochastic=True, step=2, round_dw=True)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert 20 < int(torch.isinf(got[:128, 1].float()).sum()) < 108 and not bool(torch.isnan(got.float()).any())
    bad = w.clone()
    bad[300, 5], bad[310, 5], bad[320, 5] = float("nan"), float("inf"), float("-inf")
    (got,), _, _, _ = _run_gpu("bf16", [bad], x, lab, -2.0 ** 60, stochastic=True, step=2, round_dw=True)
    rows = torch.zeros(L, dtype=torch.bool)
    rows[[300, 310, 320]] = True
    assert bool(torch.isnan(got[rows].float()).all()) and not bool(torch.isnan(got[~rows].float()).any())
    assert bool(torch.isinf(got[~rows][:, 1].float()).all())
