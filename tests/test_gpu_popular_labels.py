"""Positives that share a bucket of 128 labels, on either side of the numbers of pairs that a warp takes at a time: 32 a load,
4 (one-kernel step, batch 48) or 8 (three kernels, batch 200, and 300 with a second tile of batch rows) loads ahead."""
import pytest
import torch

from tests._util import rel_inf
from tests.test_gpu_step import _check_weights, _inputs, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [48, 200, 300])
@pytest.mark.parametrize("pairs", [31, 33, 127, 129, 255, 257, 2100])
def test_pairs_of_one_bucket(batch, pairs):
    from oracle import xmc_oracle as O
    w, x, _ = _inputs(600, 128, batch, 1, seed=batch + pairs)
    at = torch.randperm(batch * 128, generator=torch.Generator().manual_seed(pairs))[:pairs]
    labels = torch.stack([at // 128, 128 + at % 128], 1).to(torch.int32)          # of the second bucket
    want_w, want_gx, want_loss = O.fp8_chunked_step([w], x, labels, 0.5, rounding="rn", seed=5, step=0, compute_loss=True)
    got_w, gx, _, loss = _run_gpu("fp8", [w], x, labels, 0.5, stochastic=False, loss=True)
    _check_weights(got_w, want_w)
    assert rel_inf(gx, want_gx) < 1e-2
    assert abs(loss - want_loss) < 1e-3 * abs(want_loss)


@pytest.mark.parametrize("pairs", [1, 33, 129, 1500])
@pytest.mark.parametrize("L,d", [(300, 64), (600, 128), (25600, 64), (19200, 320)])
def test_pairs_of_one_bucket_bf16(L, d, pairs):
    """One-kernel step of bf16 weights: clusters with one tile and with several, CTAs with no box, one and two."""
    from oracle import xmc_oracle as O
    w, x, _ = _inputs(L, d, 48, 1, seed=L + pairs, w_dtype=torch.bfloat16)
    at = torch.randperm(48 * 128, generator=torch.Generator().manual_seed(pairs))[:pairs]
    last = (L - 1) // 128 * 128                                                      # half of them in the last bucket
    label = torch.where(at % 2 == 0, at // 48, last + at // 48 % (L - last))
    labels = torch.stack([at % 48, label], 1).to(torch.int32)
    want_w, want_gx, want_loss = O.chunked_step(w, x, labels, 0.5, num_chunks=1, rounding="rn", seed=5, step=0, compute_loss=True)
    got_w, gx, _, loss = _run_gpu("bf16", [w], x, labels, 0.5, stochastic=False, loss=True, round_dw=True)
    assert rel_inf(got_w[0], want_w) < 1e-2
    assert rel_inf(gx, want_gx) < 1e-2
    assert abs(loss - want_loss) < 1e-3 * abs(want_loss)
