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
