"""Launches over several weight chunks and chunks over several launches, on CTA pairs: tiles that pad a chunk lie in
the middle of a launch, a launch may begin and end inside a chunk, the last chunk is shorter."""
import pytest
import torch

from tests._util import rel_inf
from tests.test_gpu_step import _check_weights, _inputs, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp8", "simfp8"])
@pytest.mark.parametrize("rows,sched", [([300, 300, 40], 0), ([300, 300, 40], 512), ([128, 128, 128, 1], 256), ([1000, 1000], 768)])
def test_step_over_chunks_and_launches(mode, rows, sched):
    from oracle import xmc_oracle as O
    B, d, L = 200, 128, sum(rows)
    w, x, lab = _inputs(L, d, B, 600, seed=L + sched)
    chunks = list(torch.split(w, rows))
    want_w, want_gx, want_loss = O.fp8_chunked_step(chunks, x, lab, 0.5, simulated=(mode == "simfp8"), rounding="sr", seed=5, step=2,
                                                    compute_loss=True)
    got_w, g32, _, loss = _run_gpu(mode, chunks, x, lab, 0.5, stochastic=True, step=2, loss=True, sched=sched)
    _check_weights(got_w, want_w)
    assert rel_inf(g32, want_gx) < 1e-2
    assert abs(loss - want_loss) < 1e-3 * abs(want_loss)
