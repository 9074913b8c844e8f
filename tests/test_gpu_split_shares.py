"""The forward of simulated FP8 in the three kernels, where a warp's columns are 16, 32 and 64 of a tile's with the loss, 32 and 64 without, and
bring their scales with them: one batch tile and two, rows of very different magnitude beside each other, positives in every share.  More
than twelve tiles for each cluster of the one-kernel step, which does not take these.  Against the CPU oracle."""
import pytest
import torch

from tests._util import rel_inf
from tests.test_gpu_step import _check_weights, _inputs, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("loss", [True, False])
@pytest.mark.parametrize("B", [5, 17, 33, 64, 65, 128, 129, 300])
def test_shares_of_columns(B, loss):
    from elmo_b200.handle import XmcHandle
    from oracle import xmc_oracle as O
    clusters = torch.cuda.get_device_properties(0).multi_processor_count // 2
    L, d = 128 * (12 * clusters + 3) - 19, 64
    w, x, lab = _inputs(L, d, B, 3 * L // 4, seed=B)             # half of the rows of a tile and more have a positive
    x *= torch.exp2(torch.arange(B) % 7 - 3.0)[:, None]
    x = x.to(torch.bfloat16)
    (want,), want_gx, want_loss = O.fp8_chunked_step([w], x, lab, 0.5, rounding="sr", seed=5, step=1, compute_loss=True, simulated=True)
    h = XmcHandle(torch.device("cuda", 0), d, B, "simfp8")
    wd = w.cuda()
    h.bind([wd])
    gx = torch.empty(B, d, dtype=torch.float32, device="cuda")
    lo = torch.zeros(1, dtype=torch.float64, device="cuda")
    before = h.launch_count
    h.step(x.cuda(), lab.cuda(), 0.5, seed=5, step=1, stochastic=True, compute_loss=loss, grad_f32=gx, loss_out=lo)
    assert h.launch_count - before == 8                            # preparation and sorting in four launches, three kernels, the reduction
    h.check()
    h.close()
    _check_weights([wd.cpu()], [want])
    assert rel_inf(gx.cpu(), want_gx) < 1e-2
    if loss:
        assert abs(float(lo) - want_loss) < 1e-3 * abs(want_loss)
