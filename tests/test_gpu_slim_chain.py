"""The one-kernel step where its links and buffers come round several times: one box of features a CTA (X^T fetched once, three
buffers for G) and more, an idle second CTA, bf16 sums that start anew while weight slots outnumber boxes, batches on either side
of 64 and 128 padded columns, both roundings, more tiles than clusters.  Against the CPU oracle."""
import pytest
import torch

from tests._util import frac_equal_bits, rel_inf
from tests.test_gpu_step import _check_weights, _inputs, _run_gpu

pytestmark = pytest.mark.gpu


def _one_kernel(mode, w, x, rounding, loss):
    from elmo_b200.handle import XmcHandle
    h = XmcHandle(torch.device("cuda", 0), x.shape[1], x.shape[0], mode)
    h.bind([w.clone().cuda()])
    lo = torch.zeros(1, dtype=torch.float64, device="cuda")
    h.profile(True)
    h.step(x.cuda(), None, 0.0, seed=1, step=2, stochastic=rounding == "sr", compute_loss=loss, round_dw_bf16=mode == "bf16", loss_out=lo)
    kinds = h.profile(False, read=True)
    h.close()
    return "forward" not in kinds


@pytest.mark.parametrize("mode,d,B,rounding", [
    ("fp8", 64, 17, "rn"), ("fp8", 64, 128, "rn"), ("fp8", 128, 64, "sr"), ("fp8", 128, 97, "rn"), ("fp8", 192, 65, "sr"),
    ("fp8", 256, 16, "sr"), ("fp8", 256, 48, "rn"), ("fp8", 256, 128, "sr"), ("fp8", 320, 100, "rn"), ("fp8", 512, 96, "sr"),
    ("fp8", 1024, 64, "rn"), ("simfp8", 64, 17, "rn"), ("simfp8", 64, 128, "rn"), ("simfp8", 128, 96, "sr"), ("simfp8", 192, 64, "sr"), ("simfp8", 256, 40, "rn"), ("simfp8", 768, 33, "sr"),
    ("simfp8", 1024, 64, "sr"), ("simfp8", 768, 128, "sr"), ("simfp8", 384, 90, "rn"), ("fp8", 384, 90, "sr"), ("fp8", 768, 128, "rn"),
    ("fp8", 512, 128, "sr"), ("fp8", 1024, 96, "sr"), ("fp8", 1536, 64, "sr"), ("bf16", 64, 32, "sr"), ("bf16", 128, 128, "rn"), ("bf16", 192, 96, "sr"), ("bf16", 256, 16, "sr"),
    ("bf16", 320, 128, "sr"), ("bf16", 384, 40, "sr"), ("bf16", 512, 100, "rn"), ("bf16", 768, 128, "sr"), ("bf16", 1024, 64, "sr"),
    ("bf16", 384, 96, "sr"), ("bf16", 512, 40, "rn"), ("bf16", 512, 96, "sr"), ("bf16", 640, 128, "sr"), ("bf16", 768, 80, "rn")])
def test_links_come_round(mode, d, B, rounding):
    from oracle import xmc_oracle as O
    clusters = torch.cuda.get_device_properties(0).multi_processor_count // 2
    L = 128 * (7 * clusters + 3) - 19                       # seven or eight tiles a cluster, the last one ragged
    bf16 = mode == "bf16"
    w, x, lab = _inputs(L, d, B, 4 * B, seed=d + B, w_std=0.05 if bf16 else 0.25, w_dtype=torch.bfloat16 if bf16 else torch.float8_e4m3fn)
    if bf16:
        want, want_gx, want_loss = O.chunked_step(w, x, lab, 0.5, num_chunks=1, rounding=rounding, seed=5, step=1, compute_loss=True)
    else:
        (want,), want_gx, want_loss = O.fp8_chunked_step([w], x, lab, 0.5, rounding=rounding, seed=5, step=1, compute_loss=True,
                                                        simulated=mode == "simfp8")
    (got,), gx, _, loss = _run_gpu(mode, [w], x, lab, 0.5, stochastic=rounding == "sr", step=1, loss=True, round_dw=bf16)
    _check_weights([got], [want], min_equal=0.995 if bf16 else 0.999)
    assert rel_inf(gx, want_gx) < 1e-2
    assert abs(loss - want_loss) < 1e-3 * abs(want_loss)
    # the kernel without the loss does the same arithmetic in the same order; real FP8 of 64 features takes three with it
    (again,), gx2, _, _ = _run_gpu(mode, [w], x, lab, 0.5, stochastic=rounding == "sr", step=1, round_dw=bf16)
    three = mode == "fp8" and d == 64 and B > 32
    assert _one_kernel(mode, w, x, rounding, False) and _one_kernel(mode, w, x, rounding, True) != three
    if not three:
        assert frac_equal_bits(again, got) == 1.0 and torch.equal(gx2, gx)
    _check_weights([again], [want], min_equal=0.995 if bf16 else 0.999)
    assert rel_inf(gx2, want_gx) < 1e-2
