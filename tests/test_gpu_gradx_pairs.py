"""grad_X on CTA pairs: batches on either side of the 128, 256 and 512 rows where the tile changes, whole and ragged slices
of the label rows (fewer stages of 64 rows than splits, several segments of 512 rows per split, several launches), against
the CPU oracle.  Results are fp32 sums of bf16 products; the oracle rounds G as the kernels do, so what differs is a
logit that falls on the other side of a bf16 rounding (2^-8 of one term in thousands)."""
import pytest
import torch

from tests._util import rel_inf
from tests.test_gpu_step import _inputs, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["bf16", "fp8", "simfp8"])
@pytest.mark.parametrize("L,d,B,nc,sched", [(100, 256, 129, 1, 0), (1500, 256, 192, 1, 0), (40000, 256, 193, 2, 0),
                                            (3000, 512, 256, 1, 1024), (2600, 256, 257, 1, 0), (9000, 256, 512, 3, 2048),
                                            (700, 256, 700, 1, 0)])
def test_grad_x_on_pairs(mode, L, d, B, nc, sched):
    from oracle import xmc_oracle as O
    bf16 = mode == "bf16"
    w, x, lab = _inputs(L, d, B, 3 * B, seed=L + B, w_dtype=torch.bfloat16 if bf16 else torch.float8_e4m3fn)
    li = ((L + nc - 1) // nc + 15) // 16 * 16
    chunks = [w[i * li:(i + 1) * li] for i in range(nc)]
    if bf16:
        _, want, _ = O.chunked_step(w, x, lab, 0.5, num_chunks=1, rounding="rn", seed=5, step=0)
    else:
        _, want, _ = O.fp8_chunked_step(chunks, x, lab, 0.5, rounding="rn", seed=5, step=0, simulated=(mode == "simfp8"))
    _, got, _, _ = _run_gpu(mode, chunks, x, lab, 0.5, stochastic=False, sched=sched, round_dw=bf16)
    assert rel_inf(got, want) < 1e-2
