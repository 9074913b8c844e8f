"""Top-k of a single window, whose logits leave in boxes of 32 batch rows x 32 labels, or at batches up to 64 (simulated FP8 with converted weights: 48) by the threads:
batches and label counts on either side of boxes, warps and tiles, real and simulated FP8 (one and two boxes per warp),
against the selection from xfc_forward's logits.  The same bf16 logits on both sides: values are equal, and labels where no
two values tie."""
import pytest
import torch

from tests.test_gpu_step import _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp8", "simfp8", "bf16"])
@pytest.mark.parametrize("B", [1, 15, 16, 33, 48, 49, 64, 65, 128, 129, 257])
@pytest.mark.parametrize("L,n_out", [(33, 20), (64, 33), (272, 255), (272, 257), (1500, 1499)])
def test_one_window(mode, B, L, n_out, d=128):
    from elmo_b200.handle import XmcHandle
    w, x, _ = _inputs(L, d, B, 1, seed=L + B, w_dtype=torch.bfloat16 if mode == "bf16" else torch.float8_e4m3fn)
    h = XmcHandle(torch.device("cuda", 0), d, B, mode)
    h.bind([w.cuda()])
    out = torch.empty(B, (n_out + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
    h.forward_logits(x.cuda(), out, n_out)
    vals, idx = h.forward_topk(x.cuda(), 9, n_out)
    h.check()
    z = out[:, :n_out].float()
    assert torch.equal(vals, z.topk(9, dim=1).values)
    assert torch.equal(z.gather(1, idx.long()), vals)
    assert all(len(set(r)) == 9 for r in idx.tolist())
    h.close()


@pytest.mark.parametrize("mode", ["fp8", "simfp8", "bf16"])
@pytest.mark.parametrize("d", [512, 576])
def test_one_window_of_longer_rows(mode, d):
    """On either side of the features up to which FP8 logits of 65 to 128 rows leave in boxes (bf16 ones: never, with rows this long)."""
    test_one_window(mode, 100, 1500, 1499, d)
