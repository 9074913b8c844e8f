"""Preparation and reduction of a step: the positives sorted by one block beside the preparation of X, or by
launches of their own (more than 8 192 pairs, pairs that are not 8-byte aligned, many buckets), and the gradient
written to tensors that start at any element."""
import pytest
import torch

from tests._util import rel_inf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp8", "bf16"])
@pytest.mark.parametrize("nnz,shift,L", [(0, 0, 900), (1, 0, 900), (1024, 0, 900), (1025, 0, 900), (2049, 0, 900), (8192, 0, 900),
                                         (8193, 0, 900), (500, 1, 900),
                                         (700, 0, 128 * 10240 + 5)])
def test_positives_reach_the_gradient(mode, nnz, shift, L):
    from elmo_b200.handle import XmcHandle
    d, B, dev = 64, 70, torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(nnz + shift)
    w = (torch.rand(L, d, generator=gen, device=dev) - 0.5).to(torch.bfloat16 if mode == "bf16" else torch.float8_e4m3fn)
    x = torch.zeros(B, d, device=dev, dtype=torch.bfloat16)          # sigmoid = 1/2 everywhere: G is 1/2 - Y
    rows = torch.randint(0, B, (nnz,), generator=gen, device=dev)
    cols = torch.randint(0, L, (nnz,), generator=gen, device=dev)
    flat = torch.zeros(2 * nnz + shift, dtype=torch.int32, device=dev)
    lab = flat[shift:].view(nnz, 2)
    lab[:, 0], lab[:, 1] = rows, cols
    h = XmcHandle(dev, d, B, mode)
    h.bind([w])
    g32 = torch.full((B, d), float("nan"), device=dev)
    g16 = torch.full((B * d + 1,), float("nan"), dtype=torch.bfloat16, device=dev)[1:].view(B, d)
    y = torch.zeros(B, L, device=dev)
    y[rows, cols] = 1.0
    want = (0.5 - y).double() @ w.double()
    h.step(x, lab if nnz else None, 0.0, stochastic=False, grad_f32=g32, grad_bf16=g16)
    h.check()
    # exact products, fp32 sums of at most 1.3 M terms of size 1/4: relative error below 2^-24 * sqrt(1.3 M) of the
    # terms' root sum of squares; 1e-4 leaves a factor of ten
    assert rel_inf(g32, want) < 1e-4
    assert torch.equal(g16.float(), g32.to(torch.bfloat16).float())
