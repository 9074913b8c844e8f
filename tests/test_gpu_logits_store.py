"""Inference logits where their stores have edges: boxes of 64 columns written by TMA, columns beyond a chunk or at
addresses TMA cannot take by the threads; nothing outside [batch, n_out] is written."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp8", "simfp8", "bf16"])
@pytest.mark.parametrize("rows,n_out,batch", [([5], 5, 1), ([64], 63, 33), ([300, 300, 77], 670, 129), ([301, 301, 20], 622, 40),
                                             ([1040, 1040, 1040], 3100, 300), ([40000], 39999, 200)])
def test_logits_match_matmul_and_stay_inside(mode, rows, n_out, batch):
    from elmo_b200.handle import XmcHandle
    d, dev = 128, torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(n_out)
    dt = torch.bfloat16 if mode == "bf16" else torch.float8_e4m3fn
    ws = [(torch.randn(r, d, generator=gen, device=dev) * 0.25).to(dt) for r in rows]
    x = torch.randn(batch, d, generator=gen, device=dev).to(torch.bfloat16)
    ld = (n_out + 7) // 8 * 8 + 8
    buf = torch.full((batch + 2, ld), 768.0, dtype=torch.bfloat16, device=dev)
    h = XmcHandle(dev, d, batch, mode, w_scale=0.5)
    h.bind(ws)
    h.forward_logits(x, buf[1:batch + 1], n_out)
    h.check()
    xq = x.to(torch.float8_e4m3fn).double() if mode == "fp8" else x.double()
    want = 0.5 * (xq @ torch.cat([w.double() for w in ws]).t())[:, :n_out]
    got = buf[1:batch + 1, :n_out].double()
    # one bf16 rounding (2^-9) of an fp32 sum of 128 exact products, itself off by less than 128 * 2^-24 of the
    # sum of their magnitudes
    bound = want.abs() * 2.0 ** -8 + 128 * 2.0 ** -23 * 0.5 * (xq.abs() @ torch.cat([w.double().abs() for w in ws]).t())[:, :n_out]
    assert bool(((got - want).abs() <= bound).all())
    assert bool((buf[0] == 768).all()) and bool((buf[batch + 1] == 768).all()) and bool((buf[:, n_out:] == 768).all())


@pytest.mark.parametrize("mode,dtype", [("bf16", torch.bfloat16), ("simfp8", torch.bfloat16), ("fp8", torch.float8_e4m3fn)])
@pytest.mark.parametrize("batch", [1, 128, 129, 300])
def test_embeddings_in_place_and_copied(mode, dtype, batch):
    """Embeddings of the operand's type are read in place, from an address that TMA cannot take through a copy: the
    same results bit for bit, though the rows behind the batch hold NaN."""
    from elmo_b200.handle import XmcHandle
    d, rows, dev = 192, 700, torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(batch)
    w = (torch.rand(rows, d, generator=gen, device=dev) - 0.5).to(torch.bfloat16 if mode == "bf16" else torch.float8_e4m3fn)
    x = torch.randn(batch, d, generator=gen, device=dev).to(dtype)
    h = XmcHandle(dev, d, batch, mode)
    h.bind([w])
    results = []
    for shift in (0, 1):
        held = torch.full((batch * d + d + shift,), float("nan"), device=dev).to(dtype)
        here = held[shift:shift + batch * d].view(batch, d)
        here.copy_(x)
        out = torch.zeros(batch, 704, dtype=torch.bfloat16, device=dev)
        h.forward_logits(here, out, rows)
        vals, idx = h.forward_topk(here, 7, rows)
        h.check()
        results.append((out, vals, idx))
    assert results[0][0].isfinite().all() and float(results[0][0].abs().max()) > 0
    for a, b in zip(*results):
        assert torch.equal(a, b)
