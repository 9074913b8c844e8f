"""fp32 grad_X of bf16 weights over many label rows, against 64 bits.

The tensor core truncates where it adds to an accumulator, so what one accumulator sums up has to stay short.  With zero
embeddings every logit is 0 and G is exactly 1/2; with positive weights nothing cancels: each of the n additions of a
sum costs at most one unit in the last place (2^-23 relative), those that put the sums together half of one.  Measured
2e-7 to 8e-7 against bounds of 6e-6 to 1.7e-5; sums as long as the launch 1e-5 to 7e-5."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS_PER_SUM = 512                       # with 74 splits and more, and on CTA pairs; 16 rows per addition


@pytest.mark.parametrize("L,d,B,chunks,sums", [
    (2000000, 64, 8, 3, 74),             # one-kernel step, one box of features: the second CTA of a cluster has none
    (700003, 256, 33, 7, 74),            # one box per CTA
    (300000, 320, 100, 1, 74),           # two boxes and one
    (120000, 768, 128, 2, 74),           # three boxes each, the largest batch
    (1000, 128, 5, 1, 8),                # fewer tiles than one sum takes
    (94720, 128, 64, 1, 74),             # ten tiles each: two sums and a remainder
    (75776, 128, 64, 1, 74),             # eight tiles each: the last sum ends with the last tile
    (2000000, 64, 130, 3, 148),          # three kernels, one launch
    (400000, 256, 256, 5, 74),           # CTA pairs: 74 splits, ten segments each in alternating accumulators
    (200000, 768, 130, 3, 24),           # three feature tiles, 24 splits; the second CTA of a pair has two of its 128 batch rows
    (100003, 768, 300, 2, 12),           # two batch tiles, the last of 44 rows: its second CTA has none
    (200001, 320, 300, 2, 37)])
def test_long_sums_stay_short_in_the_accumulator(L, d, B, chunks, sums):
    from elmo_b200.handle import XmcHandle
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(L + d)
    per = -(-L // chunks)
    # of all magnitudes from 2^-12 on, so that a sum needs more than 24 bits
    ws = [torch.exp2(torch.rand(min(per, L - i * per), d, generator=gen, device=dev) * -12).to(torch.bfloat16) for i in range(chunks)]
    want = 0.5 * sum(p.double().sum(0) for w in ws for p in w.split(1 << 18))
    x = torch.zeros(B, d, dtype=torch.bfloat16, device=dev)
    h = XmcHandle(dev, d, B, "bf16", sched_labels=-(-L // 256) * 256 + 256 * chunks)
    h.bind(ws)
    got = []
    for _ in range(2):
        g = torch.full((B, d), float("nan"), dtype=torch.float32, device=dev)
        h.step(x, None, 0.0, seed=1, step=2, stochastic=False, round_dw_bf16=True, grad_f32=g)
        got.append(g)
    h.check()
    h.close()
    err = float(((got[0].double() - want) / want).abs().max())
    added = L / sums / ROWS_PER_SUM + sums + 8
    assert err < (2 * (ROWS_PER_SUM + 192) / 16 + added) * 2.0 ** -24, err
    assert torch.equal(got[0], got[1])                        # one order of additions


@pytest.mark.parametrize("mode,L,d,B,chunks,additions", [
    ("fp8", 670091, 768, 140, 11, 59), ("fp8", 670091, 768, 256, 11, 34), ("fp8", 500000, 768, 200, 10, 31),
    ("fp8", 670091, 768, 300, 11, 34), ("simfp8", 400000, 512, 230, 5, 43), ("fp8", 300000, 768, 100, 4, 75)])
def test_e4m3_weights(mode, L, d, B, chunks, additions):
    """Weights U(+-1/sqrt(d)), whose sums the accumulators hold exactly: they are multiples of 2^-9 and G, between 0.2 and 0.8, of
    2^-10, so that a sum below 32 needs no more than 24 bits.  What is left are the fp32 additions of splits and launches, each
    off by half a unit in the last place of a sum that is, in its 2-norm, no larger than the result: sqrt(additions) * 2^-24
    where they are independent, measured 4.2e-8 to 5.1e-8.  Embeddings with one feature each make every logit one product, so
    that G is known: the bf16 sigmoid as the library's own hook gives it."""
    from elmo_b200 import _lib
    from elmo_b200.handle import XmcHandle
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(L + d)
    per = -(-L // chunks)
    ws = [((torch.rand(min(per, L - i * per), d, generator=gen, device=dev) * 2 - 1) / d ** 0.5).to(torch.float8_e4m3fn) for i in range(chunks)]
    rows = torch.arange(B, device=dev)
    x = torch.zeros(B, d, device=dev)
    x[rows, rows % d] = torch.exp2((rows % 4 + 2).float())
    x = x.to(torch.bfloat16)
    want = torch.zeros(B, d, dtype=torch.float64, device=dev)
    lib = _lib.load()
    for w in ws:
        for p in w.split(1 << 16):
            z = (p.double() @ x.double().t()).float().to(torch.bfloat16).contiguous()
            g = torch.empty_like(z)
            _lib.check(lib.xmc_test_sigmoid(0, z.data_ptr(), g.data_ptr(), z.numel(), _lib.raw_stream(0)))
            assert float(g.min()) > 0.2 and float(g.max()) < 0.8
            want += g.double().t() @ p.double()
    h = XmcHandle(dev, d, B, mode)
    h.bind(ws)
    got = torch.zeros(B, d, dtype=torch.float32, device=dev)
    h.step(x, None, 0.0, seed=1, step=2, stochastic=False, grad_f32=got)
    h.check()
    h.close()
    assert float((got.double() - want).norm() / want.norm()) < additions ** 0.5 * 2.0 ** -24
