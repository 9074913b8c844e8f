"""Sums of grad_X over e4m3 weights in the one-kernel step, where it ends them: simulated FP8, and layers rounded to nearest with more
than half as many batch rows as features.  Against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _step_twice(h, x, sr):
    got = []
    for _ in range(2):
        g = torch.full(x.shape, float("nan"), dtype=torch.float32, device="cuda")
        before = h.launch_count
        h.step(x, None, 0.0, seed=1, step=2, stochastic=sr, grad_f32=g)
        assert h.launch_count - before in (3, 6)              # one kernel, the pairs sorted by one block or by others
        got.append(g)
    h.check()
    h.close()
    assert torch.equal(got[0], got[1])                        # one order of additions
    return got[0].double()


@pytest.mark.parametrize("mode,L,B,rows_per_sum", [("fp8", 2800000, 128, 4096), ("fp8", 1000000, 40, 4096), ("simfp8", 1000000, 24, 4096)])
def test_64_features(mode, L, B, rows_per_sum):
    """Weights U(+-1/8) and embeddings with one feature each, so that G is known: the sum of that feature, G times the weights it
    depends on, grows by a unit in 20 rows and outgrows the 24 bits in which products of 2^-19 add up exactly after a few thousand.
    What is left are fp32 additions, of a cluster's sums and of 74 clusters: sqrt(additions) * 2^-24 where they are independent.
    Measured 4.8e-8 to 7.1e-8; sums of all tiles of a cluster 1.2e-6 and 2.9e-5."""
    from elmo_b200 import _lib
    from elmo_b200.handle import XmcHandle
    d, chunks = 64, 8
    gen = torch.Generator(device="cuda").manual_seed(L + B)
    per = -(-L // chunks)
    ws = [((torch.rand(min(per, L - i * per), d, generator=gen, device="cuda") * 2 - 1) / 8).to(torch.float8_e4m3fn) for i in range(chunks)]
    rows = torch.arange(B, device="cuda")
    x = torch.zeros(B, d, device="cuda")
    x[rows, rows % d] = torch.exp2((rows % 4).float())
    x = x.to(torch.bfloat16)
    want = torch.zeros(B, d, dtype=torch.float64, device="cuda")
    lib = _lib.load()
    for w in ws:
        for p in w.split(1 << 16):
            z = (p.double() @ x.double().t()).float().to(torch.bfloat16).contiguous()
            g = torch.empty_like(z)
            _lib.check(lib.xmc_test_sigmoid(0, z.data_ptr(), g.data_ptr(), z.numel(), _lib.raw_stream(0)))
            want += g.double().t() @ p.double()
    h = XmcHandle(torch.device("cuda", 0), d, B, mode)
    h.bind(ws)
    got = _step_twice(h, x, False)
    additions = L / 74 / rows_per_sum + 74 + 8
    assert float((got - want).norm() / want.norm()) < additions ** 0.5 * 2.0 ** -24


@pytest.mark.parametrize("mode,L,d,B,chunks,sr,rows_per_sum", [
    ("fp8", 1400000, 192, 128, 8, False, 4096),
    ("simfp8", 1400000, 64, 16, 8, False, 5120),          # batches up to 64: launches are twice as long
    ("simfp8", 1400000, 256, 100, 8, True, 4096),
    ("simfp8", 1400000, 320, 60, 8, False, 10240),        # 74 splits
    ("simfp8", 606209, 256, 128, 1, True, 4096)])         # the second sum of a cluster has 32 tiles, of one of them 33 and a third
def test_positive_weights(mode, L, d, B, chunks, sr, rows_per_sum):
    """With zero embeddings every logit is 0 and G is exactly 1/2; with positive weights nothing cancels: each addition of 16 rows to
    an accumulator costs at most one unit in the last place (2^-23 relative), each of the fp32 additions behind it half of one."""
    from elmo_b200.handle import XmcHandle
    gen = torch.Generator(device="cuda").manual_seed(L + d)
    per = -(-L // chunks)
    ws, want = [], torch.zeros(d, dtype=torch.float64, device="cuda")
    for i in range(chunks):
        w = torch.empty(min(per, L - i * per), d, dtype=torch.float8_e4m3fn, device="cuda")
        for p in w.split(1 << 18):
            p.copy_(torch.exp2(torch.rand(p.shape, generator=gen, device="cuda") * -10))
            want += 0.5 * p.double().sum(0)
        ws.append(w)
    h = XmcHandle(torch.device("cuda", 0), d, B, mode)
    h.bind(ws)
    got = _step_twice(h, torch.zeros(B, d, dtype=torch.bfloat16, device="cuda"), sr)
    added = L / 74 / rows_per_sum + 74 + 8
    assert float(((got - want) / want).abs().max()) < (2 * rows_per_sum / 16 + added) * 2.0 ** -24
