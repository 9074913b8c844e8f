"""Split embeddings where they are split for certain -- a call that splits has a launch of its own for it, one that converts the weights
reads aligned bf16 embeddings in place -- on single CTAs and CTA pairs: infinities and NaNs, embeddings at an odd address, e4m3
embeddings, and the fused top-k, whose first window leaves by threads up to 64 rows and by boxes beyond."""
import pytest
import torch

from tests._util import rel_inf

pytestmark = pytest.mark.gpu
E4M3 = torch.float8_e4m3fn
SHAPES = [(60000, 768, 40), (95000, 512, 140)]        # one CTA: 2 rounds of 24 k-steps of 64; pairs: 6 rounds of 8


def _handle(L, d, B, seed, chunks=1, **kw):
    from elmo_b200.handle import XmcHandle
    g = torch.Generator(device="cuda").manual_seed(seed)
    per = -(-L // chunks // 16) * 16
    ws = []
    for i in range(chunks):
        w = torch.randn(min(per, L - i * per), d, generator=g, device="cuda").mul_(0.25)
        ws.append(torch.where(w.abs() < 2.0 ** -8, 2.0 ** -8, w).to(E4M3))       # no zeros: infinity times one is a NaN
    h = XmcHandle(torch.device("cuda", 0), d, B, "simfp8", **kw)
    h.bind(ws)
    x = (torch.randn(B, d, generator=g, device="cuda") / d ** 0.5).to(torch.bfloat16)
    return h, torch.cat([w.float() for w in ws]), x


def _logits(h, x, L, launches=2):
    out = torch.empty(x.shape[0], (L + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
    before = h.launch_count
    h.forward_logits(x, out, L)
    assert h.launch_count - before == launches
    h.check()
    return out[:, :L]


def _special(x):
    x = x.clone()
    x[1, 7] = float("inf")
    x[2, 9] = float("-inf")
    x[3, 100] = float("nan")
    x[4, 11], x[4, 12] = float("inf"), float("-inf")
    x[5, 3], x[5, 4] = float("inf"), 2.0 ** 20                # a wide row
    x[6, 3], x[6, 4] = float("nan"), 2.0 ** 20
    return x


def _odd(x):
    odd = torch.empty(x.numel() + 1, dtype=x.dtype, device="cuda")[1:].view(x.shape)
    return odd.copy_(x)


@pytest.mark.parametrize("L,d,B", SHAPES)
def test_infinities_and_nan(L, d, B):
    h, w, x = _handle(L, d, B, 3)
    x = _special(x)
    z = _logits(h, x, L).float()
    want = x.float() @ w.t()
    assert torch.equal(torch.isnan(z), torch.isnan(want)) and torch.equal(torch.isinf(z), torch.isinf(want))
    inf = torch.isinf(want)
    assert torch.equal(z[inf], want[inf])
    fin = torch.isfinite(want)
    assert rel_inf(z[fin], want[fin]) < 1e-2
    h.close()


@pytest.mark.parametrize("L,d,B", SHAPES)
def test_embeddings_at_an_odd_address(L, d, B):
    h, _, x = _handle(L, d, B, 4)
    x[2, 5] = 2.0 ** 16
    assert torch.equal(_logits(h, _odd(x), L), _logits(h, x, L))
    h.close()


@pytest.mark.parametrize("d,B,launches", [(768, 40, 3), (768, 140, 5)])
def test_steps_with_infinities_and_at_an_odd_address(d, B, launches):
    L = 5000
    h, w, x = _handle(L, d, B, 5)
    keep = w.to(E4M3)

    def step(x):
        h._keep[0].copy_(keep)
        gx = torch.empty(B, d, dtype=torch.float32, device="cuda")
        before = h.launch_count
        h.step(x, None, 0.0, seed=1, step=2, stochastic=True, grad_f32=gx)
        assert h.launch_count - before == launches
        h.check()
        return gx
    assert torch.equal(step(_odd(x)), step(x))
    x = _special(x)
    z = (x.double() @ w.double().t()).to(torch.bfloat16)
    want = torch.sigmoid(z.double()).to(torch.bfloat16).double() @ w.double()
    gx = step(x)
    assert torch.equal(torch.isnan(gx), torch.isnan(want))
    rows = ~torch.isnan(want).any(1)
    assert bool(rows[[1, 2, 5]].all()) and not bool(rows[[3, 4, 6]].any())
    assert rel_inf(gx[rows], want[rows]) < 1e-2
    h.close()


@pytest.mark.parametrize("L,d,B", SHAPES)
def test_e4m3_embeddings(L, d, B):
    h, w, x = _handle(L, d, B, 6, w_scale=0.5)
    x8 = (x.float() * d ** 0.5).to(E4M3)
    z = _logits(h, x8, L)
    want = 0.5 * (x8.double() @ w.double().t())
    size = 0.5 * (x8.double().abs() @ w.double().abs().t())
    assert bool(((z.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * size).all())
    h.close()


@pytest.mark.parametrize("embed", [torch.bfloat16, E4M3])
@pytest.mark.parametrize("L,d,B,chunks,sched,n_out", [
    (60000, 768, 1, 1, 0, 60000), (60000, 768, 64, 2, 16384, 59990), (60000, 768, 65, 2, 16384, 59990), (120000, 256, 128, 3, 0, 120000),
    (60016, 768, 129, 1, 0, 60001), (60000, 768, 300, 2, 16384, 59990)])
def test_topk_selects_from_the_logits(L, d, B, chunks, sched, n_out, embed):
    """Bit for bit what the layer's own logits say; the logits against 64 bits."""
    h, w, x = _handle(L, d, B, L + B, chunks, sched_labels=sched, w_scale=2.0)
    if B > 5 and embed is torch.bfloat16:
        x[3, 8] = 2.0 ** 14                                    # a wide row
    if embed is E4M3:
        x = (x.float() * d ** 0.5).to(E4M3)
    z = _logits(h, x, n_out)
    want = 2.0 * (x.double() @ w[:n_out].double().t())
    size = 2.0 * (x.double().abs() @ w[:n_out].double().abs().t())
    assert bool(((z.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * size).all())
    before = h.launch_count
    v, i = h.forward_topk(x, 20, n_out)
    assert (h.launch_count - before) % 2 == 1                  # a window is two launches, the split one
    h.check()
    sv, si = torch.sort(z.float(), dim=1, descending=True, stable=True)
    assert torch.equal(v, sv[:, :20]) and torch.equal(i.long(), si[:, :20])
    h.close()


# simulated FP8 on either side of the lines between one kernel (3 launches, or 6 where the pairs are sorted by launches of their own) and three
T = 74 * 128


@pytest.mark.parametrize("L,d,B,sr,loss,one", [
    (4 * T, 64, 128, True, True, True), (4 * T + 1, 64, 33, True, True, False), (12 * T, 64, 32, True, True, True),
    (12 * T, 64, 128, True, False, True), (12 * T + 1, 64, 8, True, False, False), (13 * T, 64, 32, False, True, True),
    (13 * T, 64, 33, False, True, False), (32 * T, 64, 64, False, False, True), (32 * T + 1, 64, 64, False, False, False),
    (33 * T, 64, 65, False, False, True), (12 * T, 128, 128, True, True, True), (13 * T, 128, 33, True, True, False),
    (32 * T, 128, 32, True, True, True), (32 * T + 1, 128, 32, True, True, False), (32 * T, 128, 64, True, False, True),
    (32 * T + 1, 128, 64, True, False, False), (33 * T, 128, 96, True, False, True), (33 * T, 128, 97, True, False, False),
    (32 * T, 192, 64, False, True, True), (32 * T + 1, 256, 64, True, True, False), (32 * T + 1, 256, 64, True, False, True),
    (32 * T + 1, 256, 65, True, True, True), (32 * T + 1, 320, 64, True, True, True)])
def test_one_kernel_or_three(L, d, B, sr, loss, one):
    from elmo_b200.handle import XmcHandle
    h = XmcHandle(torch.device("cuda", 0), d, B, "simfp8")
    h.bind([torch.full((L, d), 2.0 ** -6, device="cuda").to(E4M3)])
    x = torch.zeros(B, d, dtype=torch.bfloat16, device="cuda")
    gx = torch.empty(B, d, dtype=torch.float32, device="cuda")
    lo = torch.zeros(1, dtype=torch.float64, device="cuda")
    h.profile(True)
    h.step(x, None, 0.0, seed=1, step=2, stochastic=sr, compute_loss=loss, grad_f32=gx, loss_out=lo)
    kinds = h.profile(False, read=True)
    h.check()
    h.close()
    assert ("forward" not in kinds) == one
    assert rel_inf(gx, torch.full_like(gx, L * 2.0 ** -7)) < 1e-5
    if loss:
        assert abs(float(lo) / (L * B) - 0.693147) < 1e-5          # log 2 each
