"""Split embeddings of simulated FP8 hold what bf16 does: every significand down to 2^-13 of a row's largest number in two parts, down to
2^-23 in the three parts of a wide row, whichever other rows are wide, and whichever were in the call before.  One-hot weights
make every logit one element of its row, so nothing is tolerated there."""
import pytest
import torch

from tests._util import rel_inf

pytestmark = pytest.mark.gpu
E4M3 = torch.float8_e4m3fn


def _one_hot(L, d, B):
    from elmo_b200.handle import XmcHandle
    w = torch.zeros(L, d, device="cuda")
    w[torch.arange(L), torch.arange(L) % d] = 1.0
    h = XmcHandle(torch.device("cuda", 0), d, B, "simfp8")
    h.bind([w.to(E4M3)])
    return h


def _elements(h, x, L):
    """The logits of one-hot labels, by feature.  A call that splits its embeddings is two launches, one that converts the weights one."""
    out = torch.empty(x.shape[0], (L + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
    before = h.launch_count
    h.forward_logits(x, out, L)
    assert h.launch_count - before == 2
    h.check()
    d = x.shape[1]
    assert torch.equal(out[:, L - d:L].roll((L - d) % d, 1), out[:, :d])
    return out[:, :d]


def _rows(B, d, down_to, seed):
    """Rows of largest magnitude 1 or 255/128, the others of all 128 significands and of all binades down to 2^-down_to, both signs."""
    g = torch.Generator().manual_seed(seed)
    n = torch.randperm(B * d, generator=g).view(B, d)
    x = (1 + (n % 128) / 128.0) * torch.exp2(-(1.0 + n // 128 % down_to)) * (1 - 2 * (n // 7 % 2))
    x[:, 0] = torch.where(torch.arange(B) % 2 == 0, 1.0, 255.0 / 128)
    x = torch.where(x.abs() < x[:, :1] * 2.0 ** -down_to, torch.zeros(()), x)
    return (x * torch.exp2(torch.tensor([0.0, 25, -50, 100, -118])[torch.arange(B) % 5])[:, None]).to(torch.bfloat16).cuda()


# one CTA; CTA pairs, one batch tile and two; rows of more than 1024 features are read twice
@pytest.mark.parametrize("d,B", [(768, 1), (768, 40), (768, 140), (768, 300), (1088, 100), (512, 129)])
def test_elements_are_exact(d, B):
    L = 95000
    h = _one_hot(L, d, B)
    x = _rows(B, d, 13, B)
    assert torch.equal(_elements(h, x, L), x)
    x = _rows(B, d, 23, B)
    assert torch.equal(_elements(h, x, L), x)
    h.close()


def test_wide_rows_come_and_go():
    L, d, B = 60000, 768, 300
    h = _one_hot(L, d, B)
    narrow, wide = _rows(B, d, 13, 1), _rows(B, d, 23, 2)
    for rows in ([], [5], [290], [5, 290], [290], [299, 0], [], list(range(B)), [255, 256]):
        for n in (B, 270, 100):                      # (a smaller call leaves what the larger one had behind its rows)
            x = narrow.clone()
            x[rows] = wide[rows]
            assert torch.equal(_elements(h, x[:n], L), x[:n])
    # e4m3 embeddings between two calls with wide rows
    x = wide.clone()
    x[::2] = narrow[::2]
    assert torch.equal(_elements(h, x, L), x)
    x8 = narrow.float().clamp(-400, 400).to(E4M3)
    assert torch.equal(_elements(h, x8, L), x8.to(torch.bfloat16))
    x[1::2], x[::2] = narrow[1::2], wide[::2]
    assert torch.equal(_elements(h, x, L), x)
    h.close()


def test_below_the_last_exact_binade():
    """Within 2^-31 of the largest below 2^-23 of it; where hardly anything lacks, within 2^-24 of all magnitudes, summed up."""
    L, d, B = 60000, 768, 40
    h = _one_hot(L, d, B)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(B, d, generator=g, device="cuda").to(torch.bfloat16)
    x[B // 2:] *= torch.exp2(-40 * torch.rand(B // 2, d, generator=g, device="cuda")).to(torch.bfloat16)
    x[B // 2:, 3] = 4.0
    z = _elements(h, x, L)
    want, size = x.double(), x.double().abs()
    room = torch.where(torch.arange(B, device="cuda")[:, None] < B // 2, size.sum(1, keepdim=True) * 2.0 ** -24, size.amax(1, keepdim=True) * 2.0 ** -31)
    assert bool(((z.double() - want).abs() <= room + 2.0 ** -9 * want.abs()).all())
    assert torch.equal(z[size >= size.amax(1, keepdim=True) * 2.0 ** -13], x[size >= size.amax(1, keepdim=True) * 2.0 ** -13])
    h.close()


# one kernel on either side of batch 64, three kernels with one batch tile and with two, the last feature box in part
@pytest.mark.parametrize("loss", [False, True])
@pytest.mark.parametrize("d,B,launches", [(768, 40, 3), (320, 128, 3), (768, 140, 5), (320, 300, 5)])
def test_steps_with_an_outlier_that_no_label_uses(d, B, launches, loss):
    """One feature at 2^15 in every third row, its weights zero: the logits are what the others, 2^-20 of it, make of them."""
    from elmo_b200.handle import XmcHandle
    L = 20000
    g = torch.Generator(device="cuda").manual_seed(d + B)
    w = torch.randn(L, d, generator=g, device="cuda") * 0.25
    w[:, 7] = 0
    w = w.to(E4M3)
    x = torch.randn(B, d, generator=g, device="cuda") / d ** 0.5
    x[::3, 7] = 32768.0
    x = x.to(torch.bfloat16)
    z = (x.double() @ w.double().t()).to(torch.bfloat16)
    want = torch.sigmoid(z.double()).to(torch.bfloat16).double() @ w.double()
    h = XmcHandle(torch.device("cuda", 0), d, B, "simfp8")
    h.bind([w])
    gx = torch.empty(B, d, dtype=torch.float32, device="cuda")
    lo = torch.zeros(1, dtype=torch.float64, device="cuda")
    before = h.launch_count
    h.step(x, None, 0.0, seed=1, step=2, stochastic=True, compute_loss=loss, grad_f32=gx, loss_out=lo)
    assert h.launch_count - before == launches
    h.check()
    h.close()
    assert rel_inf(gx, want) < 1e-2
    if loss:
        assert abs(float(lo) - float(torch.nn.functional.softplus(z.double()).sum())) < 1e-4 * float(lo)
