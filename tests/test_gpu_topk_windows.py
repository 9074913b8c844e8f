"""The fused top-k over windows of label columns: selection against torch on the layer's own logits (bit for
bit, so nothing is tolerated), at the edges of groups of 32, tiles, chunks and windows, with ties, few labels
and non-finite logits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
NEG = float("-inf")


def _check(h, x, k, n_out, total):
    z = torch.empty(x.shape[0], (total + 7) // 8 * 8, dtype=torch.bfloat16, device=x.device)
    h.forward_logits(x, z, n_out)
    v, i = h.forward_topk(x, k, n_out)
    h.check()
    zf = z[:, :n_out].float()
    zf = torch.where(zf.isnan(), torch.full_like(zf, NEG), zf)
    sv, si = torch.sort(zf, dim=1, descending=True, stable=True)      # equal values keep label order
    kk = min(k, n_out)
    assert torch.equal(v[:, :kk], sv[:, :kk])
    want = torch.where(sv[:, :kk] == NEG, torch.full_like(si[:, :kk], -1 - h.label_offset), si[:, :kk])
    assert torch.equal(i[:, :kk].long(), want + h.label_offset)
    assert bool((v[:, kk:] == NEG).all()) and bool((i[:, kk:] == -1).all())


def _handle(rows, d, max_batch, mode, sched=0, off=0, scale=0.5, seed=0, equal=False):
    from elmo_b200.handle import XmcHandle
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(seed)
    dt = torch.bfloat16 if mode == "bf16" else torch.float8_e4m3fn
    ws = [torch.full((r, d), 0.25, device=dev).to(dt) if equal else (torch.randn(r, d, generator=gen, device=dev) * scale).to(dt)
          for r in rows]
    h = XmcHandle(dev, d, max_batch, mode, sched_labels=sched, label_offset=off)
    h.bind(ws)
    return h, ws, gen, dev


@pytest.mark.parametrize("mode", ["fp8", "simfp8", "bf16"])
@pytest.mark.parametrize("rows,n_out,sched,max_batch,batch,k", [
    ([20], 17, 0, 4, 1, 128),                          # fewer labels than wanted
    ([33], 33, 0, 1, 1, 1),
    ([1000, 1000, 250], 2230, 256, 64, 64, 20),        # several windows per chunk
    ([528, 528, 528, 16], 1600, 0, 256, 129, 100),     # windows of several padded chunks; 129 rows: CTA pairs
    ([70000], 70000, 0, 300, 300, 7),
    ([70000, 69001], 139001, 0, 300, 3, 128),          # a small batch: both chunks in one window
    ([65536], 65536, 0, 4, 3, 128),                    # as many threads with maxima as the bound by thread needs
    ([65280], 65280, 0, 4, 3, 128),                    # one fewer
])
def test_topk_windows(mode, rows, n_out, sched, max_batch, batch, k):
    h, _, gen, dev = _handle(rows, 64, max_batch, mode, sched, off=1000, seed=k)
    x = torch.randn(batch, 64, generator=gen, device=dev).to(torch.bfloat16)
    _check(h, x, k, n_out, sum(rows))


@pytest.mark.parametrize("batch", [2, 200])
def test_topk_few_distinct_values(batch):
    """Thousands of equal logits: more candidates than fit into shared memory, decided by the label."""
    h, ws, gen, dev = _handle([40000, 40000], 64, 256, "fp8", equal=True)
    ws[1][35000:] = (ws[1][35000:].float() * 2).to(ws[1].dtype)       # the last window holds the best ones
    x = torch.rand(batch, 64, generator=gen, device=dev).to(torch.bfloat16)
    for k in (1, 128):
        _check(h, x, k, 80000, 80000)


def test_topk_ignores_nan_and_minus_infinity():
    h, ws, gen, dev = _handle([900], 64, 64, "bf16")
    ws[0][5:700] = float("nan")
    ws[0][700:800] = NEG
    x = torch.rand(40, 64, generator=gen, device=dev).to(torch.bfloat16) + 0.5
    _check(h, x, 120, 900, 900)
