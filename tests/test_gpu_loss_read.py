"""The loss a layer returns is the one of the step it belongs to, call after call, on the default and on a side stream.  (It
counts the rows that pad the layer, as it always did.)"""
import pytest
import torch

from tests.test_gpu_kahan import _cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [False, True])
def test_every_call_returns_its_own_loss(side):
    from elmo_b200.xmc_classifiers import Fp8XMCBCEChunkedLayer
    L, d, B = 500, 64, 20
    layer = Fp8XMCBCEChunkedLayer(_cfg(L, d, B, 1, False, 0.1, "rn"))
    x = torch.randn(B, d, device="cuda").to(torch.bfloat16)
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for n in (0, 40, 7, 0):
            lab = torch.stack([torch.arange(n) % B, torch.arange(n) * 3 % L], 1).to(torch.int32).cuda()
            out = torch.empty(B, layer.num_labels, dtype=torch.bfloat16, device="cuda")
            layer._bind()
            layer._handle.forward_logits(x, out, layer.num_labels)
            z = out.double()
            want = torch.nn.functional.softplus(z).sum() - (z[lab[:, 0].long(), lab[:, 1].long()].sum() if n else 0.0)
            got = layer.xfc_forward_backward(x, lab, [0.0], skip_loss=False)
            assert abs(got - float(want)) < 3e-5 * abs(float(want))          # sums of fp32 terms off by 2^-22 each


def test_where_a_loss_may_go():
    """Device memory and pinned host memory; nothing else, whether or not assertions are compiled in."""
    import copy

    from elmo_b200.handle import HostLoss, XmcHandle
    L, d, B = 300, 64, 10
    h = XmcHandle(torch.device("cuda", 0), d, B, "fp8")
    h.bind([torch.zeros(L, d, dtype=torch.float8_e4m3fn, device="cuda")])
    x = torch.zeros(B, d, dtype=torch.bfloat16, device="cuda")
    for refused in (None, torch.zeros(1, dtype=torch.float64), torch.zeros(1, device="cuda")):
        with pytest.raises(ValueError):
            h.step(x, None, 0.0, compute_loss=True, loss_out=refused)
    host = copy.deepcopy(HostLoss())
    assert host.cell.is_pinned()
    places = [torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, pin_memory=True), host]
    for place in places:
        h.step(x, None, 0.0, compute_loss=True, loss_out=place)
    h.check()
    want = L * B * 0.6931471805599453
    for got in (float(places[0]), float(places[1]), h.read_loss(host)):
        assert abs(got - want) < 1e-5 * want
    h.close()
