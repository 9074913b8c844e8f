"""How many label rows a launch of the three kernels takes where a weight chunk has more than 65 536 and the batch is large: G of at
most 65 536 rows and a quarter, so that sums of grad_X over e4m3 weights, which last as long as a launch, and the workspace do not
grow with the chunk."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp8", "simfp8"])
def test_launch_of_a_large_batch(mode):
    from elmo_b200.handle import XmcHandle
    dev = torch.device("cuda", 0)
    L, d, B, rows = 300000, 64, 1024, 65536
    gen = torch.Generator(device=dev).manual_seed(3)
    ws = [(torch.randn(L // 2, d, generator=gen, device=dev) * 0.25).to(torch.float8_e4m3fn) for _ in range(2)]
    x = (torch.randn(B, d, generator=gen, device=dev) / d ** 0.5).to(torch.bfloat16)
    grads = []
    # what the two chunks of 586 tiles of 256 rows need, in equal launches, each in whole rounds of 74 CTA pairs
    for sched in (0, 296 * 256):
        h = XmcHandle(dev, d, B, mode, sched_labels=sched)
        h.bind(ws)
        g = torch.empty(B, d, dtype=torch.float32, device=dev)
        before = h.launch_count
        h.step(x, None, 0.0, seed=1, step=2, stochastic=False, grad_f32=g)
        launches, held = h.launch_count - before, h.workspace_bytes
        h.check()
        h.close()
        assert launches == 2 + 3 * 4                         # preparation and reduction, and three kernels a launch
        assert held < rows * 5 // 4 * B * 2 + (64 << 20)     # G, and less than 64 MB of everything else
        grads.append(g)
    assert torch.equal(grads[0], grads[1])
