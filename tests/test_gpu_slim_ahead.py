"""The one-kernel step with U two boxes ahead (e4m3, stochastic rounding, three boxes of 128 features and more): CTAs of a
cluster with unequal numbers of boxes, one among them, and with one, two and several tiles, against the CPU oracle."""
import pytest
import torch

from tests._util import rel_inf
from tests.test_gpu_step import _check_weights, _inputs, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [3, 40, 64])
@pytest.mark.parametrize("d", [320, 384, 512, 576, 768])
@pytest.mark.parametrize("tiles", [1, 74, 75, 230])
def test_two_boxes_ahead(tiles, d, B):
    if tiles == 230 and (B, d) not in ((3, 320), (40, 576), (64, 320)):
        pytest.skip("the CPU oracle takes the largest size at three shapes only")
    from oracle import xmc_oracle as O
    L = 128 * tiles - 7 * (tiles > 1)
    w, x, lab = _inputs(L, d, B, 3 * B, seed=tiles + d)
    (want,), want_gx, want_loss = O.fp8_chunked_step([w], x, lab, 0.5, rounding="sr", seed=5, step=1, compute_loss=True)
    (got,), gx, _, loss = _run_gpu("fp8", [w], x, lab, 0.5, stochastic=True, step=1, loss=True)
    _check_weights([got], [want])
    assert rel_inf(gx, want_gx) < 1e-2
    assert abs(loss - want_loss) < 1e-3 * abs(want_loss)
