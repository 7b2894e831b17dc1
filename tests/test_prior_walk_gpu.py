"""The prior's loss and gradient at the edges of its blocks (qggmrf.cu): single rows, columns and slices, cylinders longer
than a block's elements, rows that leave the last walk short, and p other than 2.  Bar: 1e-5 relative, as every test of
this function (float32 powers)."""
import numpy as np
import pytest

import mbirjax_b200 as mb
import oracle as O
from cases import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('p', [2.0, 1.7])
@pytest.mark.parametrize('shape', [(1, 1, 1), (1, 6, 4), (40, 1, 1), (9, 1, 200), (17, 3, 700), (25, 30, 33), (64, 16, 8)])
def test_loss_grad_shapes(cuda, shape, p):
    x = np.random.default_rng(2).random(shape).astype(np.float32)
    params = (mb.get_b_from_nbr_wts([0.5, 1, 1]), 0.25, p, 1.2, 0.8)
    loss, grad = mb.qggmrf_loss_and_grad(x, params)
    ref = O.qggmrf_loss(x, params)
    assert float(loss) == pytest.approx(ref, rel=1e-5, abs=1e-12)
    want = O.qggmrf_loss_grad(x, params)
    if np.linalg.norm(want) == 0:
        assert not grad.cpu().numpy().any()
    else:
        assert rel_l2(grad.cpu().numpy(), want) <= 1e-5
