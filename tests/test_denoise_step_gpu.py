"""The denoiser's subset update at the edges of its grid (denoise.cu): one voxel, one block and its neighbours, partials
that leave the lanes of a warp uneven, and more voxels than the grid has threads.  With a zero error image the update's
delta is the prior's alone, and the new error image is -alpha delta exactly, so all four statistics follow from it.
Bars: l1 is a float64 sum of n values that are known exactly, at most n 2^-53 off; the step's numerator and
denominator sum float32 products of one sign, each a few roundings off (16 x 2^-24); alpha is their float32 quotient."""
import numpy as np
import pytest
import torch

import mbirjax_b200 as mb
from mbirjax_b200 import _capi

pytestmark = pytest.mark.gpu
U32, U64 = 2.0 ** -24, 2.0 ** -53


@pytest.mark.parametrize('shape, n', [((1, 2, 1), 1), ((16, 16, 1), 255), ((16, 16, 1), 256), ((20, 20, 1), 257),
                                      ((40, 40, 33), 1000), ((64, 60, 100), 3000)])
def test_denoise_step_statistics(cuda, shape, n):
    rng = np.random.default_rng(4)
    nr, nc, ns = shape
    x = torch.as_tensor(rng.random((nr * nc, ns)).astype(np.float32), device=cuda)
    pix = torch.as_tensor(rng.permutation(nr * nc)[:n].astype(np.int32), device=cuda)
    qp = _capi.qggmrf_params(mb.get_b_from_nbr_wts([1, 1, 1]), 0.25, 2.0, 1.2, 1.0)
    grad, hess = _capi.qggmrf_grad_hess(x, shape, pix, qp)
    d = -(grad / (1.0 + hess))
    fm, eps = 4.0, 2.0 ** -23
    num = -float((grad.double() * d.double()).sum())
    den = fm * float((d.double() ** 2).sum()) + float((hess.double() * d.double() ** 2).sum()) / 1.1 + eps
    alpha = min(max(num / den, eps), 1.5)
    for _ in range(2):  # the second update finds the workspace as the first left it
        image, err = x.clone(), torch.zeros_like(x)
        stats = torch.full((4,), -1.0, dtype=torch.float64, device=cuda)
        ws = _capi._workspace(_capi.load_library().mbx_qggmrf_denoise_step_workspace_bytes(n, ns), cuda)
        _capi.qggmrf_denoise_step(image, err, shape, pix, fm, qp, stats, ws)
        _capi.qggmrf_denoise_step(image.copy_(x), err.zero_(), shape, pix, fm, qp, stats, ws)
        got = stats.tolist()
        assert got[2] == pytest.approx(num, rel=16 * U32) and got[3] == pytest.approx(den, rel=16 * U32)
        assert got[0] == pytest.approx(alpha, rel=64 * U32)
        assert got[1] == pytest.approx(float(err.abs().double().sum()), rel=max(n * ns, 1) * U64)
        moved = torch.zeros_like(x)
        moved[pix.long()] = err[pix.long()]
        assert torch.equal(moved, err) and torch.equal(image, x - err)
