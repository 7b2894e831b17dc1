"""The ramp filter at the edges of its tiles (direct_filter.cuh): rows shorter than a lane's outputs, on either side of
one, two and four 128-channel tiles and of one pass, row counts that leave a block partly empty.  Taps, samples and sums
are float64 and each output is rounded once, so the bar is a rounding: 2e-7 relative L2 of the float64 convolution."""
import numpy as np
import pytest
import torch

from cases import make_case, rel_l2

pytestmark = pytest.mark.gpu


def _reference(sino, model, cone):
    V, R, C = sino.shape
    d = np.arange(C)[:, None] - np.arange(C)[None, :]
    taps = np.where(d == 0, 0.25, np.where(d % 2 != 0, -1.0 / (np.pi * np.where(d == 0, 1, d)) ** 2, 0.0))
    x = sino.astype(np.float64)
    if cone:
        D = float(model.get_params('source_detector_dist'))
        u, w = np.arange(C) - (C - 1) / 2, np.arange(R) - (R - 1) / 2
        x = x * (D / np.sqrt(D * D + u[None, :] ** 2 + w[:, None] ** 2))
    return (np.pi / V) * (x @ taps.T)


@pytest.mark.parametrize('channels', [3, 15, 64, 127, 128, 129, 200, 256, 257, 384, 513, 700, 1030])
@pytest.mark.parametrize('kind', ['parallel', 'cone'])
def test_filter_tiles(cuda, kind, channels):
    model, _ = make_case(kind, views=5, rows=7, channels=channels)
    sino = np.random.default_rng(channels).standard_normal((5, 7, channels)).astype(np.float32)
    out = model.direct_filter(torch.as_tensor(sino, device=cuda)).cpu().numpy()
    assert rel_l2(out, _reference(sino, model, kind == 'cone')) <= 2e-7
