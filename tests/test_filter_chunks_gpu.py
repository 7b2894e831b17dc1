"""The ramp filter on both sides of the line that takes whole chunks of samples (direct_filter.cuh, filter_whole), and with
enough rows for blocks of the default height, where shorter calls take lower ones.  Taps, samples and sums are float64 and
each output is rounded once, so the bar is a rounding: 2e-7 relative L2 of the float64 convolution."""
import numpy as np
import pytest
import torch

from cases import make_case, rel_l2
from test_filter_tiles_gpu import _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('views,rows,channels', [(5, 7, 479), (5, 7, 486), (5, 7, 487), (5, 7, 511), (5, 7, 512),
                                                 (3, 5, 1000), (150, 127, 120), (150, 127, 122), (150, 127, 128),
                                                 (150, 65, 230), (150, 65, 256)])
@pytest.mark.parametrize('kind', ['parallel', 'cone'])
def test_whole_and_short_chunks(cuda, kind, views, rows, channels):
    model, _ = make_case(kind, views=views, rows=rows, channels=channels)
    sino = np.random.default_rng(channels).standard_normal((views, rows, channels)).astype(np.float32)
    out = model.direct_filter(torch.as_tensor(sino, device=cuda)).cpu().numpy()
    assert rel_l2(out, _reference(sino, model, kind == 'cone')) <= 2e-7
