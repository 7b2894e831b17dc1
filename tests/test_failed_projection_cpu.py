"""A projection that failed on the device (device error word, bit 2) ends a reconstruction with an error, on the host with
the oracle answering the library calls."""
import numpy as np
import pytest
import torch

import mbirjax_b200 as mb
from mbirjax_b200 import batched as B
from cases import make_case
from fake_library import oracle_library  # noqa: F401  (fixture)


def _recon():
    model, geom = make_case('parallel', views=8, rows=2, channels=12)
    model.set_params(sharpness=0.0, granularity=[2], partition_sequence=[0], verbose=0)
    np.random.seed(1)
    sino = np.random.default_rng(1).random(geom.sinogram_shape).astype(np.float32)
    return model.recon(sino, max_iterations=1, stop_threshold_change_pct=0, logfile_path=None, print_logs=False)


def test_recon_raises_when_a_projection_failed(oracle_library, monkeypatch):
    cleared = []
    monkeypatch.setattr(oracle_library, 'get_device_error', lambda: cleared.append(1) or 4)
    monkeypatch.setattr(oracle_library, 'peek_device_error', lambda device: 4)
    with pytest.raises(mb.MbxError, match='projection failed'):
        _recon()
    assert cleared == [1]
    with pytest.raises(mb.MbxError, match='projection failed'):
        B._results([], [torch.zeros(2, 3)], [], [], [], [], np.zeros((1, 1, 4)), np.zeros((1, 1, 4)), 1, 1, clone=True)


def test_recon_keeps_a_callers_bad_index_apart(oracle_library, monkeypatch):
    monkeypatch.setattr(oracle_library, 'peek_device_error', lambda device: 3)
    _recon()
