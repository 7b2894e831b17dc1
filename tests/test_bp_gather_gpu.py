"""Parallel-beam back projection on both sides of the lines that choose between gathering and windows (bp_gather.cuh:
slices, and how many of the grid's pixels the list holds), at the edges of the gather's slice tiles, and the windows with
two and three taps, against the oracle.  Bar: 1e-5 relative L2, the bar of every projector test (float32 sums of the same
terms in either order)."""
import numpy as np
import pytest
import torch

import oracle as O
from mbirjax_b200 import _capi
from cases import make_case, rel_l2

pytestmark = pytest.mark.gpu


def _check(model, geom, pix, coeff_power=1, weighted=False, views=None):
    rng = np.random.default_rng(6)
    sino = rng.standard_normal(geom.sinogram_shape).astype(np.float32)
    w = rng.uniform(0.2, 1.0, geom.sinogram_shape).astype(np.float32) if weighted else None
    ref = O.sparse_back_project(geom, sino if w is None else w * sino, pix, view_indices=views, coeff_power=coeff_power)
    dev = torch.device('cuda')
    args = dict(view_indices=None if views is None else torch.as_tensor(views, device=dev), coeff_power=coeff_power,
                weights=None if w is None else torch.as_tensor(w, device=dev))
    s, p = torch.as_tensor(sino, device=dev), torch.as_tensor(pix, device=dev)
    got = _capi.back_project(model._geometry(), s, p, **args)
    assert torch.equal(got, _capi.back_project(model._geometry(), s, p, **args))
    plain = _capi.back_project_noalloc(model._geometry(), s, p, **args)
    assert _capi.get_device_error() == 0
    assert rel_l2(got.cpu().numpy(), ref) <= 1e-5
    assert rel_l2(plain.cpu().numpy(), ref) <= 1e-5


@pytest.mark.parametrize('share', [1, 6, 8])
@pytest.mark.parametrize('rows', [1, 2, 15, 16, 17, 26, 27, 28, 33, 130])
def test_slices_and_density(cuda, rows, share):
    model, geom = make_case('parallel', views=19, rows=rows, channels=38)
    n = geom.recon_shape[0] * geom.recon_shape[1]
    pix = np.sort(np.random.default_rng(rows).permutation(n)[:-(-n // share)]).astype(np.int32)
    _check(model, geom, pix)


@pytest.mark.parametrize('rows', [11, 29])
@pytest.mark.parametrize('delta_voxel', [0.6, 1.0, 1.7])
def test_taps_weights_powers_and_views(cuda, rows, delta_voxel):
    model, geom = make_case('parallel', views=21, rows=rows, channels=50, delta_voxel=delta_voxel)
    n = geom.recon_shape[0] * geom.recon_shape[1]
    _check(model, geom, np.arange(n, dtype=np.int32))
    _check(model, geom, np.arange(n, dtype=np.int32), coeff_power=2, weighted=True)
    _check(model, geom, np.arange(0, n, 9, dtype=np.int32), weighted=True,
           views=np.array([20, 3, 3, 0, 11, 7, 8, 9, 10, 1, 2, 19, 18, 17, 4, 5, 6], dtype=np.int32))


def test_more_views_than_a_table(cuda):
    model, geom = make_case('parallel', views=1030, rows=3, channels=24)
    n = geom.recon_shape[0] * geom.recon_shape[1]
    _check(model, geom, np.tile(np.arange(n, dtype=np.int32), 140))  # enough pixels for one split of all views
