"""Back projections large enough to read windows of a transposed copy (bp_fast.cuh, bp_windows), and calls on the other side
of its lines, which read their taps from the sinogram: both against the oracle at sampled entries of the pixel list, and
against the entry point that has no room for a copy over the whole output.  The launches and the workspace of a call tell
its route.  Bar: 1e-5 relative L2, the bar of every projector test (float32 sums of the same terms in either order)."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from mbirjax_b200 import _capi
from mbirjax_b200.vcd_utils import gen_pixel_partition, morton_sorted_partition
from cases import make_case, rel_l2

pytestmark = pytest.mark.gpu


def _pixels(shape, order, seed=3):
    rng = np.random.default_rng(seed)
    if order == 'raster':
        return np.arange(shape[0] * shape[1], dtype=np.int32)
    part = gen_pixel_partition(shape, 2, rng=np.random.RandomState(seed))
    if order == 'subset':
        return morton_sorted_partition(part, shape[1])[1]
    if order == 'sorted-subset':
        return part[0]
    return rng.integers(0, shape[0] * shape[1], part.shape[1]).astype(np.int32)  # scattered, with duplicates, corners too


def _check(model, geom, pix, windows, coeff_power=1, weighted=False, views=None):
    g, dev = model._geometry(), torch.device('cuda')
    assert g.psf_radius == 1
    rng = np.random.default_rng(5)
    sino = rng.standard_normal(geom.sinogram_shape).astype(np.float32)
    w = rng.uniform(0.2, 1.0, geom.sinogram_shape).astype(np.float32) if weighted else None
    nv = g.num_views if views is None else len(views)
    args = dict(view_indices=None if views is None else torch.as_tensor(views.astype(np.int32), device=dev),
                coeff_power=coeff_power, weights=None if w is None else torch.as_tensor(w, device=dev))
    s, p = torch.as_tensor(sino, device=dev), torch.as_tensor(pix, device=dev)
    _capi.get_device_error()
    lib = _capi.load_library()
    before = lib.mbx_launch_count()
    got = _capi.back_project(g, s, p, **args).cpu().numpy()
    launches = lib.mbx_launch_count() - before
    # the copy, the projection, the sum of the view splits where the workspace holds more than the copy
    need = lib.mbx_back_project_workspace_bytes(ctypes.byref(g), len(pix), nv)
    copy = 4 * min(nv, g.num_views) * (g.num_det_channels + 4) * (g.num_det_rows + 3 & ~3) + 255 & ~255
    assert launches == (2 + (need > copy) if windows else 1 + (need > 0))
    assert not windows or need >= copy
    direct = _capi.back_project_noalloc(g, s, p, **args).cpu().numpy()
    assert _capi.get_device_error() == 0
    assert rel_l2(direct, got) <= 1e-5
    some = rng.permutation(len(pix))[:96]
    ref = O.sparse_back_project(geom, sino if w is None else w * sino, pix[some], view_indices=views,
                                coeff_power=coeff_power)
    assert rel_l2(got[some], ref) <= 1e-5
    assert rel_l2(direct[some], ref) <= 1e-5


@pytest.mark.parametrize('order', ['raster', 'subset', 'sorted-subset', 'scattered'])
@pytest.mark.parametrize('kind', ['parallel', 'cone'])
def test_windows_and_orders(cuda, kind, order):
    if kind == 'parallel':
        model, geom = make_case('parallel', views=260, rows=37, channels=150)
    else:
        model, geom = make_case('cone', views=256, rows=66, channels=160)
    _check(model, geom, _pixels(geom.recon_shape, order), True)


@pytest.mark.parametrize('kind', ['parallel', 'cone', 'translation'])
def test_windows_with_weights_powers_and_views(cuda, kind):
    if kind == 'parallel':
        model, geom = make_case('parallel', views=200, rows=34, channels=140, det_channel_offset=2.3)
    elif kind == 'cone':
        model, geom = make_case('cone', views=256, rows=66, channels=160, det_channel_offset=2.3, det_row_offset=-1.6)
    else:
        model, geom = make_case('translation', views=100, rows=128, channels=128, sdd_factor=0.5)
    n = geom.recon_shape[0] * geom.recon_shape[1]
    pix = np.arange(n, dtype=np.int32)
    _check(model, geom, pix, True, coeff_power=2, weighted=True)
    v = geom.sinogram_shape[0]
    some = np.random.default_rng(1).permutation(v)[:v - 3]
    some[5] = some[6]
    _check(model, geom, pix, True, views=some)
    _check(model, geom, pix, True, weighted=True, views=np.arange(v + 40) % v)  # more than the geometry has: some repeat


@pytest.mark.parametrize('delta_voxel', [0.6, 1.0, 1.7])
def test_windows_of_two_and_three_taps(cuda, delta_voxel):
    model, geom = make_case('parallel', views=300, rows=33, channels=130, delta_voxel=delta_voxel)
    n = geom.recon_shape[0] * geom.recon_shape[1]
    views = np.arange(round(60e6 / (n * 33))) % 300  # more views for a smaller grid: past the line
    _check(model, geom, np.arange(n, dtype=np.int32), True, views=views)
    _check(model, geom, _pixels(geom.recon_shape, 'scattered')[:n // 4], False, coeff_power=2, weighted=True)


@pytest.mark.parametrize('rows,channels', [(27, 152), (28, 152), (32, 152), (33, 152), (64, 140), (65, 152)])
def test_windows_at_the_edges_of_slice_tiles(cuda, rows, channels):
    model, geom = make_case('parallel', views=150, rows=rows, channels=channels)
    _check(model, geom, np.arange(channels * channels, dtype=np.int32), True)


@pytest.mark.parametrize('kind', ['cone', 'translation'])
def test_taps_from_the_sinogram(cuda, kind):
    """Calls below the lines: tiles at their edges, weights, powers, view lists, pixels off the detector, no sinogram."""
    model, geom = make_case(kind, views=24, rows=35, channels=66, det_channel_offset=-3.4)
    _check(model, geom, _pixels(geom.recon_shape, 'raster'), False)
    _check(model, geom, _pixels(geom.recon_shape, 'scattered'), False, coeff_power=2, weighted=True)
    _check(model, geom, _pixels(geom.recon_shape, 'subset'), False, views=np.array([3, 3, 20, 7, 0, 23]))
    g, n = model._geometry(), geom.recon_shape[0] * geom.recon_shape[1]
    pix = np.arange(n, dtype=np.int32)
    for power in (1, 2):
        ones = _capi.back_project(g, None, torch.as_tensor(pix, device=cuda), coeff_power=power).cpu().numpy()
        ref = O.sparse_back_project(geom, np.ones(geom.sinogram_shape, np.float32), pix, coeff_power=power)
        assert rel_l2(ones, ref) <= 1e-5


def test_bad_views_are_flagged_whatever_the_first_pixels_are(cuda):
    """Bad indices are skipped and flagged: a bad view too when none of a warp's pixels is in the grid."""
    model, geom = make_case('parallel', views=260, rows=37, channels=150)
    g, n = model._geometry(), 150 * 150
    pix = torch.arange(n, dtype=torch.int32, device=cuda)
    pix[:64] = -1
    views = torch.arange(260, dtype=torch.int32, device=cuda)
    sino = torch.rand(geom.sinogram_shape, device=cuda)
    _capi.get_device_error()
    _capi.back_project(g, sino, pix, view_indices=views)
    assert _capi.get_device_error() == 1
    views[130] = 260
    _capi.back_project(g, sino, pix, view_indices=views)
    assert _capi.get_device_error() == 3


@pytest.mark.parametrize('kind', ['parallel', 'cone'])
def test_without_room_for_a_copy(cuda, kind, monkeypatch):
    """A workspace without room for the copy, down to the least: the same sums; below that, an error.  The Python call
    falls back by itself when the full workspace cannot be allocated."""
    model, geom = make_case(kind, views=256, rows=66, channels=160)
    g, lib = model._geometry(), _capi.load_library()
    n = 160 * 160
    pix = torch.arange(n, dtype=torch.int32, device=cuda)
    sino = torch.randn(geom.sinogram_shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(1))
    ref = _capi.back_project(g, sino, pix)
    full = lib.mbx_back_project_workspace_bytes(ctypes.byref(g), n, g.num_views)
    least = lib.mbx_back_project_least_workspace_bytes(ctypes.byref(g), n, g.num_views)
    assert full >= 4 * 256 * 68 * 164 and least < full
    ws = torch.empty(full, dtype=torch.uint8, device=cuda)
    for nbytes, rc in ((full - 1, 0), (least, 0), (least - 1, _capi.MBX_ERR_WORKSPACE)):
        if nbytes < 0:
            continue
        out = torch.full_like(ref, 7.0)
        assert lib.mbx_sparse_back_project(ctypes.byref(g), _capi._ptr(sino), None, _capi._ptr(pix), n, None, g.num_views,
                                           1, 1.0, _capi._ptr(out), _capi._ptr(ws), nbytes, _capi._stream()) == rc
        torch.cuda.synchronize()
        assert bool(torch.all(out == 7.0)) if rc else rel_l2(out.cpu().numpy(), ref.cpu().numpy()) <= 1e-5

    asked, real = [], _capi._workspace

    def short_of_memory(nbytes, device):
        asked.append(nbytes)
        if nbytes >= full:
            raise torch.OutOfMemoryError('no room')
        return real(nbytes, device)

    monkeypatch.setattr(_capi, '_workspace', short_of_memory)
    got = _capi.back_project(g, sino, pix)
    assert asked == [full, least]
    assert rel_l2(got.cpu().numpy(), ref.cpu().numpy()) <= 1e-5
