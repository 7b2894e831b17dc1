"""The back projector's windows (bp_fast.cuh) against the oracle where they can go wrong: pixel lists with and without
locality (one window, several, private columns), slice counts at the edges of the tiles, taps of two and three
channels, squared coefficients and weights, view lists, pixels off the detector, and the call without a transposed
copy.  Bar: 1e-5 relative L2, the bar of every projector test (float32 sums of the same terms in either order)."""
import ctypes

import numpy as np
import pytest
import torch

import mbirjax_b200 as mb
import oracle as O
from mbirjax_b200 import _capi
from mbirjax_b200.vcd_utils import gen_full_indices, gen_pixel_partition, morton_sorted_partition
from cases import make_case, rel_l2

pytestmark = pytest.mark.gpu


def _pixels(shape, order, seed=3):
    rng = np.random.default_rng(seed)
    if order == 'raster':
        return np.asarray(gen_full_indices(shape, rng=np.random.RandomState(seed)), dtype=np.int32)
    if order == 'subset':
        part = gen_pixel_partition(shape, 4, rng=np.random.RandomState(seed))
        return morton_sorted_partition(part, shape[1])[1]
    if order == 'sorted-subset':
        return gen_pixel_partition(shape, 16, rng=np.random.RandomState(seed))[2]
    if order == 'few':
        return rng.integers(0, shape[0] * shape[1], 5).astype(np.int32)
    return rng.integers(0, shape[0] * shape[1], 700).astype(np.int32)  # scattered, with duplicates, corners too


def _check(model, geom, order, coeff_power=1, weighted=False, views=None):
    rng = np.random.default_rng(5)
    sino = rng.standard_normal(geom.sinogram_shape).astype(np.float32)
    w = rng.uniform(0.2, 1.0, geom.sinogram_shape).astype(np.float32) if weighted else None
    pix = _pixels(geom.recon_shape, order)
    ref = O.sparse_back_project(geom, sino if w is None else w * sino, pix, view_indices=views, coeff_power=coeff_power)
    g = model._geometry()
    dev = torch.device('cuda')
    args = dict(view_indices=None if views is None else torch.as_tensor(views.astype(np.int32), device=dev),
                coeff_power=coeff_power, weights=None if w is None else torch.as_tensor(w, device=dev))
    s, p = torch.as_tensor(sino, device=dev), torch.as_tensor(pix, device=dev)
    got = _capi.back_project(g, s, p, **args).cpu().numpy()
    plain = _capi.back_project_noalloc(g, s, p, **args).cpu().numpy()  # windows by plain loads
    assert _capi.get_device_error() == 0
    assert rel_l2(got, ref) <= 1e-5
    assert rel_l2(plain, ref) <= 1e-5


@pytest.mark.parametrize('order', ['raster', 'subset', 'sorted-subset', 'scattered', 'few'])
@pytest.mark.parametrize('kind', ['parallel', 'cone', 'translation'])
def test_pixel_orders(cuda, kind, order):
    model, geom = make_case(kind, views=20, rows=37, channels=90)
    _check(model, geom, order)


@pytest.mark.parametrize('rows', [1, 3, 4, 31, 32, 33, 65])
@pytest.mark.parametrize('kind', ['parallel', 'cone'])
def test_slice_tiles(cuda, kind, rows):
    model, geom = make_case(kind, views=17, rows=rows, channels=45)
    _check(model, geom, 'subset')


@pytest.mark.parametrize('delta_voxel', [0.6, 1.0, 1.7])
def test_two_and_three_taps(cuda, delta_voxel):
    model, geom = make_case('parallel', views=18, rows=9, channels=50, delta_voxel=delta_voxel)
    assert model._geometry().psf_radius == 1
    _check(model, geom, 'raster')
    _check(model, geom, 'scattered', coeff_power=2, weighted=True)


@pytest.mark.parametrize('kind', ['parallel', 'cone', 'translation'])
def test_weights_powers_and_views(cuda, kind):
    model, geom = make_case(kind, views=24, rows=30, channels=64, det_channel_offset=2.3)
    _check(model, geom, 'subset', coeff_power=2, weighted=True)
    _check(model, geom, 'scattered', weighted=True)
    _check(model, geom, 'raster', views=np.array([3, 3, 20, 7, 0, 23]))
    _check(model, geom, 'subset', views=np.arange(60) % 24)  # more than the geometry has: some repeat


@pytest.mark.parametrize('kind', ['parallel', 'cone'])
def test_pixels_off_the_detector(cuda, kind):
    """A grid wider than the detector sees: pixels with no tap, with one, and rows beyond the detector."""
    model, geom = make_case(kind, views=16, rows=12, channels=40)
    model.set_params(recon_shape=(70, 64, 12 if kind == 'parallel' else 40))
    from cases import oracle_geometry
    if model._geometry().psf_radius != 1:
        pytest.skip('the wider grid needs the general kernel')
    _check(model, oracle_geometry(model), 'scattered')
    _check(model, oracle_geometry(model), 'subset')


def test_workspace_off_a_16_byte_boundary(cuda):
    """A workspace the TMA cannot read falls back to plain loads, with the same result."""
    model, geom = make_case('cone', views=16, rows=20, channels=48)
    g, lib = model._geometry(), _capi.load_library()
    rng = np.random.default_rng(7)
    sino = torch.as_tensor(rng.standard_normal(geom.sinogram_shape).astype(np.float32), device=cuda)
    pix = torch.as_tensor(_pixels(geom.recon_shape, 'subset'), device=cuda)
    ref = _capi.back_project(g, sino, pix)
    n = int(pix.shape[0])
    need = lib.mbx_back_project_workspace_bytes(ctypes.byref(g), n, g.num_views)
    ws = torch.empty(need + 16, dtype=torch.uint8, device=cuda)
    out = torch.empty_like(ref)
    rc = lib.mbx_sparse_back_project(ctypes.byref(g), _capi._ptr(sino), None, _capi._ptr(pix), n, None, g.num_views, 1,
                                     1.0, _capi._ptr(out), ctypes.c_void_p(ws.data_ptr() + 4), need, _capi._stream())
    assert rc == 0
    torch.cuda.synchronize()
    assert rel_l2(out.cpu().numpy(), ref.cpu().numpy()) <= 1e-6


def test_batched_workspace_off_the_tensor_map_boundary(cuda, monkeypatch):
    """A batch whose workspace starts 16 bytes past a 64-byte boundary copies its windows by plain loads (the same sums
    in the same order), and reconstructs what the aligned one does."""
    from mbirjax_b200 import _capi, batched as B

    class Shifted:
        def __getattr__(self, name):
            return getattr(torch, name)

        def empty(self, *size, **kw):
            if kw.get('dtype') is torch.uint8:
                return torch.empty(size[0] + 64, **kw)[16:16 + size[0]]
            return torch.empty(*size, **kw)

    models, sinos = [], []
    for v, r, c in ((40, 12, 64), (30, 8, 50)):
        m = mb.ParallelBeamModel((v, r, c), np.linspace(0, np.pi, v, endpoint=False).astype(np.float32))
        m.set_params(sharpness=0.0, granularity=[4], partition_sequence=[0], verbose=0)
        models.append(m)
        sinos.append(np.random.default_rng(v).random((v, r, c)).astype(np.float32))
    out = []
    for shift in (False, True):
        B.release_batched_sessions()
        if shift:
            monkeypatch.setattr(_capi, 'torch', Shifted())
        recons, _ = B.BatchedVCD(models, sinos, seeds=[1, 2]).recon(max_iterations=2)
        out.append([x.cpu().numpy() for x in recons])
    B.release_batched_sessions()
    for a, b in zip(*out):
        assert rel_l2(b, a) <= 1e-5
