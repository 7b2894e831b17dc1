"""Batched reconstructions at the sizes where the windows of the batched back projections can go wrong, against the plain
path (whose back projections make their plans and maps call by call)."""
import numpy as np
import pytest
import torch

import mbirjax_b200 as mb
from mbirjax_b200 import _capi
from mbirjax_b200.batched import BatchedVCD, release_batched_sessions
from mbirjax_b200.utilities import gen_ellipsoid_phantom
from cases import rel_l2

pytestmark = pytest.mark.gpu


def _scan(kind, views, rows, channels, seed, subsets=4):
    ang = np.linspace(0, np.pi if kind == 'parallel' else 2 * np.pi, views, endpoint=False).astype(np.float32)
    if kind == 'parallel':
        model = mb.ParallelBeamModel((views, rows, channels), ang)
    else:
        model = mb.ConeBeamModel((views, rows, channels), ang, 4.0 * channels, 4.0 * channels)
    model.set_params(sharpness=0.0, granularity=[subsets], partition_sequence=[0], verbose=0)
    ph = gen_ellipsoid_phantom(tuple(model.get_params('recon_shape')), 5, seed).numpy()
    np.random.seed(seed)
    sino = model.forward_project(torch.as_tensor(ph, device='cuda')).cpu().numpy()
    noise = np.random.default_rng(seed).normal(0, 0.01 * np.abs(sino).max(), sino.shape)
    return model, (sino + noise).astype(np.float32)


def _batch_matches_plain(items, weights, seeds, iters=2):
    """Both paths add the same float32 terms in other orders: a few 1e-7 a projection, and some 1e-6 of the recon after
    a few iterations; the bar is the one of the batched tests, 1e-5."""
    release_batched_sessions()
    _capi.get_device_error()
    models, sinos = [m for m, _ in items], [s for _, s in items]
    recons, _ = BatchedVCD(models, sinos, weights=weights, seeds=seeds).recon(max_iterations=iters)
    assert _capi.get_device_error() == 0
    for i, (model, sino) in enumerate(items):
        np.random.seed(seeds[i])
        plain, _ = model.recon(sino, weights=None if weights is None else weights[i], max_iterations=iters,
                               stop_threshold_change_pct=0, logfile_path=None, print_logs=False)
        assert rel_l2(recons[i].cpu().numpy(), plain.cpu().numpy()) <= 1e-5
    release_batched_sessions()


@pytest.mark.parametrize('weighted', [False, True])
def test_cone_scans_whose_back_projections_differ_in_tile_height(cuda, weighted):
    """The subsets of these scans take lower slice tiles than their set-up's back projections."""
    items = [_scan('cone', 60, 32, 64, 3), _scan('cone', 60, 32, 96, 4), _scan('cone', 60, 40, 64, 5)]
    ws = [np.exp(-s / s.max()).astype(np.float32) for _, s in items] if weighted else None
    _batch_matches_plain(items, ws, [3, 4, 5])


@pytest.mark.parametrize('weighted', [False, True])
def test_cone_batch_that_fills_the_chip(cuda, weighted):
    """Subset, initial and (weighted) Hessian back projections read windows."""
    items = [_scan('cone', 20 + i, 96 - i, 96 + i, i, 1) for i in range(8)]
    ws = [np.exp(-s / s.max()).astype(np.float32) for _, s in items] if weighted else None
    _batch_matches_plain(items, ws, list(range(8)))


@pytest.mark.parametrize('channels', [256, 260, 300])
@pytest.mark.parametrize('subsets', [1, 4, 48])
def test_parallel_scans_of_few_slices(cuda, channels, subsets):
    """With at most 4 slices a window holds up to 288 channels, and warps whose pixels lie across the grid (where the
    Z-order jumps) take windows of that width (1 subset; the others read their taps from the sinograms)."""
    items = [_scan('parallel', 90, rows, channels, rows, subsets) for rows in (1, 3, 4)]
    _batch_matches_plain(items, None, [1, 3, 4], iters=1 if subsets == 48 else 2)


def test_batches_of_different_shapes_one_after_another(cuda):
    """Each batch's tensor maps stand where those of the batch before may have stood."""
    for kind, shapes in (('cone', [(40, 28, 64), (30, 20, 48)]), ('parallel', [(60, 30, 80), (50, 12, 60)]),
                         ('cone', [(30, 20, 48), (40, 28, 64)]), ('parallel', [(50, 12, 60), (60, 30, 80)])):
        _batch_matches_plain([_scan(kind, *s, i) for i, s in enumerate(shapes)], None, [0, 1])


def test_a_copy_that_never_completes_is_given_up(cuda, tmp_path):
    """One warp waits for a barrier that nothing completes: the wait ends within its limit, with the error flagged."""
    import os
    import shutil
    import subprocess
    nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    if not os.path.exists(nvcc):
        pytest.skip('nvcc is not available')
    exe = str(tmp_path / 'bp_wait_check')
    subprocess.run([nvcc, '-std=c++17', '--expt-relaxed-constexpr', '-gencode', 'arch=compute_100a,code=sm_100a', '-o', exe,
                    os.path.join(os.path.dirname(os.path.abspath(__file__)), 'bp_wait_check.cu')], check=True,
                   capture_output=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0 and res.stdout.startswith('ok '), res.stdout + res.stderr


def test_peek_leaves_the_error_word(cuda):
    """peek_device_error reads the word after the stream's work, and leaves it for get_device_error; a caller's bad index
    (bit 0) is no failure of the library."""
    model, sino = _scan('parallel', 8, 4, 32, 1)
    _capi.get_device_error()
    _capi.back_project(model._geometry(), torch.as_tensor(sino, device=cuda),
                       torch.tensor([5, -1, 7], dtype=torch.int32, device=cuda))
    assert _capi.peek_device_error(cuda) == 1
    _capi.raise_on_failed_projection(cuda)
    assert _capi.get_device_error() == 1
    assert _capi.peek_device_error(cuda) == 0
