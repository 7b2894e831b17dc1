"""Sizes of the workspaces that hold a transposed copy of the sinogram (host-side queries of the library): the copy costs a
VCD step and a batch no memory of its own, and a plain back projection can do without it."""
import ctypes

import pytest

from mbirjax_b200 import _capi


def _geom(kind, views, rows, channels):
    g = _capi.MbxGeom()
    g.kind = kind
    g.num_views, g.num_det_rows, g.num_det_channels = views, rows, channels
    g.num_recon_rows = g.num_recon_cols = channels
    g.num_recon_slices = rows
    g.delta_det_channel = g.delta_det_row = g.delta_voxel = 1.0
    g.psf_radius = g.bp_psf_radius = 1
    g.entries_per_cylinder_batch = 128
    g.magnification = 1.0
    g.source_detector_dist = float('inf') if kind == _capi.MBX_GEOM_PARALLEL else 4.0 * channels
    g.angles = 16  # a device pointer; not read by a size query
    return g


@pytest.mark.parametrize('kind', [_capi.MBX_GEOM_PARALLEL, _capi.MBX_GEOM_CONE])
def test_copy_shares_memory_with_the_projection_it_precedes(kind):
    lib = _capi.load_library()
    views, rows, channels = 652, 60, 436
    g = _geom(kind, views, rows, channels)
    n = 50000
    sino, copy = 4 * views * rows * channels, 4 * views * rows * (channels + 4)
    full = lib.mbx_back_project_workspace_bytes(ctypes.byref(g), n, views)
    least = lib.mbx_back_project_least_workspace_bytes(ctypes.byref(g), n, views)
    assert full >= copy and least <= full - copy + (12 << 20)
    fp = lib.mbx_forward_project_workspace_bytes(ctypes.byref(g), n, views)
    step = lib.mbx_vcd_subset_step_workspace_bytes(ctypes.byref(g), n)
    assert step <= 2 * 4 * n * rows + max(sino + fp, full) + (1 << 16)


def test_batch_holds_one_sinogram_per_scan_beside_the_caller():
    views, rows, channels = 400, 40, 300
    scans = []
    for i in range(4):
        sc = _capi.MbxScan()
        sc.geom = _geom(_capi.MBX_GEOM_PARALLEL, views, rows, channels)
        sc.flat_recon = sc.error_sinogram = sc.fm_hessian = sc.partition = sc.sinogram = sc.full_indices = 16
        sc.num_subsets, sc.subset_size, sc.num_full_indices = 4, 17000, 68000
        sc.qp = _capi.qggmrf_params([1 / 6.0] * 6, 1.0, 2.0, 1.2, 1.0)
        scans.append(sc)
    got = _capi.vcd_batched_workspace_bytes(scans, 16)
    copy = 4 * views * rows * (channels + 4)
    assert got >= 4 * copy  # (windows are read, so the copies are there)
    assert got <= 4 * (copy + 2 * 4 * 17000 * rows) + (16 << 20)
