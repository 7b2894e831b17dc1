"""What a batch prepares for the windows of its back projections: host-only programs over the library's headers, compiled
with nvcc and run on the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _run(name, tmp_path):
    nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    if not os.path.exists(nvcc):
        pytest.skip('nvcc is not available')
    exe = str(tmp_path / name)
    subprocess.run([nvcc, '-std=c++17', '--expt-relaxed-constexpr', '-gencode', 'arch=compute_100a,code=sm_100a',
                    '-o', exe, os.path.join(HERE, name + '.cu')], check=True, capture_output=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    assert res.stdout.startswith('ok ')
    return [int(v) for v in res.stdout.split()[1:]]


def test_each_back_projection_has_a_tensor_map_of_its_own_rows(tmp_path):
    """Subset, initial and Hessian back projections of a scan can have slice tiles of different heights (a list that leaves
    the chip idle takes lower ones): each that reads windows copies through a map whose box has its own rows."""
    scans, differ, with_windows, without = _run('batch_windows_check', tmp_path)
    assert scans > 5000 and differ > 100  # the sweep holds scans that one map could not serve
    assert with_windows > 300 and without > 300


def test_windows_of_few_slices_keep_their_width(tmp_path):
    """With at most 4 slices a window holds up to 288 channels: its width and first channel survive the word they share.
    A box's window holds the taps of its pixels whichever way their centre channel is rounded."""
    windows, big, pixels = _run('bp_window_check', tmp_path)
    assert windows > 100000 and big > 1000 and pixels > 1000000


def test_maps_in_global_memory_are_acquired_before_their_first_copy():
    """The batched stages read their tensor maps from the workspace, where older maps may have stood: the kernel that hands
    a record's map on acquires it first (a stale map can not be brought about on demand, so this reads the source)."""
    with open(os.path.join(HERE, os.pardir, 'mbirjax_b200', 'csrc', 'vcd_batched.cu')) as f:
        text = f.read()
    for use in [i for i in range(len(text)) if text.startswith('bp_fast_run<', i)]:
        kernel = text[text.rindex('__global__', 0, use):use]
        assert 'bpf_acquire_map(' in kernel
    assert 'bp_fast_run<' in text


def test_plans_of_the_second_forward_variant_and_of_the_scratch(tmp_path):
    """The 4-CTA forward plans hold what each mode reads, and the partial sums of the entry point that allocates nothing
    fit its scratch."""
    assert _run('many_plan_check', tmp_path)[0] > 50000
