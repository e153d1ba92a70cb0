"""Batched scans of float rows that only the slice-chunk form holds: windows of
more than 8 half turns with rows off 16 bytes (130 samples), and a large image
under a detector of two rows beside a small one that is staged.  With the launch
shape chosen by the autotuner for the scan alone too, a stack of the batch is
the same to the bit."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests import helpers as H
from tests.test_gpu_batch import _alone
from tests.test_gpu_batch_forms import _batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds", [[dict(n_channels=65, n_rows_raw=8, nx=48, ny=48, seed=1),
                                    dict(n_channels=65, n_rows_raw=4, nx=33, ny=20, seed=2, table_dir="in")],
                                   [dict(n_channels=64, n_rows_raw=2, nx=120, ny=120, seed=3),
                                    dict(n_channels=64, n_rows_raw=2, nx=40, ny=40, seed=4)]],
                         ids=["rows_of_130", "two_rows"])
def test_batch_equals_tuned_scan_alone(lib, tmp_path, kinds):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    batch = [H.Scan(scans.tiny(0, 0, n_proj_turn=96, n_slices=4, **k), str(tmp_path / str(i)))
             for i, k in enumerate(kinds)]
    got = _batch(torch, batch)
    L.call("ctbb_set_autotune", 1)
    try:
        for g, s in zip(got, batch):
            np.testing.assert_array_equal(g, _alone(torch, lib, s))
    finally:
        L.call("ctbb_set_autotune", 0)
        for s in batch:
            s.close()


def test_small_batch_runs_its_angle_chunks_together(lib, tmp_path):
    """Two scans of two tiles each: their angle chunks are one launch, not one
    launch after another over a handful of CTAs."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    batch = [H.Scan(scans.tiny(0, 0, n_proj_turn=96, n_slices=4, n_channels=64, n_rows_raw=2, nx=16, ny=16, seed=s),
                    str(tmp_path / str(s))) for s in (6, 7)]
    ins = [torch.from_numpy(np.ascontiguousarray(s.frames.reshape(-1))).cuda() for s in batch]
    outs = [torch.empty(lib.ctbb_n_slices_final(C.byref(s.mr)) * 256, device="cuda") for s in batch]
    L.call("ctbb_batch_begin")
    for s, d, o in zip(batch, ins, outs):
        L.call("ctbb_batch_add_device", C.byref(s.mr), C.c_void_p(d.data_ptr()), C.c_void_p(o.data_ptr()),
               C.c_float(0.0))
    before = lib.ctbb_kernel_launch_count()
    L.call("ctbb_batch_run")
    assert lib.ctbb_kernel_launch_count() - before <= 6  # chunks, combine, a finalize for each scan; 18 one by one
    for s in batch:
        s.close()
