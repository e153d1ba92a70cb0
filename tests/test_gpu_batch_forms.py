"""Batches whose blocks take different backprojectors: the staged form with
enough tiles to halve its angle chunks, two of its tiles side by side, and rows
that it leaves to the other forms (130 samples, not a multiple of 16 bytes).
With the launch shape of a scan alone chosen by the autotuner too, a stack is
the same to the bit."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests import helpers as H
from tests.test_gpu_batch import _alone

pytestmark = pytest.mark.gpu


def _scan(path, channels=64, n=200, fov=100.0, **kw):
    spec = scans.tiny(0, 0, n_rows_raw=16, n_proj_turn=192, n_channels=channels, nx=n, ny=n, n_slices=4, **kw)
    spec.recon_fov = fov
    return H.Scan(spec, str(path))


def _batch(torch, batch):
    ins = [torch.from_numpy(np.ascontiguousarray(s.frames.reshape(-1))).cuda() for s in batch]
    outs = []
    L.call("ctbb_batch_begin")
    for s, d in zip(batch, ins):
        n = L.load().ctbb_n_slices_final(C.byref(s.mr)) * s.mr.rp.nx * s.mr.rp.ny
        outs.append(torch.full((n,), -1.0, device="cuda"))
        L.call("ctbb_batch_add_device", C.byref(s.mr), C.c_void_p(d.data_ptr()), C.c_void_p(outs[-1].data_ptr()),
               C.c_float(0.0))
    L.call("ctbb_batch_run")
    torch.cuda.synchronize()
    return [o.cpu().numpy() for o in outs]


@pytest.mark.parametrize("kinds", [[dict(seed=1)], [dict(seed=1), dict(seed=2, n=40, fov=250.0), dict(seed=3, n=40)],
                                   [dict(channels=65, seed=4, n=48), dict(channels=65, seed=5, n=33, table_dir="in")]],
                         ids=["325_tiles", "two_tiles", "rows_of_130"])
def test_batch_equals_tuned_scan_alone(lib, tmp_path, kinds):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    batch = [_scan(tmp_path / str(i), **k) for i, k in enumerate(kinds)]
    got = _batch(torch, batch)
    L.call("ctbb_set_autotune", 1)
    try:
        for g, s in zip(got, batch):
            np.testing.assert_array_equal(g, _alone(torch, lib, s))
    finally:
        L.call("ctbb_set_autotune", 0)
        for s in batch:
            s.close()


def test_autotuner_times_each_tile(lib, tmp_path):
    """Two fields of view of the same counts run different staged kernels: each
    is timed."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    L.call("ctbb_set_autotune", 1)
    try:
        for i, fov in enumerate((50.0, 250.0)):
            s = _scan(tmp_path / str(i), n=38, fov=fov)
            _alone(torch, lib, s)
            s.close()
    finally:
        L.call("ctbb_set_autotune", 0)
    buf = C.create_string_buffer(1 << 16)
    assert lib.ctbb_autotune_report(buf, len(buf)) > 0
    entries = [e for e in buf.value.decode().splitlines() if e.startswith("38x38x32 ")]
    assert len(entries) == 2, buf.value
