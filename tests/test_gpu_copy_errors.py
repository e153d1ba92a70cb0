"""The word a kernel sets when its bounded wait on a copy into shared memory
runs out (here set by hand): the next call of that context that looks reports
it, once, and no other context does."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.fixture
def word(lib):
    """The library-wide context's word (an internal symbol)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    f = lib._ZN4ctbb15copy_error_wordEv
    f.restype = C.POINTER(C.c_int)
    w = f()
    assert w and w[0] == 0
    yield w
    w[0] = 0


@pytest.fixture
def scan(tmp_path):
    s = H.Scan(scans.tiny(1, 1, adaptive_filtration=1.0, nx=16, ny=16, n_slices=4), str(tmp_path))
    yield s
    s.close()


def _stage_calls(lib, scan, torch):
    mr, d = scan.mr, H.dims(scan.mr)
    raw = torch.zeros(d["n_raw"], device="cuda")
    out = torch.zeros(d["n_raw"], device="cuda")
    rows = torch.zeros(d["n_rebin"], device="cuda")
    n_os, n_lines = mr.cg.n_channels_oversampled, d["n_views"] * mr.cg.n_rows
    quads = torch.zeros(d["n_rebin"] * 4, dtype=torch.float16, device="cuda")
    scale = torch.ones(n_lines, device="cuda")
    block = torch.zeros(d["n_block"], device="cuda")
    image = torch.zeros(d["n_image"], device="cuda")
    final = torch.zeros(lib.ctbb_n_slices_final(C.byref(mr)) * d["plane"], device="cuda")
    taps = H.taps_of(mr)
    p = lambda t: C.c_void_p(t.data_ptr())
    h_taps = taps.ctypes.data_as(C.POINTER(C.c_float))
    keep = (raw, out, rows, quads, scale, block, image, final, taps)
    return keep, {
        "adaptive": lambda: lib.ctbb_adaptive_filter_device(C.byref(mr), p(raw), p(out)),
        "adaptive_noalloc": lambda: lib.ctbb_adaptive_filter_device_noalloc(C.byref(mr), p(raw), p(out)),
        "rebin": lambda: lib.ctbb_rebin_device(C.byref(mr), p(raw), p(rows)),
        "ramp": lambda: lib.ctbb_ramp_filter_device(p(rows), n_lines, n_os, h_taps),
        "ramp_fp16": lambda: lib.ctbb_ramp_filter_fp16_device(p(rows), n_lines, n_os, h_taps, mr.cg.n_rows, p(quads),
                                                              p(scale)),
        "backproject": lambda: lib.ctbb_backproject_device(C.byref(mr), p(rows), p(block)),
        "backproject_fp16": lambda: lib.ctbb_backproject_fp16_device(C.byref(mr), p(quads), p(scale), p(block)),
        "finalize": lambda: lib.ctbb_finalize_device(C.byref(mr), p(image), p(final), C.c_float(0.0)),
    }


@pytest.mark.parametrize("stage", ["adaptive", "adaptive_noalloc", "rebin", "ramp", "ramp_fp16", "backproject",
                                   "backproject_fp16", "finalize"])
def test_next_stage_call_reports_it_once(lib, word, scan, stage):
    import torch
    scan.next_block()
    keep, calls = _stage_calls(lib, scan, torch)
    assert calls[stage]() == 0
    torch.cuda.synchronize()
    word[0] = 1
    assert L.STATUS[calls[stage]()] == "CTBB_ERR_CUDA"
    assert b"copy into shared memory" in lib.ctbb_last_error()
    assert calls[stage]() == 0
    torch.cuda.synchronize()


def test_other_contexts_do_not_report_it(lib, word, scan):
    import torch
    n_final = lib.ctbb_n_slices_final(C.byref(scan.mr)) * scan.mr.rp.nx * scan.mr.rp.ny
    frames = torch.from_numpy(np.ascontiguousarray(scan.frames.reshape(-1))).cuda()
    out = torch.zeros(n_final, device="cuda")
    ctx = C.c_void_p()
    L.call("ctbb_context_create", C.byref(ctx))
    args = (C.byref(scan.mr), C.c_void_p(frames.data_ptr()), C.c_void_p(out.data_ptr()), C.c_float(0.0))
    try:
        word[0] = 1
        assert lib.ctbb_context_reconstruct_scan_device(ctx, *args) == 0
        assert L.STATUS[lib.ctbb_reconstruct_scan_device(*args)] == "CTBB_ERR_CUDA"
        assert lib.ctbb_reconstruct_scan_device(*args) == 0
    finally:
        L.call("ctbb_context_destroy", ctx)
