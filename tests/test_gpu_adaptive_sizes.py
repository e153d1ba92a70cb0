"""The adaptive filter against the oracle, bit for bit, where its copy and its
smoothing change form: frames that are not whole groups of four samples, a
pointer off 16 bytes, frames with few samples above their threshold and frames
with nearly all (the list of samples is smoothed in several goes)."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,channels", [(5, 65), (4, 66), (3, 64), (16, 72), (32, 332)])
@pytest.mark.parametrize("dense", [0, 1])
@pytest.mark.parametrize("shift", [0, 1])
def test_adaptive_filter_equals_oracle(oracle_lib, lib, tmp_path, rows, channels, dense, shift):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    scan = H.Scan(scans.tiny(1, 1, n_rows_raw=rows, n_channels=channels, n_proj_turn=96, nx=8, ny=8, n_slices=4,
                             adaptive_filtration=30.0 if dense else 2.0, seed=channels), str(tmp_path))
    raw = scan.next_block().reshape(-1, rows, channels)
    if dense:  # an ellipse's swing over the turn, the same for nearly every sample of a frame
        rng = np.random.default_rng(channels)
        swing = 3.0 + 2.0 * np.cos(4 * np.pi * np.arange(len(raw)) / 96 / 4)
        raw = (swing[:, None, None] * rng.uniform(0.9, 1.0, raw.shape)).astype(np.float32)
    raw = np.ascontiguousarray(raw.ravel())
    want = H.oracle_block(oracle_lib, scan, raw)["adaptive"]
    assert (want != raw).any()
    held = torch.full((raw.size + 8,), float("nan"), device="cuda")
    held[shift:shift + raw.size].copy_(torch.from_numpy(raw))
    out = torch.full((raw.size + 64,), -3.0, device="cuda")
    L.call("ctbb_adaptive_filter_device", C.byref(scan.mr), C.c_void_p(held[shift:].data_ptr()),
           C.c_void_p(out[shift:].data_ptr()))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[shift:shift + raw.size], want)
    assert (got[:shift] == -3.0).all() and (got[shift + raw.size:] == -3.0).all()
    scan.close()
