"""The staged rebinning (a tile's frames in shared memory) against the oracle,
bit for bit, where its tiles end: output channels past a tile of 128, raw rows
past a group of 4, views past a chunk of 16, every focal spot mode, rows in
either order, a raw pointer off 16 bytes and channel counts it leaves to the
gathering form."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests import helpers as H

pytestmark = pytest.mark.gpu

CASES = [
    # z, phi, raw rows, channels, views per turn, reversed rows
    (0, 0, 5, 64, 96, 0), (0, 0, 4, 68, 100, 0), (0, 1, 6, 96, 98, 0), (1, 0, 3, 132, 96, 1), (1, 1, 7, 128, 102, 0),
    (1, 1, 4, 196, 96, 1), (0, 1, 4, 66, 96, 0), (1, 1, 4, 65, 96, 0), (1, 0, 4, 20, 96, 0),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "z%d_p%d_r%d_c%d_v%d_rev%d" % c)
@pytest.mark.parametrize("shift", [0, 1])
def test_rebin_equals_oracle(oracle_lib, lib, tmp_path, case, shift):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    z, phi, rows, channels, views, rev = case
    scan = H.Scan(scans.tiny(z, phi, n_rows_raw=rows, n_channels=channels, n_proj_turn=views, nx=8, ny=8, n_slices=4,
                             reverse_row_interleave=rev, seed=channels), str(tmp_path))
    raw = scan.next_block()
    want = H.oracle_block(oracle_lib, scan, raw, adaptive=False)["rebin"]
    held = torch.full((raw.size + 8,), float("nan"), device="cuda")
    held[shift:shift + raw.size].copy_(torch.from_numpy(raw))
    out = torch.full((want.size + 64,), -3.0, device="cuda")
    L.call("ctbb_rebin_device", C.byref(scan.mr), C.c_void_p(held[shift:].data_ptr()), C.c_void_p(out.data_ptr()))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[:want.size], want)
    assert np.all(got[want.size:] == -3.0)
    scan.close()
