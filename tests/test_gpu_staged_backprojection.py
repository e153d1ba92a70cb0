"""The staged backprojector (detector boxes of a tile in shared memory) against
the oracle at the sizes where it can go wrong: images that end inside a tile,
pixels on either side of the box widths it holds (and so of its 16 x 8 and
8 x 8 tiles and of the other forms), 8 to 128 detector rows (boxes of one copy
to sixteen, steps of one visit to four), windows of few and of many half
turns, tables moving in, every focal spot mode, a rows pointer off 16 bytes.

Bars: those of the other backprojection tests, 1 HU max and 0.1 HU RMS against
the reference's float arithmetic on the same rows."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests import helpers as H

pytestmark = pytest.mark.gpu

CASES = [
    # z, phi, raw rows, views per turn, channels, nx, ny, pitch, table
    (0, 0, 8, 96, 64, 17, 9, 1.0, "out"),      # one column past a tile in x and y, 1-copy boxes
    (1, 1, 64, 192, 64, 33, 31, 0.8, "out"),   # 128 rows, 3 half turns, one visit to a half
    (0, 1, 32, 192, 96, 16, 8, 1.4, "in"),     # exactly one tile; pixels of 6.3 mm
    (1, 0, 10, 96, 64, 40, 24, 0.6, "out"),    # 20 rows: boxes past the last view's rows
    (0, 0, 64, 100, 128, 47, 50, 1.1, "in"),   # 8 x 8 tiles
    (1, 1, 4, 96, 66, 32, 32, 1.0, "out"),     # 8 rows after z-FFS, 17 or more half turns
    (0, 0, 16, 96, 65, 20, 20, 1.0, "out"),    # 130 samples a row: not a multiple of 16 bytes
    (0, 0, 16, 96, 320, 12, 12, 1.0, "out"),   # pixels wider than any box
]


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _block(tmp_path, oracle_lib, z, phi, rows, views, channels, nx, ny, pitch, table):
    spec = scans.tiny(z, phi, n_rows_raw=rows, n_proj_turn=views, n_channels=channels, nx=nx, ny=ny, n_slices=6,
                      pitch=pitch, table_dir=table, seed=3 + nx)
    scan = H.Scan(spec, str(tmp_path))
    raw = scan.next_block()
    return scan, H.oracle_block(oracle_lib, scan, raw, adaptive=False)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "z%d_p%d_r%d_v%d_c%d_%dx%d_%s" % (c[:7] + (c[8],)))
def test_block_vs_oracle(torch_cuda, oracle_lib, lib, tmp_path, case):
    torch = torch_cuda
    scan, st = _block(tmp_path, oracle_lib, *case)
    mr = scan.mr
    d = H.dims(mr)
    rows = torch.zeros(st["filtered"].size + 8, device="cuda")
    for shift in (0, 1):  # a rows pointer on and off a 16-byte boundary
        view = rows[shift:shift + st["filtered"].size]
        view.copy_(torch.from_numpy(st["filtered"]))
        out = torch.full((d["n_block"],), -7.0, device="cuda")
        L.call("ctbb_backproject_device", C.byref(mr), C.c_void_p(view.data_ptr()), C.c_void_p(out.data_ptr()))
        torch.cuda.synchronize()
        mx, rms = H.hu_errors(out.cpu().numpy(), st["block"])
        print("shift %d: max %.4f HU rms %.5f HU" % (shift, mx, rms))
        assert mx <= 1.0 and rms <= 0.1, (shift, mx, rms)
    scan.close()


def test_rows_past_the_buffer_are_not_used(torch_cuda, oracle_lib, lib, tmp_path):
    """Non-finite values around the rows buffer do not reach the image: the
    boxes' extra rows and channels are read but not used."""
    torch = torch_cuda
    scan, st = _block(tmp_path, oracle_lib, 1, 0, 10, 96, 64, 40, 24, 0.6, "out")
    n = st["filtered"].size
    padded = torch.full((n + 8192,), float("nan"), device="cuda")
    padded[4096:4096 + n].copy_(torch.from_numpy(st["filtered"]))
    out = torch.empty(H.dims(scan.mr)["n_block"], device="cuda")
    L.call("ctbb_backproject_device", C.byref(scan.mr), C.c_void_p(padded[4096:].data_ptr()),
           C.c_void_p(out.data_ptr()))
    torch.cuda.synchronize()
    mx, rms = H.hu_errors(out.cpu().numpy(), st["block"])
    assert np.isfinite(mx) and mx <= 1.0 and rms <= 0.1, (mx, rms)
    scan.close()
