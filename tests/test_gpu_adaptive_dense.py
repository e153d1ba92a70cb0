"""The adaptive filter on frames with many samples above their threshold, which
are smoothed tile by tile: against the oracle bit for bit, where tiles and the
parts of a frame end and where dense frames alternate with sparse ones, and
against the time of a window with few such samples."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _scan(path, rows, channels, seed):
    scan = H.Scan(scans.tiny(1, 1, n_rows_raw=rows, n_channels=channels, n_proj_turn=96, nx=8, ny=8, n_slices=4,
                             adaptive_filtration=30.0, seed=seed), str(path))
    scan.next_block()
    return scan


def _window(scan, low, every=1):
    """Frames that swing over the turn, samples in [low, 1] of their frame's
    level; with `every` > 1 all others hold one such sample only."""
    d = H.dims(scan.mr)
    rng = np.random.default_rng(int(scan.mr.cg.n_channels))
    n = d["n_raw"] // d["P"]
    swing = 3.0 + 2.0 * np.cos(4 * np.pi * np.arange(d["P"]) / scan.mr.cg.n_proj_ffs)
    raw = swing[:, None] * rng.uniform(low, 1.0, (d["P"], n))
    sparse = np.arange(d["P"]) % every != 0
    raw[sparse] *= 0.1
    raw[sparse, rng.integers(0, n, int(sparse.sum()))] = swing[sparse]
    return np.ascontiguousarray(raw.astype(np.float32).ravel())


@pytest.mark.parametrize("rows,channels", [(1, 1100), (2, 513), (9, 130), (33, 129), (17, 128), (7, 257), (40, 36)])
@pytest.mark.parametrize("low,every", [(0.9, 1), (0.0, 1), (0.5, 5)])
def test_dense_frames_equal_oracle(oracle_lib, lib, tmp_path, rows, channels, low, every):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    scan = _scan(tmp_path, rows, channels, 3)
    raw = _window(scan, low, every)
    scan.set_raw(raw)
    oracle_lib.oracle_adaptive_filter(C.byref(scan.mr))
    want = H.view(scan.mr.ctd.raw, raw.size).copy()
    d_in = torch.from_numpy(raw).cuda()
    out = torch.full_like(d_in, -1.0)
    L.call("ctbb_adaptive_filter_device", C.byref(scan.mr), C.c_void_p(d_in.data_ptr()), C.c_void_p(out.data_ptr()))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), want)
    scan.close()


@pytest.mark.parametrize("channels", [736, 738])
def test_dense_window_costs_a_few_sparse_ones(lib, tmp_path, channels):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    scan = _scan(tmp_path, 32, channels, 4)
    out = torch.empty(H.dims(scan.mr)["n_raw"], device="cuda")

    def us(raw):
        d_in = torch.from_numpy(raw).cuda()
        times = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            L.call("ctbb_adaptive_filter_device", C.byref(scan.mr), C.c_void_p(d_in.data_ptr()),
                   C.c_void_p(out.data_ptr()))
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        return sorted(times)[len(times) // 2]

    sparse, dense = us(_window(scan, 0.9, 1 << 20)), us(_window(scan, 0.9))
    print("sparse %.0f us, dense %.0f us" % (sparse, dense))
    assert dense <= 10 * sparse
    scan.close()
