"""The adaptive filter with averaging windows up to and past the shared memory
of the kernel that forms the moving means (12 161 frames), against the oracle,
bit for bit."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views", [96, 243220, 243240, 500000])
def test_long_averaging_window(oracle_lib, lib, tmp_path, views):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    scan = H.Scan(scans.tiny(0, 0, n_rows_raw=3, n_channels=12, n_proj_turn=96, nx=8, ny=8, n_slices=4,
                             adaptive_filtration=30.0), str(tmp_path))
    scan.next_block()
    scan.mr.cg.n_proj_ffs = views
    d = H.dims(scan.mr)
    rng = np.random.default_rng(views)
    swing = 3.0 + 2.0 * np.cos(4 * np.pi * np.arange(d["P"]) / d["P"])
    raw = (swing[:, None] * rng.uniform(0.5, 1.0, (d["P"], 36))).astype(np.float32).ravel()
    scan.set_raw(raw)
    oracle_lib.oracle_adaptive_filter(C.byref(scan.mr))
    want = H.view(scan.mr.ctd.raw, d["n_raw"]).copy()
    d_in = torch.from_numpy(raw).cuda()
    out = torch.full_like(d_in, -1.0)
    L.call("ctbb_adaptive_filter_device", C.byref(scan.mr), C.c_void_p(d_in.data_ptr()), C.c_void_p(out.data_ptr()))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), want)
    scan.close()
