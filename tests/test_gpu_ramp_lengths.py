"""The FFT ramp filter at the row lengths where its transform changes (powers of
two, 1024 / 1025, 1535 / 1536) and inside each range (short transforms share a
CTA), with one row, an odd and an even
number of rows, against the oracle's double-precision FFT convolution; bar as
in the other filter tests, 2e-5 of the largest sample."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L

pytestmark = pytest.mark.gpu

fptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))


@pytest.mark.parametrize("n_os", [5, 16, 48, 128, 129, 256, 500, 1024, 1026, 1344, 1535, 1536, 1537])
@pytest.mark.parametrize("n_lines", [1, 2, 777])
def test_ramp_filter_vs_oracle(oracle_lib, lib, n_os, n_lines):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n_os + n_lines)
    rows = rng.standard_normal((n_lines, n_os)).astype(np.float32)
    taps = rng.standard_normal(2 * n_os).astype(np.float32) if n_lines == 2 else np.zeros(2 * n_os, np.float32)
    if n_lines != 2:
        L.call("ctbb_ramp_filter_taps", n_os, C.c_float(0.3), C.c_float(1.0), C.c_float(1.0), fptr(taps))
    d = torch.from_numpy(np.concatenate([rows.ravel(), np.full(64, 5.0, np.float32)])).cuda()
    L.call("ctbb_ramp_filter_device", C.c_void_p(d.data_ptr()), n_lines, n_os, fptr(taps))
    torch.cuda.synchronize()
    want = rows.copy()
    oracle_lib.oracle_filter_rows(fptr(want), n_lines, n_os, fptr(taps))
    got = d.cpu().numpy()
    assert np.all(got[rows.size:] == 5.0)
    err = float(np.abs(got[:rows.size].reshape(rows.shape).astype(np.float64) - want).max())
    assert err <= 2e-5 * float(np.abs(want).max()), err
