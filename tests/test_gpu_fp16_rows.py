"""The reduced-storage ramp filter's footprint words where their stores change
form -- one tile and several, a ragged last tile of columns and of rows, views
of 1 to 128 rows, output on and off 16 bytes -- and the split of the rows from
pointers on and off 16 bytes: every word against the FP64 filter, with the bar
of the other tests of this filter, and nothing written outside."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from tests.test_gpu_precision import assert_close, fp64_filter, fptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_os", [64, 256, 320, 512, 1472])
@pytest.mark.parametrize("rpv,views", [(1, 131), (4, 50), (64, 3), (128, 1)])
@pytest.mark.parametrize("shift", [0, 1])
def test_footprint_words(oracle_lib, lib, n_os, rpv, views, shift):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n_lines = rpv * views
    rng = np.random.default_rng(n_os + rpv)
    bump = 3.0 * np.clip(1.0 - ((np.arange(n_os) - n_os / 2) / (0.4 * n_os)) ** 2, 0, None)
    rows = (bump[None, :] * rng.uniform(0.5, 1.5, (n_lines, 1)) +
            0.05 * rng.standard_normal((n_lines, n_os))).astype(np.float32)
    taps = np.zeros(2 * n_os, np.float32)
    L.call("ctbb_ramp_filter_taps", n_os, C.c_float(0.352), C.c_float(1.0), C.c_float(1.0), fptr(taps))
    held = torch.full((rows.size + 8,), float("nan"), device="cuda")
    held[shift:shift + rows.size].copy_(torch.from_numpy(rows.ravel()))
    out = torch.full(((rows.size + 4) * 4,), -3.0, dtype=torch.float16, device="cuda")
    scale = torch.empty(n_lines, device="cuda")
    L.call("ctbb_ramp_filter_fp16_device", C.c_void_p(held[shift:].data_ptr()), n_lines, n_os, fptr(taps), rpv,
           C.c_void_p(out[4 * shift:].data_ptr()), C.c_void_p(scale.data_ptr()))
    torch.cuda.synchronize()
    words = out.float().cpu().numpy().reshape(-1, 4)
    assert (words[:shift] == -3.0).all() and (words[shift + rows.size:] == -3.0).all()
    sc = scale.cpu().numpy().astype(np.float64).reshape(views, rpv)
    assert np.all(sc == sc[:, :1])
    q = words[shift:shift + rows.size].reshape(views, rpv, n_os, 4) * sc[:, :1, None, None]
    want = fp64_filter(oracle_lib, rows, taps).reshape(views, rpv, n_os)
    assert_close(q[..., 0].reshape(-1, n_os), want.reshape(-1, n_os))
    assert_close(q[:, :, :-1, 1].reshape(-1, n_os - 1), want[:, :, 1:].reshape(-1, n_os - 1))
    assert np.all(q[:, :, -1, 1] == 0) and np.all(q[:, -1, :, 2:] == 0)
    if rpv > 1:
        assert_close(q[:, :-1, :, 2].reshape(-1, n_os), want[:, 1:].reshape(-1, n_os))
        assert_close(q[:, :-1, :-1, 3].reshape(-1, n_os - 1), want[:, 1:, 1:].reshape(-1, n_os - 1))
