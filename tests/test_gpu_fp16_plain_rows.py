"""The reduced-storage ramp filter's rows (no footprint words) where the split
of the rows takes another number of registers, from pointers on and off 16
bytes: against the FP64 filter, with the bar of the other tests of this filter,
and nothing written outside."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from tests.test_gpu_precision import assert_close, fp64_filter, fptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_os", [64, 128, 192, 256, 320, 512, 576, 1472, 1536])
@pytest.mark.parametrize("n_lines", [1, 7, 131])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows(oracle_lib, lib, n_os, n_lines, shift):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n_os + n_lines)
    bump = 3.0 * np.clip(1.0 - ((np.arange(n_os) - n_os / 2) / (0.4 * n_os)) ** 2, 0, None)
    rows = (bump[None, :] * rng.uniform(0.5, 1.5, (n_lines, 1)) +
            0.05 * rng.standard_normal((n_lines, n_os))).astype(np.float32)
    taps = np.zeros(2 * n_os, np.float32)
    L.call("ctbb_ramp_filter_taps", n_os, C.c_float(0.352), C.c_float(1.0), C.c_float(1.0), fptr(taps))
    held = torch.full((rows.size + 8,), float("nan"), device="cuda")
    held[shift:shift + rows.size].copy_(torch.from_numpy(rows.ravel()))
    out = torch.full((rows.size + 64,), -3.0, dtype=torch.float16, device="cuda")
    scale = torch.full((n_lines + 1,), -3.0, device="cuda")
    L.call("ctbb_ramp_filter_fp16_device", C.c_void_p(held[shift:].data_ptr()), n_lines, n_os, fptr(taps), 0,
           C.c_void_p(out.data_ptr()), C.c_void_p(scale.data_ptr()))
    torch.cuda.synchronize()
    got, sc = out.float().cpu().numpy(), scale.cpu().numpy().astype(np.float64)
    assert (got[rows.size:] == -3.0).all() and sc[n_lines] == -3.0
    assert_close(got[:rows.size].reshape(n_lines, n_os) * sc[:n_lines, None], fp64_filter(oracle_lib, rows, taps))
