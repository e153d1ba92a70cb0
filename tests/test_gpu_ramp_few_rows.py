"""Short rows through the FFT ramp filter, from a handful, which get a CTA to a
pair, to as many as share CTAs: against the oracle with the bar of the other
filter tests, and the time of a handful."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from tests.test_gpu_ramp_lengths import test_ramp_filter_vs_oracle as check_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_os", [12, 128, 300, 1000])
@pytest.mark.parametrize("n_lines", [15, 1217, 2433, 4865, 9731])
def test_rows_sharing_a_cta(oracle_lib, lib, n_os, n_lines):
    check_rows(oracle_lib, lib, n_os, n_lines)


@pytest.mark.parametrize("n_os", [32, 512])
def test_few_rows_cost_less_than_rows_that_share_ctas(lib, n_os):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")

    def us(n_lines):
        rows = torch.rand(n_lines * n_os, device="cuda")
        taps = np.zeros(2 * n_os, np.float32)
        f = lambda: L.call("ctbb_ramp_filter_device", C.c_void_p(rows.data_ptr()), n_lines, n_os,
                           taps.ctypes.data_as(C.POINTER(C.c_float)))
        f()
        best = 1e9
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(200):
                f()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 5.0)
        return best

    few, many = us(16), us(1300)
    print("16 rows of %d: %.1f us, 1300: %.1f us" % (n_os, few, many))
    assert few <= 0.75 * many
