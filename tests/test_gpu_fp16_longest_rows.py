"""The reduced-storage ramp filter at its longest row, 1536 samples: seven tiles
of footprint words, the last past the padded kernel's end; and a whole scan of
768 channels in that storage, streamed and resident."""
import ctypes as C

import numpy as np
import pytest

from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests import helpers as H
from tests.test_gpu_fp16_rows import test_footprint_words as check_words
from tests.test_gpu_precision import _whole_scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rpv,views", [(1, 131), (4, 50), (64, 3), (128, 1)])
@pytest.mark.parametrize("shift", [0, 1])
def test_footprint_words_of_1536_samples(oracle_lib, lib, rpv, views, shift):
    check_words(oracle_lib, lib, 1536, rpv, views, shift)


def test_whole_scan_of_768_channels(lib, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    scan = H.Scan(scans.tiny(0, 0, n_rows_raw=8, n_channels=768, nx=24, ny=24, n_slices=4, i0=1e6), str(tmp_path))
    resident = _whole_scan(torch, scan.mr, scan.frames, L.STORAGE_FP16)
    streamed = _whole_scan(torch, scan.mr, scan.frames, L.STORAGE_FP16, host=True)
    assert np.isfinite(resident).all() and resident.any()
    np.testing.assert_array_equal(streamed, resident)
    scan.close()
