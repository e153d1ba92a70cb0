"""Each tile of the staged backprojector, by blocks that are known to run it
(tests/test_cpu_staged_forms.py), against the oracle: images of one tile, of a
part of one and ending past one, and blocks that end inside a group of eight
slices.  Bars of the other backprojection tests: 1 HU max, 0.1 HU RMS against
the reference's float arithmetic on the same rows."""
import ctypes as C

import pytest

from ctbangbang_gb300 import lib as L
from tests import helpers as H
from tests.test_cpu_staged_forms import TILES, tile_spec

pytestmark = pytest.mark.gpu


def _check(torch, oracle_lib, path, name, slices=None):
    scan = H.Scan(tile_spec(name), str(path))
    raw = scan.next_block()
    st = H.oracle_block(oracle_lib, scan, raw, adaptive=False)
    mr, d = scan.mr, H.dims(scan.mr)
    rows = torch.from_numpy(st["filtered"]).cuda()
    want = st["block"]
    if slices is not None:
        mr.ri.n_slices_block = slices
        want = want[:slices * d["plane"]]
    out = torch.full((want.size + 4096,), -7.0, device="cuda")
    L.call("ctbb_backproject_device", C.byref(mr), C.c_void_p(rows.data_ptr()), C.c_void_p(out.data_ptr()))
    torch.cuda.synchronize()
    mx, rms = H.hu_errors(out[:want.size].cpu().numpy(), want)
    print("%s: max %.4f HU rms %.5f HU" % (name, mx, rms))
    assert mx <= 1.0 and rms <= 0.1, (mx, rms)
    assert (out[want.size:] == -7.0).all()
    mr.ri.n_slices_block = 32
    scan.close()


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("name", TILES)
def test_block_vs_oracle(torch_cuda, oracle_lib, lib, tmp_path, name):
    _check(torch_cuda, oracle_lib, tmp_path, name)


@pytest.mark.parametrize("slices", [1, 5, 8, 9, 31])
@pytest.mark.parametrize("name", ["one_16x8_tile", "8x8_tiles", "128_rows", "rows_of_130"])
def test_blocks_of_fewer_slices(torch_cuda, oracle_lib, lib, tmp_path, name, slices):
    _check(torch_cuda, oracle_lib, tmp_path, name, slices)
