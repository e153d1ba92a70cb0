"""The rules that send a call to the kernels that stage detector samples in
shared memory, and the extents of what those copy, checked on the host over
plans of many shapes: every sample such a kernel addresses lies in its copy."""
import ctypes as C
import os
import subprocess

import pytest

from ctbangbang_gb300 import build as B
from ctbangbang_gb300 import lib as L
from ctbangbang_gb300 import scans
from tests.conftest import REPO


def _native(name):
    """tests/native/<name>.cu as a library on top of the built one."""
    src = os.path.join(REPO, "tests", "native", name + ".cu")
    out = os.path.join(B.BUILD, name + "_check.so")
    deps = [src, L.LIB_PATH, *(os.path.join(B.CSRC, f) for f in os.listdir(B.CSRC) if f.endswith((".h", ".cuh")))]
    if B._stale(out, deps):
        cmd = [B._nvcc(), *B.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I", os.path.join(REPO, "include"),
               "-I", B.CSRC, "-Xcompiler", "-fPIC,-ffp-contract=off", "-shared", "-o", out, src, L.LIB_PATH,
               "-Xlinker", "-rpath=" + os.path.dirname(L.LIB_PATH)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
    return C.CDLL(out)


@pytest.fixture(scope="module")
def rebin_check(lib):
    return _native("staged_rebin")


def _rebin(check, spec, tmp_path):
    mr = scans.plan_spec(spec, str(tmp_path))
    L.call("ctbb_update_block_info", C.byref(mr))
    frames, outside = C.c_int(-1), C.c_longlong(-1)
    assert check.check_staged_rebin(C.byref(mr), C.byref(frames), C.byref(outside)) == 0
    scans.free_plan(mr)
    return frames.value, outside.value


# z, phi, channels, views per turn, fan angle, staged
REBIN = [(z, p, c, v, 0.48, True) for z in (0, 1) for p in (0, 1)
         for c, v in ((64, 96), (68, 101), (256, 384), (736, 1152))]
REBIN += [(0, 0, 64, 1152, 0.96, True), (0, 0, 66, 96, 0.48, False),
          # channels past 90 degrees: their view coordinate is not a number
          (0, 0, 64, 96, 2.4, False), (1, 0, 64, 96, 2.4, False), (0, 1, 64, 96, 2.4, False), (1, 1, 64, 96, 2.4, False)]


@pytest.mark.parametrize("z,phi,channels,views,fan,staged", REBIN)
def test_rebin_taps_lie_in_their_box(rebin_check, tmp_path, z, phi, channels, views, fan, staged):
    spec = scans.tiny(z, phi, n_channels=channels, n_proj_turn=views, fan_angle_increment=fan / channels, nx=8, ny=8,
                      n_slices=4)
    frames, outside = _rebin(rebin_check, spec, tmp_path)
    assert (frames > 0) == staged and outside == 0, (frames, outside)
