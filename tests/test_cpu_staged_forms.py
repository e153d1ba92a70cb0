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


@pytest.fixture(scope="module")
def box_check(lib):
    return _native("staged_backproject")


def _boxes(check, spec, tmp_path, n_slices=None, angle_step=1):
    mr = scans.plan_spec(spec, str(tmp_path))
    L.call("ctbb_update_block_info", C.byref(mr))
    if n_slices is not None:
        mr.ri.n_slices_block = n_slices
    visits, outside, misread = C.c_longlong(-1), C.c_longlong(-1), C.c_longlong(-1)
    assert check.check_staged_boxes(C.byref(mr), angle_step, C.byref(visits), C.byref(outside), C.byref(misread)) == 0
    scans.free_plan(mr)
    return visits.value, outside.value, misread.value


# z, phi, raw rows, views per turn, channels, nx, ny, pitch, table
BOXES = [(0, 0, 8, 96, 64, 17, 9, 1.0, "out"), (1, 1, 64, 192, 64, 33, 31, 0.8, "out"),
         (0, 1, 32, 192, 96, 48, 24, 1.4, "in"), (1, 0, 10, 101, 64, 40, 24, 0.6, "out")]


@pytest.mark.parametrize("z,phi,rows,views,channels,nx,ny,pitch,table", BOXES)
def test_backprojection_samples_lie_in_their_box(box_check, tmp_path, z, phi, rows, views, channels, nx, ny, pitch,
                                                 table):
    spec = scans.tiny(z, phi, n_rows_raw=rows, n_proj_turn=views, n_channels=channels, nx=nx, ny=ny, n_slices=6,
                      pitch=pitch, table_dir=table)
    visits, outside, misread = _boxes(box_check, spec, tmp_path)
    assert visits > 0 and outside == 0 and misread == 0, (visits, outside, misread)


@pytest.mark.parametrize("n_slices", [1, 5, 9, 31])
@pytest.mark.parametrize("z,phi,rows,channels,nx,ny,coll", [(0, 1, 64, 166, 35, 28, 0.3), (1, 0, 8, 60, 12, 14, 3.0),
                                                            (1, 1, 16, 48, 33, 9, 1.0)])
def test_slices_past_the_end_of_a_block(box_check, tmp_path, z, phi, rows, channels, nx, ny, coll, n_slices):
    """A block of fewer slices than whole groups of 8: a warp reads for all 8."""
    spec = scans.tiny(z, phi, n_rows_raw=rows, n_proj_turn=40, n_channels=channels, nx=nx, ny=ny, n_slices=4)
    spec.coll = spec.slice_thickness = coll
    spec.start_pos = scans.allowed_margin(spec) + 2.0
    spec.turns = scans.needed_turns(spec)
    visits, outside, misread = _boxes(box_check, spec, tmp_path, n_slices)
    assert visits > 0 and outside == 0 and misread == 0, (visits, outside, misread)


# channels, nx, ny, field of view, origin
COARSE = [(16, 19, 9, 374.0, 0.0), (16, 6, 6, 370.0, 0.0), (20, 12, 5, 300.0, 60.0), (24, 30, 30, 380.0, 0.0)]


@pytest.mark.parametrize("channels,nx,ny,fov,x0", COARSE)
@pytest.mark.parametrize("fan", [0.46, 1.2])
def test_tiles_of_tens_of_centimetres(box_check, tmp_path, channels, nx, ny, fov, x0, fan):
    """Few channels, large pixels: a tile's bounds may reach the source's circle
    where its voxels do not; such images take another form."""
    spec = scans.tiny(1, 1, n_rows_raw=32, n_proj_turn=100, n_channels=channels, nx=nx, ny=ny, n_slices=4,
                      fan_angle_increment=fan / channels)
    spec.recon_fov, spec.x_origin = fov, x0
    visits, outside, misread = _boxes(box_check, spec, tmp_path)
    assert outside == 0 and misread == 0, (visits, outside, misread)


def _shape(check, spec, tmp_path):
    mr = scans.plan_spec(spec, str(tmp_path))
    L.call("ctbb_update_block_info", C.byref(mr))
    cw, pitch = C.c_int(-1), C.c_int(-1)
    assert check.check_staged_shape(C.byref(mr), C.byref(cw), C.byref(pitch)) == 0
    scans.free_plan(mr)
    return cw.value, pitch.value


# z, raw rows, pitch, pixels, staged; all windows of more than 8 half turns
WINDOWS = [(0, 2, 1.0, 80, True), (0, 2, 1.0, 120, False), (0, 4, 0.8, 80, True), (0, 4, 0.8, 150, False),
           (1, 4, 1.0, 256, False), (0, 8, 0.5, 200, True), (0, 8, 0.3, 384, False), (0, 16, 0.25, 384, True)]


@pytest.mark.parametrize("z,rows,pitch,pixels,staged", WINDOWS)
def test_windows_of_many_half_turns(box_check, tmp_path, z, rows, pitch, pixels, staged):
    """A detector of few slices' height takes the staged form for small images only."""
    spec = scans.tiny(z, 0, n_rows_raw=rows, n_proj_turn=96, n_channels=128, nx=pixels, ny=pixels, n_slices=4, pitch=pitch)
    assert (_shape(box_check, spec, tmp_path)[0] > 0) == staged


# what a scan's blocks run: channels, raw rows, z, phi, views, nx, ny, field of view, pitch, table -> columns / 32
# of a tile, channels of its box
TILES = {
    "one_16x8_tile": ((64, 8, 0, 0, 96, 16, 8, 30.0, 1.0, "out"), (4, 56)),
    "one_16x8_tile_wide_box": ((64, 8, 0, 0, 96, 16, 8, 60.0, 1.0, "in"), (4, 88)),
    "half_a_tile": ((64, 8, 0, 0, 96, 8, 8, 30.0, 1.0, "out"), (4, 88)),
    "past_a_tile": ((64, 8, 0, 0, 96, 17, 9, 40.0, 1.0, "out"), (4, 56)),
    "8x8_tiles": ((256, 64, 0, 0, 100, 50, 47, 100.0, 1.1, "in"), (2, 88)),
    "8x8_tiles_past_both": ((64, 8, 0, 0, 96, 9, 17, 60.0, 1.0, "out"), (2, 88)),
    "8x8_tiles_2mm_pixels": ((128, 8, 1, 1, 96, 47, 50, 160.0, 1.0, "out"), (2, 88)),
    "128_rows": ((64, 64, 1, 1, 192, 31, 33, 100.0, 0.8, "out"), (4, 56)),
    "too_coarse": ((320, 8, 0, 0, 96, 47, 50, 100.0, 1.0, "out"), (0, 0)),
    "rows_of_130": ((65, 16, 0, 0, 96, 20, 20, 30.0, 1.0, "out"), (0, 0)),
}


def tile_spec(name):
    channels, rows, z, phi, views, nx, ny, fov, pitch, table = TILES[name][0]
    spec = scans.tiny(z, phi, n_rows_raw=rows, n_proj_turn=views, n_channels=channels, nx=nx, ny=ny, n_slices=6,
                      pitch=pitch, table_dir=table, seed=5)
    spec.recon_fov = fov
    return spec


@pytest.mark.parametrize("name", TILES)
def test_tile_of_a_block(box_check, tmp_path, name):
    assert _shape(box_check, tile_spec(name), tmp_path) == TILES[name][1]
