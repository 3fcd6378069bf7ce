"""GPU kernels at the sizes where their dispatch or tiling can go wrong, against the FP64 oracle."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from conftest import relative_rmse

pytestmark = pytest.mark.gpu


# The march differs from the FP64 restatement by the FP32 rounding of the
# sample position (at most 2 ulp of the largest index, 8e-6 voxel below 64) times
# the slope between neighbouring voxels (below 1 for values in [0, 1]), random
# over ~60 samples of mean 0.5, and of the sum (60 x 6e-8): below 1e-5.
TOL_FORWARD = 1e-5


@pytest.mark.parametrize("cone", [True, False])
@pytest.mark.parametrize("nx,ny,nz", [(33, 5, 33), (33, 6, 33), (31, 17, 31), (5, 33, 5), (48, 64, 48), (1, 40, 1),
                                      (30, 1, 30), (34, 29, 26)])
def test_forward_row_counts(fbp, oracle, nx, ny, nz, cone):
    """Detector rows either side of the column march's limit and of a warp, on
    volumes without structure (every voxel counts) and without padding."""
    views, odd_views = 7, 11
    vol = np.random.default_rng(nx * 100 + ny).random((nz, ny, nx), np.float32)
    s = fbp.FBP3D(0)
    s.generate_blank_volume(nx, ny, nz)
    s.write_volume_data(vol)
    if cone:
        s.project_forward_cone_to_projections(4.0 * nx, 2.0 * nx, 1.5 * nx, float(nx), 1.0, views, 0.3)
        c = dict(vox=1.0, du=1.5, dv=1.5, span=2 * math.pi, offset=np.float32(0.3), sod=4.0 * nx, sdd=6.0 * nx)
    else:
        views = odd_views
        s.project_forward_parallel_to_projections(0.5, views, 0.3)
        c = dict(vox=1.0, du=1.0, dv=1.0, span=math.pi, offset=np.float32(0.3))
    got = s.download_projections()
    s.ctx.close()
    ref = oracle.forward_project(vol, dict(c, nu=nx, nv=ny, nviews=views), cone=cone)
    assert relative_rmse(got, ref) < TOL_FORWARD


# FP32 taps of white-noise rows: the position's rounding (2 ulp of a window
# column below 128, 2e-5 of a column) moves a linear tap of unit-variance
# samples by ~2e-5, independent over the views; fraction, weight and sum add a
# few 1e-7: 3e-5 of the image, whose sum over views is as incoherent.
TOL_BP2D = 3e-5


@pytest.mark.parametrize("kind", ["fan", "parallel"])
@pytest.mark.parametrize("nx,nz,views,bins,turns", [
    (64, 64, 96, 90, 1.0), (65, 65, 96, 90, 1.0), (33, 33, 4, 40, 1.0), (1, 1, 8, 5, 1.0),  # quarter turns
    (64, 64, 90, 90, 0.5), (65, 65, 34, 71, 0.5), (97, 97, 2, 70, 0.5),                      # half a turn
    (64, 48, 96, 90, 1.0), (65, 47, 98, 90, 1.0), (31, 2, 6, 40, 1.0), (70, 70, 58, 64, 1.0),  # half turns
    (64, 64, 91, 90, 1.0), (48, 65, 37, 33, 0.5), (40, 40, 64, 41, 0.3), (50, 50, 48, 55, 2.0),  # no / mirror symmetry
    (300, 300, 260, 301, 1.0), (447, 447, 40, 300, 1.0), (450, 450, 38, 300, 0.5), (449, 449, 38, 300, 0.5),
    (600, 600, 44, 300, 1.0), (40, 40, 48, 9, 1.0), (24, 24, 1, 30, 1.0)])
def test_bp2d_view_sets_and_sizes(fbp, oracle, kind, nx, nz, views, bins, turns):
    """Every orbit the 2D backprojector packs (four and two slots, mirrored
    ones, none), odd and non-square images, tiles past the image, detectors
    narrower than the image, on white noise with a start angle, twice (same bits)."""
    rng = np.random.default_rng(nx + 1000 * views)
    sino = rng.standard_normal((views, bins)).astype(np.float32)
    offset = float(np.float32(0.4))
    f2 = fbp.FBP2D(0)
    if kind == "fan":
        far = 3.0 * nx if nx > 1 else 200.0  # a tile's 32 pixels lie in front of the source
        sod, sdd, det = far, far + 2.0 * nx, 2.4 * nx
        g = fbp.Geometry.cone(sod, sdd - sod, det, float(nx), turns, offset)
    else:
        sod, sdd, det = 0.0, 0.0, 1.3 * nx
        g = fbp.Geometry.parallel(det, float(nx), turns, offset)
    img = f2.project_backward(sino, g, (nx, nz))
    assert np.array_equal(img, f2.project_backward(sino, g, (nx, nz)))
    c = dict(nx=nx, ny=1, nz=nz, vox=1.0, nu=bins, nv=1, nviews=views, du=float(np.float32(det)) / bins, dv=1.0,
             span=2 * math.pi * float(np.float32(turns)), offset=offset, sod=float(np.float32(sod)),
             sdd=float(np.float32(sod)) + float(np.float32(sdd - sod)))
    ref = (oracle.bp_fan2d if kind == "fan" else oracle.bp_parallel2d)(sino.astype(np.float64), c)
    assert relative_rmse(img, ref) < TOL_BP2D


# FP32 transform of n <= 4096 samples and its inverse: rounding 6e-8 per stage,
# independent over 2 log2 n = 24 stages (3e-7), on white noise whose filtered
# rows are of its own scale.
TOL_ROWS = 1e-6


@pytest.mark.parametrize("rows", [1, 2, 7, 700])
@pytest.mark.parametrize("m", [1, 2, 3, 5, 9, 17, 33, 64, 65, 128, 129, 257, 511, 513, 1000, 1025, 2049, 4096])
def test_fft_filter_every_length(fbp, oracle, m, rows):
    """Each register-phase split of the row transform, padded and unpadded
    rows, odd row counts (an unpaired last row), fewer and more pairs than the
    GPU has SMs; the allocation-free entry point gives the same bits."""
    import torch
    x = np.random.default_rng(m * 10 + rows).standard_normal((rows, m)).astype(np.float32)
    filt = m % 4
    f2 = fbp.FBP2D(0)
    got = f2.apply_filter(x.copy(), filt)
    ref = oracle.filter_rows(x.astype(np.float64), filt)
    assert relative_rmse(got, ref) < TOL_ROWS
    d = torch.as_tensor(x, device="cuda")
    assert fbp.library().fbp2d_filter_sinogram_noalloc(d.data_ptr(), m, rows, filt, 0.0, 0.0, 0, None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy(), got)


@pytest.mark.parametrize("layout", ["projections", "sinograms"])
@pytest.mark.parametrize("u,v,n", [(70, 1, 5), (70, 2, 3), (130, 3, 5), (301, 4, 6), (9, 5, 7), (600, 7, 3)])
def test_fft_filter_pair_layout(fbp, oracle, layout, u, v, n):
    """Rows filtered into the pair layout (a pair inside one view, across two
    views, at a view's edges) and back, with log and weight in the load."""
    rng = np.random.default_rng(u)
    counts = (rng.random((n, v, u)) * 900 + 100).astype(np.float32)
    s = fbp.FBP3D(0)
    sod, odd, width = 200.0, 100.0, 150.0
    if layout == "projections":
        s.upload_projections(counts)
        s.log_normalize_projections(1000.0)
        s.apply_fdk_weights_to_projections(sod, odd, width)
        s.apply_filter_to_projections(1)
        got = s.download_projections()
    else:
        s.upload_sinograms(np.ascontiguousarray(counts.transpose(1, 0, 2)))
        s.log_normalize_sinograms(1000.0)
        s.apply_fdk_weights_to_sinograms(sod, odd, width)
        s.apply_filter_to_sinograms(1)
        got = s.download_sinograms(np.empty((v, n, u), np.float32)).transpose(1, 0, 2)
    s.ctx.close()
    p = oracle.fdk_weight(oracle.log_normalize(counts.astype(np.float64), 1000.0), sod + odd, width / u, width / u)
    assert relative_rmse(got, oracle.filter_rows(p, 1)) < TOL_ROWS


# Backprojection of white noise (no filter): the sum over views is as
# incoherent as the taps' errors, so the relative error is one tap's. FP32:
# position rounding, as TOL_BP2D. 24-bit views: 16 significant bits, 2^-17 RMS
# a value, four values a tap. FP16 views: 2^-12 a value (2.4e-4).
TOL_BP = {"FP32": 3e-5, "MIXED24": 5e-5, "MIXED": 4e-4}


def _noise_bp(fbp, oracle, c, precision, variant, tile=0, sinograms=False):
    rng = np.random.default_rng(c["nx"] + 7 * c["nviews"])
    proj = rng.standard_normal((c["nviews"], c["nv"], c["nu"])).astype(np.float32)
    s = fbp.FBP3D(0)
    s.set_clip_after_backprojection(False)
    s.set_precision(getattr(fbp.Precision, precision))
    s.set_backprojector(getattr(fbp.Backprojector, variant))
    if tile:
        s.set_symmetric_tile(tile)
    args = (c["sod"], c["sdd"] - c["sod"], c["nu"] * c["du"], c["nx"] * c["vox"], c["span"] / (2 * math.pi),
            c["nx"], c["ny"], c["offset"])
    if sinograms:
        s.upload_sinograms(np.ascontiguousarray(proj.transpose(1, 0, 2)))
        s.project_backward_cone_fdk_from_sinograms(*args)
    else:
        s.upload_projections(proj)
        s.project_backward_cone_fdk_from_projections(*args)
    got, info = s.read_volume(), s.last_backprojection()
    s.ctx.close()
    ref = oracle.bp_cone(proj.astype(np.float64), c)
    return relative_rmse(got, ref), info


@pytest.mark.parametrize("precision", ["FP32", "MIXED", "MIXED24"])
@pytest.mark.parametrize("tile", [0, 8, 16])
@pytest.mark.parametrize("n,ny,views,du", [(32, 2, 4, 1.5), (32, 25, 8, 2.25), (64, 13, 12, 1.5), (64, 47, 20, 0.75),
                                           (96, 24, 36, 0.5), (64, 12, 132, 1.5)])
def test_symmetric_tile_heights(fbp, oracle, precision, tile, n, ny, views, du):
    """Every tile height the symmetric kernel has, volumes that end inside a
    tile, walks shorter than a block of quads, rows that advance by less than
    one, about one, two and three per voxel."""
    c = dict(sod=3.0 * n, sdd=4.5 * n, du=du, dv=du, span=2 * math.pi, offset=0.0, nu=int(2.4 * n / du), nv=int(2 * n / du),
             nviews=views, nx=n, ny=ny, nz=n, vox=1.0)
    err, info = _noise_bp(fbp, oracle, c, precision, "SYMMETRIC", tile, sinograms=ny == 13)
    assert info["kernel"] == "symmetric" and (not tile or info["tile_ny"] == tile)
    assert err < TOL_BP[precision]


def test_symmetric_fp32_unstaged_windows(fbp, oracle):
    """High magnification: windows wider than the widest box (128 elements) are
    gathered from global memory (zero outside the detector)."""
    c = dict(sod=120.0, sdd=360.0, du=0.6, dv=0.6, span=2 * math.pi, offset=0.0, nu=330, nv=300, nviews=48, nx=64,
             ny=40, nz=64, vox=1.0)
    err, info = _noise_bp(fbp, oracle, c, "FP32", "SYMMETRIC")
    assert info["kernel"] == "symmetric" and info["layout"] == "quads32"
    assert info["box"][0] > 128
    assert err < TOL_BP["FP32"]


@pytest.mark.parametrize("precision", ["FP32", "MIXED", "MIXED24"])
@pytest.mark.parametrize("variant", ["GENERIC", "GENERIC_Y8"])
@pytest.mark.parametrize("n,ny,views,du", [(17, 1, 3, 1.5), (33, 25, 9, 2.25), (50, 47, 21, 0.75), (30, 16, 35, 0.5)])
def test_generic_row_steps(fbp, oracle, precision, variant, n, ny, views, du):
    """The generic kernel's march for every row step, off the symmetric sizes."""
    c = dict(sod=3.0 * n, sdd=4.5 * n, du=du, dv=du, span=2 * math.pi, offset=0.0, nu=int(2.4 * n / du), nv=int(2 * n / du),
             nviews=views, nx=n, ny=ny, nz=n, vox=1.0)
    err, info = _noise_bp(fbp, oracle, c, precision, variant, sinograms=ny == 47)
    assert info["kernel"] == (variant.lower() if ny > 1 else "generic")  # one slice: the 2D tile
    assert err < TOL_BP["FP32" if precision == "MIXED24" else precision]


@pytest.mark.parametrize("precision", ["FP32", "MIXED", "MIXED24"])
@pytest.mark.parametrize("beam,n,ny,views,turns,du", [
    ("cone", 50, 9, 8, 1.0, 1.5), ("cone", 49, 20, 12, 1.0, 2.25), ("cone", 33, 17, 4, 1.0, 0.75),     # quarter turns
    ("cone", 64, 33, 10, 1.0, 1.5), ("cone", 49, 18, 14, 1.0, 0.5), ("cone", 17, 5, 2, 1.0, 2.25),      # half turns
    ("cone", 40, 16, 9, 1.0, 1.5), ("cone", 40, 16, 12, 0.25, 1.5), ("cone", 40, 7, 12, 2.0, 1.5),      # none
    ("parallel", 64, 24, 10, 0.5, 1.0), ("parallel", 49, 11, 66, 0.5, 0.8), ("parallel", 50, 8, 2, 0.5, 1.3),
    ("parallel", 48, 16, 11, 0.5, 1.0), ("parallel", 49, 17, 13, 1.0, 0.7), ("parallel", 50, 40, 6, 0.3, 1.0),
    ("parallel", 50, 21, 8, 1.0, 1.0), ("parallel", 17, 3, 6, 1.0, 1.0)])
def test_orbits_of_the_generic_geometries(fbp, oracle, precision, beam, n, ny, views, turns, du):
    """Two- and four-fold orbits off the symmetric kernel's sizes, mirrored
    ones of parallel beam, odd sizes with their centre column or middle row,
    and view sets without any, on white noise with a start angle, through
    projections and sinograms."""
    offset = float(np.float32(0.7))
    c = dict(du=du, dv=du, span=2 * math.pi * float(np.float32(turns)), offset=offset, nu=int(2.0 * n / du),
             nv=int(1.6 * n / du), nviews=views, nx=n, ny=ny, nz=n, vox=1.0)
    if beam == "cone":
        err, info = _noise_bp(fbp, oracle, dict(c, sod=4.0 * n, sdd=6.0 * n), precision, "AUTO", sinograms=n % 2 == 1)
    else:
        proj = np.random.default_rng(n + views).standard_normal((views, c["nv"], c["nu"])).astype(np.float32)
        s = fbp.FBP3D(0)
        s.set_clip_after_backprojection(False)
        s.set_precision(getattr(fbp.Precision, precision))
        if n % 2:
            s.upload_sinograms(np.ascontiguousarray(proj.transpose(1, 0, 2)))
            s.project_backward_parallel_from_sinograms(turns, n, ny, offset)
        else:
            s.upload_projections(proj)
            s.project_backward_parallel_from_projections(turns, n, ny, offset)
        got, info = s.read_volume(), s.last_backprojection()
        s.ctx.close()
        ref = oracle.bp_parallel3d(proj.astype(np.float64), dict(c, du=n / c["nu"], dv=ny / c["nv"]))
        err = relative_rmse(got, ref)
    assert info["kernel"] == "generic" and info["layout"] == ("pairs16" if precision == "MIXED" else "rows32")
    assert err < TOL_BP["FP32" if precision == "MIXED24" else precision]


@pytest.mark.parametrize("precision", ["FP32", "MIXED"])
@pytest.mark.parametrize("views", [24, 26])
def test_orbit_unstaged_windows(fbp, oracle, precision, views):
    """Windows wider than the widest box of the four- and two-view elements."""
    c = dict(sod=110.0, sdd=330.0, du=0.84, dv=0.84, span=2 * math.pi, offset=0.0, nu=260, nv=150, nviews=views, nx=50,
             ny=16, nz=50, vox=1.0)
    err, info = _noise_bp(fbp, oracle, c, precision, "AUTO")
    assert info["kernel"] == "generic" and info["box"][0] > 128
    assert err < TOL_BP[precision]


@pytest.mark.parametrize("n,ny", [(64, 16), (120, 64)])
def test_no_room_for_the_interleaved_copy(fbp, oracle, n, ny):
    """FP32 views that fill the device: the interleaved copy (as many bytes
    again) does not fit, and the plain kernel runs on the rows themselves."""
    views, nu, nv = 128, 1024, 256
    c = dict(sod=300.0, sdd=400.0, du=1.0, dv=1.0, span=2 * math.pi, offset=0.0, nu=nu, nv=nv, nviews=views, nx=n,
             ny=ny, nz=n, vox=1.0)
    proj = np.random.default_rng(n).standard_normal((views, nv, nu)).astype(np.float32)
    s = fbp.FBP3D(0)
    s.set_clip_after_backprojection(False)
    s.set_precision(fbp.Precision.FP32)
    s.upload_projections(proj)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    spare = torch.empty(max(0, torch.cuda.mem_get_info()[0] - proj.nbytes // 2), dtype=torch.uint8, device="cuda")
    s.project_backward_cone_fdk_from_projections(300.0, 100.0, float(nu), float(n), 1.0, n, ny, 0.0)
    got, info = s.read_volume(), s.last_backprojection()
    s.ctx.close()
    del spare
    torch.cuda.empty_cache()
    assert info["kernel"] == "generic" and info["layout"] == "rows32" and info["tile_ny"] == 16
    assert relative_rmse(got, oracle.bp_cone(proj.astype(np.float64), c)) < TOL_BP["FP32"]


# Split-BF16 rows: 2^-17 of white noise through the filter, as for the row
# tests of the tensor-core filter (0.7e-5 to 1.3e-5 in an emulation).
TOL_TOEPLITZ = 5e-5


@pytest.mark.parametrize("views,nv,m", [
    (1, 1, 64), (1, 3, 65), (1, 127, 95), (2, 64, 96), (3, 43, 97), (5, 26, 127), (1, 131, 128), (7, 11, 129),  # one tile
    (1, 130, 191), (1, 130, 193), (2, 65, 255), (1, 129, 256), (1, 129, 257), (2, 61, 320), (1, 200, 383),
    (2, 67, 385), (1, 77, 511), (1, 77, 513), (1, 130, 769), (3, 9, 1151), (1, 9, 2048), (1, 9, 2049), (1, 5, 8191),
    (3, 1601, 70), (7, 1601, 640), (7, 1601, 641), (3, 1601, 650), (3, 1601, 2100),   # rows a warp, staged or not
    (9, 8601, 130), (2, 20001, 700)])                                                     # more than one chunk
@pytest.mark.parametrize("pre", [False, True])
def test_toeplitz_rows_and_widths(fbp, oracle, views, nv, m, pre):
    """The tensor-core row filter at the edges of its tiles, K blocks, rows a
    warp and chunks, with and without the fused log and weight."""
    rng = np.random.default_rng(m + nv)
    proj = (np.exp(-0.5 * rng.random((views, nv, m))) * 1e4 if pre else rng.standard_normal((views, nv, m)) + 2.0)
    proj = proj.astype(np.float32)
    s = fbp.FBP3D(0)
    s.set_filter_impl(fbp.FilterImpl.TOEPLITZ)
    s.upload_projections(proj)
    ref = proj.astype(np.float64)
    if pre:
        s.log_normalize_projections(1e4)
        s.apply_fdk_weights_to_projections(3.0 * m, 1.0 * m, float(m))
        ref = oracle.fdk_weight(-np.log(ref / 1e4), 4.0 * m, 1.0, 1.0)
    s.apply_filter_to_projections(0)
    got = s.download_projections()
    s.ctx.close()
    ref = oracle.filter_rows(ref.reshape(-1, m), 0).reshape(proj.shape)
    assert relative_rmse(got, ref) < TOL_TOEPLITZ


def test_more_view_groups_than_the_packer_takes(fbp):
    """65540 views without a turn (one group each) run on the plain kernel."""
    views, n, ny = 65540, 208, 8
    sino = np.random.default_rng(3).standard_normal((2, views, 32)).astype(np.float32)
    out = []
    for variant in (fbp.Backprojector.AUTO, fbp.Backprojector.GENERIC_Y8):
        s = fbp.FBP3D(0)
        s.set_clip_after_backprojection(False)
        s.set_precision(fbp.Precision.FP32)
        s.set_backprojector(variant)
        s.upload_sinograms(sino)
        s.project_backward_parallel_from_sinograms(0.3, n, ny, 0.1)
        out.append(s.read_volume())
        s.ctx.close()
    assert relative_rmse(out[0], out[1]) < TOL_BP["FP32"]
