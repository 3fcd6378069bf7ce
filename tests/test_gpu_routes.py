"""Calls whose kernel goes by the volume's size, the detector windows or the room left: what one call leaves on a context
must not show in the next, and what one kernel does not take another one does."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from conftest import relative_rmse

pytestmark = pytest.mark.gpu

# FP32 backprojection of ramp-filtered white noise: position rounding moves a
# linear tap of unit-variance samples by ~2e-5, independent over the views.
TOL_BP = 3e-5


def _solver(fbp, precision="FP32", tune=False, variant=None):
    s = fbp.FBP3D(0)
    s.set_clip_after_backprojection(False)
    s.set_precision(getattr(fbp.Precision, precision))
    s.set_autotune(tune)
    if variant:
        s.set_backprojector(getattr(fbp.Backprojector, variant))
    return s


def _noise(seed, views, rows, cols):
    return np.random.default_rng(seed).standard_normal((views, rows, cols)).astype(np.float32)


# --------------------------------------------------------------- views packed by an earlier call
@pytest.mark.parametrize("precision", ["FP32", "MIXED", "MIXED24"])
@pytest.mark.parametrize("n,ny,views,slabs", [(100, 97, 180, 2), (65, 321, 36, 4), (100, 97, 182, 2)])
def test_slabs_of_another_call(fbp, precision, n, ny, views, slabs):
    """Slabs of one volume whose heights choose different kernels (48 slices
    of 100 x 100 run on the rows, 49 on interleaved views): on a context that
    has reconstructed other projections, the same bits as on a new one."""
    g = fbp.Geometry.cone(3.0 * n, 1.5 * n, 2.2 * n, float(n), 1.0, 0.0)
    a, b = (_noise(seed, views, ny, int(1.4 * n)) for seed in (1, 2))
    s = _solver(fbp, precision)
    first = s.reconstruct_fdk_to_host(a, g, 0, n, ny, slabs=slabs)
    again = s.reconstruct_fdk_to_host(b, g, 0, n, ny, slabs=slabs)
    back = s.reconstruct_fdk_to_host(a, g, 0, n, ny, slabs=slabs)
    s.ctx.close()
    t = _solver(fbp, precision)
    alone = t.reconstruct_fdk_to_host(b, g, 0, n, ny, slabs=slabs)
    t.ctx.close()
    assert np.array_equal(again, alone)
    assert np.array_equal(back, first) and not np.array_equal(first, again)


@pytest.mark.parametrize("to_host", [False, True])
def test_tuned_call_after_another(fbp, to_host):
    """The tuner times a slab of 48 slices (on the rows), the whole height of
    64 may take interleaved views: never those of the call before."""
    n, ny, views = 100, 64, 180
    cols = 140
    s = _solver(fbp, tune=True)
    got = {}
    for name, seed, scale in (("other", 1, 2.0), ("this", 2, 2.2)):  # another geometry: tuned anew
        g = fbp.Geometry.cone(3.0 * n, 1.5 * n, scale * n, float(n), 1.0, 0.0)
        proj = _noise(seed, views, 97, cols)
        s.set_autotune(name == "this")
        if name == "other" or not to_host:
            s.upload_projections(proj)
            s.reconstruct_fdk(g, 0, n, 97 if name == "other" else ny)
            got[name] = s.read_volume()
        else:
            got[name] = s.reconstruct_fdk_to_host(proj, g, 0, n, ny, slabs=1)
    s.ctx.close()
    t = _solver(fbp)
    ref = t.reconstruct_fdk_to_host(proj, g, 0, n, ny, slabs=1)
    t.ctx.close()
    assert relative_rmse(got["this"], ref) < TOL_BP


def test_slabs_after_a_packing_that_found_no_room(fbp):
    """Each slab would take interleaved views, and the device has no room for
    them: every slab runs on the rows, also where an earlier call has packed
    (smaller) views."""
    n, ny, views, rows, cols = 120, 192, 128, 256, 1024
    g = fbp.Geometry.cone(300.0, 100.0, 700.0, float(n), 1.0, 0.0)
    small, big = _noise(1, 8, rows, cols), _noise(2, views, rows, cols)
    s = _solver(fbp)
    s.reconstruct_fdk_to_host(small, g, 0, n, ny, slabs=2)
    s.upload_projections(big)  # the stack is allocated: what follows asks for the packed views alone
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    spare = torch.empty(max(0, torch.cuda.mem_get_info()[0] - big.nbytes // 2), dtype=torch.uint8, device="cuda")
    got = s.reconstruct_fdk_to_host(big, g, 0, n, ny, slabs=4)
    layout = s.last_backprojection()["layout"]
    s.ctx.close()
    del spare
    torch.cuda.empty_cache()
    t = _solver(fbp)
    ref = t.reconstruct_fdk_to_host(big, g, 0, n, ny, slabs=1)
    t.ctx.close()
    assert layout == "rows32"
    assert relative_rmse(got, ref) < TOL_BP


# --------------------------------------------------------------- windows near the kernels' limits
@pytest.mark.parametrize("precision,views,cols,rows", [
    ("FP32", 180, 217, 217), ("FP32", 182, 217, 217),                           # 67 x 87 samples a 16-high tile
    ("MIXED24", 180, 300, 300), ("MIXED", 180, 300, 300), ("MIXED", 182, 300, 300)])  # 91 x 119
def test_windows_too_large_for_an_estimate(fbp, oracle, precision, views, cols, rows):
    """Volumes off the symmetric sizes whose 8- or 12-high tiles' windows,
    taken to 16 voxels, would not fit twice in half an SM, while the plain
    kernel's do."""
    n, ny, width, sod, odd = 100, 100, 193.33, 150.0, 50.0
    c = dict(sod=sod, sdd=sod + odd, du=float(np.float32(width)) / cols, dv=float(np.float32(width)) / cols,
             span=2 * math.pi, offset=0.0, nu=cols, nv=rows, nviews=views, nx=n, ny=ny, nz=n, vox=1.0)
    proj = _noise(5, views, rows, cols)
    s = _solver(fbp, precision)
    s.upload_projections(proj)
    s.apply_filter_to_projections(0)
    filtered = s.download_projections()
    s.project_backward_cone_fdk_from_projections(sod, odd, width, float(n), 1.0, n, ny, 0.0)
    got = s.read_volume()
    s.ctx.close()
    ref = oracle.bp_cone(filtered.astype(np.float64), c)
    # FP16 views: 2^-12 of a value (2.4e-4)
    assert relative_rmse(got, ref) < (4e-4 if precision == "MIXED" else TOL_BP)


@pytest.mark.parametrize("variant,height,rows,ny", [("AUTO", 8, 271, 16), ("GENERIC", 8, 271, 16), ("AUTO", 8, 542, 32),
                                                    ("GENERIC", 16, 270, 16), ("GENERIC_Y8", 1, 582, 16),
                                                    ("SYMMETRIC", 8, 582, 16)])
def test_windows_of_257_rows(fbp, oracle, variant, height, rows, ny):
    """Parallel beam with 17 detector rows a voxel (36 for tiles of eight):
    the filtered rows of a tile are one more than a staged box holds."""
    n, views, turns = (64, 92, 1.0) if variant == "SYMMETRIC" else (48, 91, 0.5)
    cols = n // 2 if variant == "SYMMETRIC" else n  # narrow enough for the ring to hold the whole height
    c = dict(du=n / cols, dv=ny / rows, span=2 * math.pi * turns, offset=0.0, nu=cols, nv=rows, nviews=views, nx=n, ny=ny,
             nz=n, vox=1.0)
    s = _solver(fbp, variant=variant)
    s.upload_projections(_noise(6, views, rows, cols))
    s.apply_filter_to_projections(0)
    filtered = s.download_projections()
    s.project_backward_parallel_from_projections(turns, n, ny, 0.0)
    got, info = s.read_volume(), s.last_backprojection()
    s.ctx.close()
    # a voxel moves the position by 17 to 36 rows, whose rounding (2 ulp below 512) is 6e-5 of a row
    assert relative_rmse(got, oracle.bp_parallel3d(filtered.astype(np.float64), c)) < 6e-5
    assert info["tile_ny"] == height


# --------------------------------------------------------------- rotational orbits off the symmetric sizes
FOUR, TWO = {"FP32": "quads32", "MIXED24": "quads32", "MIXED": "quads_pairs16"}, \
            {"FP32": "duos32", "MIXED24": "duos32", "MIXED": "duos_pairs16"}
FOUR_HIGH = dict(FOUR, MIXED="pairs16")  # 588 plain tiles: four waves, as many as FP16 orbits eight high would take
# 24-bit views exist for the symmetric kernel only: FP32 here. FP16 views: 2^-12 a value (2.4e-4).
TOL_ORBIT = {"FP32": TOL_BP, "MIXED24": TOL_BP, "MIXED": 4e-4}


def _orbit_case(fbp, oracle, precision, beam, n, ny, views, turns, cols, rows, sinograms=False, scale=2.0):
    offset = float(np.float32(0.7))
    proj = _noise(n + views, views, rows, cols)
    s = _solver(fbp, precision)
    width = scale * n if beam == "cone" else float(n)
    c = dict(span=2 * math.pi * float(np.float32(turns)), offset=offset, nu=cols, nv=rows, nviews=views, nx=n, ny=ny,
             nz=n, vox=1.0, du=float(np.float32(width)) / cols)
    what = "sinograms" if sinograms else "projections"
    getattr(s, "upload_" + what)(np.ascontiguousarray(proj.transpose(1, 0, 2)) if sinograms else proj)
    if beam == "cone":
        c.update(dv=c["du"], sod=4.0 * n, sdd=6.0 * n)
        getattr(s, "project_backward_cone_fdk_from_" + what)(4.0 * n, 2.0 * n, width, float(n), turns, n, ny, offset)
        ref = oracle.bp_cone(proj.astype(np.float64), c)
    else:
        c.update(dv=ny / rows)
        getattr(s, "project_backward_parallel_from_" + what)(turns, n, ny, offset)
        ref = oracle.bp_parallel3d(proj.astype(np.float64), c)
    got, info = s.read_volume(), s.last_backprojection()
    s.ctx.close()
    return relative_rmse(got, ref), info


@pytest.mark.parametrize("precision", ["FP32", "MIXED", "MIXED24"])
@pytest.mark.parametrize("beam,n,ny,views,turns,cols,rows,layout,height", [
    # quarter turns: whole and odd sizes, one group, more turns, 12-high tiles
    ("cone", 100, 49, 12, 1.0, 130, 80, FOUR, 8), ("cone", 97, 50, 4, 1.0, 90, 70, FOUR, 8),
    ("cone", 111, 60, 36, 5.0, 300, 200, FOUR, 8), ("cone", 97, 177, 8, 1.0, 130, 240, FOUR_HIGH, 12),
    # half turns, the other way round, an odd number of them
    ("cone", 100, 49, 14, 1.0, 130, 80, TWO, 16), ("cone", 97, 53, 2, 1.0, 90, 70, TWO, 16),
    ("cone", 99, 64, 12, -1.0, 260, 180, TWO, 16), ("cone", 112, 50, 10, 3.0, 130, 80, TWO, 16),
    # parallel beam: half a turn (mirrored quarter turns), half turns, the half-turned voxel in the same view
    ("parallel", 100, 49, 10, 0.5, 130, 49, FOUR, 8), ("parallel", 97, 51, 66, 0.5, 110, 77, FOUR, 8),
    ("parallel", 113, 50, 2, 0.5, 100, 40, FOUR, 8), ("parallel", 100, 49, 12, 1.0, 130, 60, FOUR, 8),
    ("parallel", 97, 52, 14, 1.0, 130, 60, TWO, 16), ("parallel", 100, 50, 11, 0.5, 111, 49, TWO, 16),
    ("parallel", 97, 49, 13, 1.0, 140, 90, TWO, 16), ("parallel", 98, 49, 9, 0.3, 120, 49, TWO, 16)])
def test_orbits(fbp, oracle, precision, beam, n, ny, views, turns, cols, rows, layout, height):
    """Volumes large enough for rotational orbits: four and two slots, mirrored
    ones, odd sizes with their centre column or middle row, volumes that end
    inside a tile, with a start angle, through projections and sinograms."""
    err, info = _orbit_case(fbp, oracle, precision, beam, n, ny, views, turns, cols, rows, sinograms=n % 2 == 1)
    plain = layout[precision] == "pairs16"
    assert info["kernel"] == ("generic" if plain else "orbits") and info["layout"] == layout[precision]
    assert info["tile_ny"] == (16 if plain else height)
    assert err < TOL_ORBIT[precision]


@pytest.mark.parametrize("precision", ["FP32", "MIXED"])
@pytest.mark.parametrize("views,layout", [(10, FOUR), (11, TWO)])
def test_orbits_unstaged_windows(fbp, oracle, precision, views, layout):
    """Windows wider than the widest box (128 elements) are gathered from the
    views in global memory (zero outside the detector)."""
    err, info = _orbit_case(fbp, oracle, precision, "parallel", 100, 49, views, 0.5, 660, 49)
    assert info["kernel"] == "orbits" and info["layout"] == layout[precision] and info["box"][0] > 128
    assert err < TOL_ORBIT[precision]


# --------------------------------------------------------------- kernels asked for and tuned
@pytest.mark.parametrize("precision,layout", [("FP32", "rows32"), ("MIXED24", "rows32"), ("MIXED", "pairs16")])
@pytest.mark.parametrize("variant,height", [("GENERIC", 16), ("GENERIC_Y8", 8)])
def test_the_generic_kernel_when_asked_for(fbp, oracle, precision, layout, variant, height):
    """GENERIC is the plain kernel, also where AUTO takes orbits."""
    n, ny, views, cols, rows = 100, 49, 12, 130, 80
    proj = _noise(8, views, rows, cols)
    c = dict(span=2 * math.pi, offset=0.0, nu=cols, nv=rows, nviews=views, nx=n, ny=ny, nz=n, vox=1.0, du=200.0 / cols,
             dv=200.0 / cols, sod=400.0, sdd=600.0)
    info = {}
    for v in (variant, "AUTO"):
        s = _solver(fbp, precision, variant=v)
        s.upload_projections(proj)
        s.project_backward_cone_fdk_from_projections(400.0, 200.0, 200.0, float(n), 1.0, n, ny, 0.0)
        got, info[v] = s.read_volume(), s.last_backprojection()
        s.ctx.close()
        assert relative_rmse(got, oracle.bp_cone(proj.astype(np.float64), c)) < TOL_ORBIT[precision]
    assert info[variant]["kernel"] == variant.lower() and info[variant]["layout"] == layout
    assert info[variant]["tile_ny"] == height and info["AUTO"]["kernel"] == "orbits"


@pytest.mark.parametrize("precision", ["FP32", "MIXED"])
@pytest.mark.parametrize("n,ny", [(100, 64), (100, 100), (96, 200), (50, 40)])
def test_the_tuned_kernel_is_the_one_that_runs(fbp, tmp_path, precision, n, ny):
    """The shape recorded in the tuner's cache file is what the whole volume
    runs on, although the tuner's slab is 48 slices high."""
    s = _solver(fbp, precision, tune=True)
    s.set_autotune_cache(tmp_path / "tune.txt")
    s.upload_projections(_noise(9, 60, 90, 130))
    s.project_backward_cone_fdk_from_projections(4.0 * n, 2.0 * n, 2.0 * n, float(n), 1.0, n, ny, 0.0)
    s.synchronize()
    info = s.last_backprojection()
    s.ctx.close()
    variant, quad_ny = (int(x) for x in (tmp_path / "tune.txt").read_text().split("|")[1].split()[:2])
    assert info["kernel"] == {1: "generic", 2: "symmetric", 3: "generic_y8", 4: "orbits"}[variant]
    assert not quad_ny or info["tile_ny"] == quad_ny


# The march's tolerance: position rounding (2 ulp of an index below 512, 6e-5
# voxel) times the slope between random voxels in [0, 1], over ~800 samples of mean 0.5.
def test_forward_of_a_large_volume_keeps_nothing(fbp, oracle):
    """A volume whose bordered copy is larger than what a context keeps (256
    MB): the device has its memory back after the call."""
    n, views = 420, 2
    vol = np.random.default_rng(15).random((n, n, n), np.float32)
    s = _solver(fbp)
    s.generate_blank_volume(n, n, n)
    s.write_volume_data(vol)
    args = (4.0 * n, 2.0 * n, 1.5 * n, float(n), 1.0, views, 0.3)
    s.project_forward_cone_to_projections(*args[:4], 1.0, 1, 0.3)  # modules, stack
    s.project_forward_cone_to_projections(*args)
    got = s.download_projections()
    torch.cuda.synchronize()
    in_use, free = s.memory_in_use(), torch.cuda.mem_get_info()[0]
    s.ctx.close()
    torch.cuda.synchronize()
    freed = torch.cuda.mem_get_info()[0] - free
    volume, stack = vol.nbytes, got.nbytes
    assert in_use < volume + stack + (8 << 20)
    assert freed < volume + stack + (32 << 20)
    c = dict(vox=1.0, du=1.5, dv=1.5, span=2 * math.pi, offset=np.float32(0.3), sod=4.0 * n, sdd=6.0 * n, nu=n, nv=n,
             nviews=views)
    assert relative_rmse(got, oracle.forward_project(vol, c, cone=True)) < 1e-5


# --------------------------------------------------------------- 2D slices
@pytest.mark.parametrize("kind", ["fan", "parallel"])
@pytest.mark.parametrize("bins", [2_100_001, 40_000_003])
def test_bp2d_wide_detectors(fbp, oracle, kind, bins):
    """Rows far wider than the image: the columns that it sees lie around a
    detector centre that FP32 no longer counts exactly (2^24 and more)."""
    n, views = 40, 3 if bins > 1 << 24 else 8
    det = 1.5 * bins
    sino = np.zeros((views, bins), np.float32)
    mid = slice(bins // 2 - 400, bins // 2 + 400)
    sino[:, mid] = np.random.default_rng(11).standard_normal((views, 800)).astype(np.float32)
    f2 = fbp.FBP2D(0)
    if kind == "fan":
        sod, sdd = 200.0, 300.0
        img = f2.project_backward(sino, fbp.Geometry.cone(sod, sdd - sod, det, 1.0 * n, 1.0, 0.1), (n, n))
    else:
        sod = sdd = 0.0
        img = f2.project_backward(sino, fbp.Geometry.parallel(det, 1.0 * n, 0.5, 0.1), (n, n))
    # the oracle sees the middle of the detector alone
    c = dict(nx=n, ny=1, nz=n, vox=1.0, nu=800 + bins % 2, nv=1, nviews=views, du=float(np.float32(det)) / bins, dv=1.0,
             span=2 * math.pi * (1.0 if kind == "fan" else 0.5), offset=float(np.float32(0.1)), sod=sod, sdd=sdd)
    part = np.ascontiguousarray(sino[:, bins // 2 - 400:bins // 2 + 400 + bins % 2]).astype(np.float64)
    ref = (oracle.bp_fan2d if kind == "fan" else oracle.bp_parallel2d)(part, c)
    assert relative_rmse(img, ref) < TOL_BP


# --------------------------------------------------------------- forward projection
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.float32(3e38)])
def test_forward_of_an_infinite_voxel(fbp, value):
    """Rays through an infinite (or the largest) voxel sum to infinity, as the
    weighted sum of the neighbours does: no NaN from a difference."""
    n, views = 24, 5
    vol = np.full((n, n, n), -1.0 if value > 0 else 1.0, np.float32)
    vol[11, 12, 13] = value
    s = fbp.FBP3D(0)
    s.generate_blank_volume(n, n, n)
    s.write_volume_data(vol)
    s.project_forward_cone_to_projections(4.0 * n, 2.0 * n, 1.5 * n, float(n), 1.0, views, 0.3)
    got = s.download_projections()
    s.ctx.close()
    assert not np.isnan(got).any()
    assert (np.abs(got) > 1e37).any(axis=(1, 2)).all() and (np.abs(got) < 1e3).any(axis=(1, 2)).all()


# --------------------------------------------------------------- FP32 sums
# K values near c added up, each addition rounded once: an error of ulp(S) /
# sqrt(12) for the running sum S, independent from one to the next. Summed over
# S = c, 2c .. 1024 c that is 4.2e-7 (1024 c a power of two) to 4.8e-7 (half way to
# the next) of the sum. Two roundings an addition: 5.9e-7 to 6.8e-7. The values
# scatter by 3%, which an error of 2e-5 of a sample in the tap's position turns
# into less than 1e-8 of the sum.
TOL_SUM = 5.3e-7


def _near_one(seed, *shape):
    return (1.0 + 0.05 * (2.0 * np.random.default_rng(seed).random(shape) - 1.0)).astype(np.float32)


@pytest.mark.parametrize("kernel,n,ny,views,rows", [
    ("symmetric", 64, 20, 1024, 60), ("symmetric", 160, 128, 1024, 260), ("orbits", 100, 49, 1024, 120),
    ("orbits", 100, 49, 1022, 120), ("generic", 50, 24, 1023, 70)])
def test_fp32_sums_round_once(fbp, oracle, kernel, n, ny, views, rows):
    cols = int(2.4 * n)
    c = dict(sod=4.0 * n, sdd=6.0 * n, du=1.2, dv=1.2, span=2 * math.pi, offset=0.0, nu=cols, nv=rows, nviews=views,
             nx=n, ny=ny, nz=n, vox=1.0)
    c["du"] = c["dv"] = float(np.float32(1.2 * cols)) / cols
    proj = _near_one(12, views, rows, cols)
    s = _solver(fbp)
    s.upload_projections(proj)
    s.project_backward_cone_fdk_from_projections(4.0 * n, 2.0 * n, 1.2 * cols, float(n), 1.0, n, ny, 0.0)
    got, info = s.read_volume(), s.last_backprojection()
    s.ctx.close()
    m = slice(n // 4, n - n // 4)  # inside the field of view
    ref = oracle.bp_cone(proj.astype(np.float64), c)[m, :, m]
    assert info["kernel"] == kernel
    assert relative_rmse(got[m, :, m], ref) < TOL_SUM


@pytest.mark.parametrize("kind,n,views,turns", [("fan", 600, 1023, 1.0), ("fan", 960, 1024, 1.0),
                                                ("parallel", 600, 1023, 0.5)])
def test_2d_sums_round_once(fbp, oracle, kind, n, views, turns):
    bins = int(2.4 * n)
    sino = _near_one(13, views, bins)
    det = 1.0 * bins if kind == "fan" else 1.5 * n
    f2 = fbp.FBP2D(0)
    if kind == "fan":
        sod, sdd = 4.0 * n, 5.0 * n
        img = f2.project_backward(sino, fbp.Geometry.cone(sod, n, det, float(n), turns, 0.0), (n, n))
    else:
        sod = sdd = 0.0
        img = f2.project_backward(sino, fbp.Geometry.parallel(det, float(n), turns, 0.0), (n, n))
    c = dict(nx=n, ny=1, nz=n, vox=1.0, nu=bins, nv=1, nviews=views, du=float(np.float32(det)) / bins, dv=1.0,
             span=2 * math.pi * turns, offset=0.0, sod=sod, sdd=sdd)
    ref = (oracle.bp_fan2d if kind == "fan" else oracle.bp_parallel2d)(sino.astype(np.float64), c)
    m = slice(n // 4, n - n // 4)
    assert relative_rmse(img.reshape(n, n)[m, m], np.asarray(ref).reshape(n, n)[m, m]) < TOL_SUM


# --------------------------------------------------------------- weights
@pytest.mark.parametrize("what", ["weights", "FFT", "TOEPLITZ"])
def test_fdk_weights_of_tiny_lengths(fbp, oracle, what):
    """Lengths in a unit that makes their squares subnormal (9e-40, with steps
    of 1.6e-6 of that: 8e-7 of the weight)."""
    views, rows, cols = 3, 5, 96
    sod, odd, width = 2e-20, 1e-20, 4e-20
    proj = _near_one(14, views, rows, cols)
    s = _solver(fbp)
    s.upload_projections(proj)
    s.apply_fdk_weights_to_projections(sod, odd, width)
    f = lambda x: float(np.float32(x))  # noqa: E731
    ref = oracle.fdk_weight(proj.astype(np.float64), f(sod) + f(odd), f(width) / cols, f(width) / cols)
    if what != "weights":
        s.set_filter_impl(getattr(fbp.FilterImpl, what))
        s.apply_filter_to_projections(0)
        ref = oracle.filter_rows(ref.reshape(-1, cols), 0).reshape(proj.shape)
    got = s.download_projections()
    s.ctx.close()
    # the filter's output is a tenth of its input here; split rows: 2^-17 of a value
    assert relative_rmse(got, ref) < {"weights": 2e-6, "FFT": 2e-5, "TOEPLITZ": 1e-4}[what]


@pytest.mark.parametrize("kind", ["fan", "parallel"])
def test_bp2d_wide_images(fbp, oracle, kind):
    """An image of one long row that spans 17 million detector columns: the
    windows at its ends lie further from the detector's centre than FP32 counts."""
    n, views, bins = 1_600_001, 2, 17_000_001
    sino = np.random.default_rng(18).standard_normal((views, bins)).astype(np.float32)
    det = 0.1 * bins if kind == "parallel" else 0.15 * bins
    f2 = fbp.FBP2D(0)
    if kind == "fan":
        sod, sdd = 4.0 * n, 6.0 * n
        img = f2.project_backward(sino, fbp.Geometry.cone(sod, sdd - sod, det, float(n), 1.0, 1.5), (n, 1))
    else:
        sod = sdd = 0.0
        img = f2.project_backward(sino, fbp.Geometry.parallel(det, float(n), 0.5, 1.5), (n, 1))
    c = dict(nx=n, ny=1, nz=1, vox=1.0, nu=bins, nv=1, nviews=views, du=float(np.float32(det)) / bins, dv=1.0,
             span=2 * math.pi * (1.0 if kind == "fan" else 0.5), offset=float(np.float32(1.5)),
             sod=float(np.float32(sod)), sdd=float(np.float32(sod)) + float(np.float32(sdd - sod)))
    ref = (oracle.bp_fan2d if kind == "fan" else oracle.bp_parallel2d)(sino.astype(np.float64), c)
    assert relative_rmse(img, ref) < TOL_BP


@pytest.mark.parametrize("kind", ["fan", "parallel"])
def test_bp2d_without_room_for_the_packed_rows(fbp, oracle, kind):
    """Rows that nearly fill the device: the packed copy does not fit, and the
    rows are read where they are (detector narrower than the image, odd sizes)."""
    n, nz, views, bins = 41, 37, 4100, 6001
    sino = np.zeros((views, bins), np.float32)
    sino[:, 2900:3101] = np.random.default_rng(16).standard_normal((views, 201))
    sino[:, 0] = sino[:, -1] = 1.0
    det = 0.2 * bins
    d = torch.as_tensor(sino, device="cuda")
    out = torch.empty((nz, n), device="cuda")
    f2 = fbp.FBP2D(0)
    if kind == "fan":
        sod, sdd = 400.0, 500.0
        g = fbp.Geometry.cone(sod, sdd - sod, det, float(n), 1.0, 0.1)
    else:
        sod = sdd = 0.0
        g = fbp.Geometry.parallel(det, float(n), 0.5, 0.1)
    f2.project_backward(d[:40, :400].contiguous(), g, (n, nz))  # modules, angles' buffer
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    spare = torch.empty(max(0, torch.cuda.mem_get_info()[0] - sino.nbytes // 2), dtype=torch.uint8, device="cuda")
    try:
        f2.project_backward(d, g, (n, nz), out=out)
        got = out.cpu().numpy()
    finally:
        f2.ctx.close()
        del spare, d, out
        torch.cuda.empty_cache()
    c = dict(nx=n, ny=1, nz=nz, vox=1.0, nu=bins, nv=1, nviews=views, du=float(np.float32(det)) / bins, dv=1.0,
             span=2 * math.pi * (1.0 if kind == "fan" else 0.5), offset=float(np.float32(0.1)), sod=sod, sdd=sdd)
    ref = (oracle.bp_fan2d if kind == "fan" else oracle.bp_parallel2d)(sino.astype(np.float64), c)
    assert relative_rmse(got, ref) < TOL_BP


# --------------------------------------------------------------- contexts
def test_contexts_report_their_own_errors(fbp):
    """More contexts than a shared page has error words: each reports its own
    device error (a voxel behind the source), once, and no other's; words that
    closed contexts gave back serve new ones."""
    def project(s, sod):
        s.upload_projections(np.ones((8, 24, 24), np.float32))
        s.project_backward_cone_fdk_from_projections(sod, 60.0, 24.0, 16.0, 1.0, 16, 8, 0.0)

    def expect(s, bad):
        if bad:
            with pytest.raises(fbp.FBPError) as e:
                s.synchronize()
            assert e.value.status == -7
        s.synchronize()

    solvers = [_solver(fbp) for _ in range(70)]
    for turn in range(2):
        bad = {3, 40, 66, 69} if turn == 0 else {0, 65}
        for i, s in enumerate(solvers):
            project(s, 2.0 if i in bad else 60.0)
        for i, s in reversed(list(enumerate(solvers))):
            expect(s, i in bad)
        for i in range(0, 70, 3):
            solvers[i].ctx.close()
            solvers[i] = _solver(fbp)
    for s in solvers:
        s.ctx.close()
