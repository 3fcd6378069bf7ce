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
