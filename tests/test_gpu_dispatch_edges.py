"""GPU kernels at the sizes where their dispatch or tiling can go wrong, against the FP64 oracle."""
from __future__ import annotations

import math

import numpy as np
import pytest

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
