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
