"""Interpolation's backward on both sides of its rule on triangles per pixel (up to
four channels or with derivatives: by columns from six pixels per triangle on):
the launch of several views against a view at a time, which is always by pixels.
Sums in another order: within 1e-5 of the largest."""
import pytest
import torch

from tests.test_gpu_walk import test_interpolate_backward as _against_single_views

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C, diff, n, res", [
    (3, None, 64, (91, 93)), (1, None, 66, (250, 257)), (4, None, 33, (250, 257)), (5, [1, 4], 66, (250, 257))])
@pytest.mark.parametrize("per_triangle", [5.99, 6.01])
def test_either_side(cuda_lib, monkeypatch, C, diff, n, res, per_triangle):
    import tests.test_gpu_walk as T
    views = T._views

    def more_triangles(n, res, detail=3):
        """The same views with degenerate triangles after the mesh's own."""
        pos, tri, rast, db = views(n, res, detail)
        extra = int(res[0] * res[1] / per_triangle) - len(tri)
        return pos, torch.cat([tri, tri.new_zeros((extra, 3))]), rast, db

    monkeypatch.setattr(T, "_views", more_triangles)
    _against_single_views(cuda_lib, C, diff, n, res, False)
