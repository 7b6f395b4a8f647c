"""Meshes without normals or albedo in frames that one warp per tile shades and
in multisampled ones: the image of the mesh with the default values written out
(albedo 1, normal 0), bit for bit."""
import numpy as np
import pytest

from edxraster_gb300 import scenes
from test_gpu_missing_attributes import render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("missing", ["albedo", "normals"])
@pytest.mark.parametrize("shader", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("msaa", [0, 1, 3, 5])
def test_large_frames_take_the_defaults(cuda_lib, msaa, shader, missing):
    import torch
    sc = scenes.terrain_scene(128, 1917, 1079)  # 8,160 tiles and 32,768 triangles, some clipped
    sc.view.shader, sc.view.depth_func = shader, msaa % 2
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    arrays = dict(positions=t(sc.mesh.positions), indices=t(sc.mesh.indices.astype(np.int32)),
                  normals=t(sc.mesh.normals), albedo=t(sc.mesh.albedo))
    written = dict(arrays, **{missing: torch.full_like(arrays[missing], 1.0 if missing == "albedo" else 0.0)})
    del arrays[missing]
    a, b = render(sc.view, msaa, **arrays), render(sc.view, msaa, **written)
    assert (a[2] != 0xFFFFFFFF).any()
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")
