"""Meshes without normals or albedo shade out of line; the image is that of the
mesh with the default values written out (albedo 1, normal 0)."""
import numpy as np
import pytest

from edxraster_gb300 import renderer as R
from edxraster_gb300 import scenes

pytestmark = pytest.mark.gpu


def render(view, msaa, **arrays):
    r = R.Renderer()
    r.Initialize(view.width, view.height)
    R.configure(r, view)
    r.SetMSAAMode(msaa)
    r.RenderMesh(R.DeviceMesh(**arrays))
    out = r.ReadOutputs()
    r.close()
    return out


@pytest.mark.parametrize("msaa", [0, 2])
@pytest.mark.parametrize("shader", [0, 2, 3])
@pytest.mark.parametrize("size", [(64, 48), (640, 360)])
def test_missing_arrays_take_their_defaults(cuda_lib, size, shader, msaa):
    import torch
    sc = scenes.small_random_scene(11, *size, ntris=300)  # clipped triangles too
    sc.view.shader = shader
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    pos, idx, nrm, alb = (t(a) for a in (sc.mesh.positions, sc.mesh.indices.astype(np.int32), sc.mesh.normals, sc.mesh.albedo))
    pairs = [(dict(normals=nrm), dict(normals=nrm, albedo=torch.ones_like(alb))),
             (dict(albedo=alb), dict(normals=torch.zeros_like(nrm), albedo=alb))]
    for missing, written in pairs:
        a, b = (render(sc.view, msaa, positions=pos, indices=idx, **k) for k in (missing, written))
        assert (a[2] != 0xFFFFFFFF).any()
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")
