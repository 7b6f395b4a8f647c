"""Batched passes of small meshes with shared vertices: a warp's 32 vertices
cross several frames, and the search for a warp's first frame (32 frames
compared at a time) runs at the edges of its rounds.  Every frame must be the
bytes of its own plain render."""
import numpy as np
import pytest

from edxraster_gb300 import renderer as R
from edxraster_gb300 import scenes

pytestmark = pytest.mark.gpu

W, H = 40, 24


def meshes():
    tri = scenes.Mesh(positions=np.float32([[-1, -1, 0], [1, -1, 0], [0, 1, 0]]),
                      normals=np.float32([[0, 0, -1]] * 3), albedo=np.float32([[0.8, 0.4, 0.2]] * 3),
                      uvs=np.zeros((3, 2), np.float32), indices=np.uint32([[0, 2, 1]]))
    return [tri] + [scenes.uv_sphere(s, t) for s, t in ((6, 8), (9, 13), (17, 6))]


@pytest.mark.parametrize("frames", [2, 31, 32, 33, 65, 1024, 1025])
def test_each_frame_is_its_plain_render(cuda_lib, frames):
    ms = meshes()
    assert all(m.nt for m in ms)
    views = scenes.orbit_views(frames, W, H, seed=frames)
    rng = np.random.default_rng(frames)
    for v in views:
        v.mesh = int(rng.integers(len(ms)))
    dms = [R.DeviceMesh.from_mesh(m) for m in ms]
    r = R.Renderer()
    r.Initialize(W, H)
    r.RenderBatched(dms, views, W, H)
    color, depth, tid = r.ReadBatchOutputs(0, frames, W, H)
    for i in sorted({0, 1, frames // 2, frames - 2, frames - 1, *rng.integers(frames, size=24).tolist()}):
        R.configure(r, views[i])
        r.RenderMesh(dms[views[i].mesh])
        o = r.ReadOutputs()
        assert np.array_equal(tid[i], o[2])
        assert np.array_equal(depth[i].view(np.uint32), o[1].view(np.uint32))
        assert np.array_equal(color[i], o[0])
    assert (tid != 0xFFFFFFFF).any()
    r.close()
