"""Several samples per pixel, where a block of warps shares a tile: triangles
smaller than a pixel (few samples covered, rarely the centre), tiles of many
more entries than one work item, several winners in one pixel, and depths that
are zeros of either sign (the key keeps no sign of zero).  Winners and depth
bits equal the oracle's exactly."""
import numpy as np
import pytest

from edxraster_gb300 import renderer as R
from edxraster_gb300 import scenes
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def check(sc, lg, depth_func):
    r = R.Renderer()
    r.Initialize(sc.view.width, sc.view.height)
    sc.view.depth_func = depth_func
    R.configure(r, sc.view)
    r.SetMSAAMode(lg)
    r.RenderMesh(sc.mesh)
    color, depth, tid = r.ReadOutputs()
    r.close()
    o = pyoracle.render_oracle(sc.mesh, sc.view, depth_func=depth_func, msaa_log2=lg)
    assert np.array_equal(tid, o["id"])
    assert np.array_equal(depth.view(np.uint32), o["depth"].view(np.uint32))
    # a sample's colour is 8 bits: FP32 and FP64 shading may round to neighbouring bytes
    assert np.abs(color.astype(np.float64) - o["color"]).max() <= 1.0 / 255.0 + 1e-6
    return tid


@pytest.mark.parametrize("lg", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("width,height,ntris,max_area", [(33, 17, 6000, 3.0), (129, 79, 3000, 40.0), (16, 16, 1, 900.0)])
def test_small_and_dense(cuda_lib, lg, width, height, ntris, max_area):
    sc = scenes.stress_scene(ntris, width, height, seed=50 + lg, min_area=0.02, max_area=max_area, dup_fraction=0.1,
                             backface_fraction=0.0)
    check(sc, lg, scenes.DEPTH_LESS if lg & 1 else scenes.DEPTH_LEQUAL)


@pytest.mark.parametrize("lg", [1, 3])
def test_zero_depths_keep_their_sign(cuda_lib, lg):
    sc = scenes.stress_scene(400, 64, 48, seed=9, max_area=300.0)
    # clip z = (0 x + 0 y - 0 w) - 0: +0 or -0 by the signs of x and y
    sc.view.proj[2] = np.array([0.0, 0.0, -0.0, -0.0], np.float32)
    check(sc, lg, scenes.DEPTH_LEQUAL)
