"""Small windows with many triangles a tile: the raster kernel (several warps an
item, or one) is chosen on the device by the bin entries a tile.  Both sides of
the number of triangles from which the choice is made and of the density give
the bytes of one warp per item, and the oracle's winners and depths."""
import numpy as np
import pytest

from edxraster_gb300 import renderer as R
from edxraster_gb300 import scenes
from oracle import pyoracle

pytestmark = pytest.mark.gpu

W, H, TILES = 90, 60, 6 * 4


def bits(out):
    return [np.ascontiguousarray(x).view(np.uint32) for x in out]


@pytest.mark.parametrize("per_tile,dense", [(63, False), (64, False), (100, False), (3000, True)])
@pytest.mark.parametrize("depth_func", [scenes.DEPTH_LESS, scenes.DEPTH_LEQUAL])
def test_both_kernels_render_the_same_bytes(cuda_lib, per_tile, dense, depth_func):
    sc = scenes.stress_scene(per_tile * TILES, W, H, seed=per_tile, max_area=6e2 if dense else 60.0)
    sc.view.depth_func = depth_func
    r = R.Renderer()
    r.Initialize(W, H)
    R.configure(r, sc.view)
    outs = []
    for variant in (0, 1, 2):
        r.SetTuning({"raster_variant": variant})
        for _ in range(3):  # the last one replays a captured graph
            r.RenderMesh(sc.mesh)
        outs.append(r.ReadOutputs())
    assert (r.Stats().bin_entries > 640 * TILES) == dense
    r.close()
    for o in outs[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(bits(outs[0]), bits(o)))
    ref = pyoracle.render_oracle(sc.mesh, sc.view)
    assert np.array_equal(outs[1][2], ref["id"])
    assert np.array_equal(outs[1][1].view(np.uint32), ref["depth"].view(np.uint32))
