"""The raster kernel with one warp per tile and with 4 or 8 (frames of few
tiles): the same bytes on both sides of each size at which the number of warps
changes, and the oracle's winners and depths.  Tiles hold more entries than a
work item, large and wrapping regions, and none at all (the empty tiles' list).
"""
import numpy as np
import pytest

from edxraster_gb300 import renderer as R
from edxraster_gb300 import scenes
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def sides():
    """Tile grids at the rule's borders (8 * tiles = 27 * SMs, tiles = 30 * SMs) and between them."""
    sms = 152
    grids = [(1, 1)]
    for tiles in (27 * sms // 8, 12 * sms, 30 * sms):
        h = int(tiles ** 0.5)
        grids += [(tiles // h, h), (tiles // h + 1, h)]
    return grids


@pytest.mark.parametrize("depth_func", [scenes.DEPTH_LESS, scenes.DEPTH_LEQUAL])
@pytest.mark.parametrize("tx,ty", sides())
def test_groups_render_the_same_bytes(cuda_lib, tx, ty, depth_func):
    w, h = 16 * tx - 3, 16 * ty - 5
    sc = scenes.stress_scene(8 * tx * ty + 600, w, h, seed=tx, max_area=2e3, dup_fraction=0.1)
    # crowd most triangles into a quarter of the screen: dense tiles there, empty ones elsewhere
    v = sc.mesh.positions.reshape(-1, 3, 3)
    v[: len(v) * 3 // 4, :, :2] = v[: len(v) * 3 // 4, :, :2] * 0.25 + 0.5 * v[: len(v) * 3 // 4, :, 2:]
    sc.view.depth_func = depth_func
    r = R.Renderer()
    r.Initialize(w, h)
    R.configure(r, sc.view)
    out = []
    for variant in (0, 1, 2):
        r.SetTuning({"raster_variant": variant})
        r.RenderMesh(sc.mesh)
        out.append(r.ReadOutputs())
    r.close()
    for o in out[1:]:
        assert all(np.array_equal(a.view(np.uint8), b.view(np.uint8)) for a, b in zip(out[0], o))
    o = pyoracle.render_oracle(sc.mesh, sc.view, depth_func=depth_func)
    assert np.array_equal(out[1][2], o["id"])
    assert np.array_equal(out[1][1].view(np.uint32), o["depth"].view(np.uint32))


@pytest.mark.parametrize("tx,ty,ntris", [(120, 76, 18240), (120, 76, 18241), (121, 76, 18240), (120, 76, 5)])
def test_few_triangles_over_many_tiles(cuda_lib, tx, ty, ntris):
    """Around tiles = 60 * SMs and triangles = 120 * SMs; most tiles hold a few large regions."""
    sc = scenes.stress_scene(ntris, 16 * tx, 16 * ty, seed=ntris, min_area=50.0, max_area=4e4)
    r = R.Renderer()
    r.Initialize(sc.view.width, sc.view.height)
    R.configure(r, sc.view)
    out = []
    for variant in (0, 1):
        r.SetTuning({"raster_variant": variant})
        r.RenderMesh(sc.mesh)
        out.append(r.ReadOutputs())
    r.close()
    assert all(np.array_equal(a.view(np.uint8), b.view(np.uint8)) for a, b in zip(*out))
    o = pyoracle.render_oracle(sc.mesh, sc.view, with_color=False)
    assert np.array_equal(out[1][2], o["id"])
