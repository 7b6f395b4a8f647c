"""Few big triangles among many small ones: the unsorted bin list holds their
entries.  It is 32 stripes of equal size, so no stripe may take many of the big
triangles' entries alone, nor more slots than there are entries: the frame
renders in the fixed scratch of edxr_render_noalloc (24,576 slots a stripe),
and in a growing renderer (32,768 at first) without being rendered again.

Two kinds of big triangles, one per SM less two, so that up to 32 warps share
each: about 100 pixels wide (16 reference tiles, work for one warp), and thin
ones from corner to corner of the image (1,024 reference tiles, some five
entries for each of 32 warps).
"""
import numpy as np
import pytest

from edxraster_gb300 import renderer as R
from edxraster_gb300 import scenes
from test_zz_no_alloc import call_noalloc

pytestmark = pytest.mark.gpu
SIDE = 1024


def scene(kind, nbig, nsmall, seed=3):
    """nsmall triangles of 4 entries each on the corners of four tiles, shared
    vertices, then nbig big ones in front of them."""
    rng = np.random.default_rng(seed)
    corner = 16.0 * np.stack(np.meshgrid(np.arange(1, 64), np.arange(1, 64), indexing="xy"), -1).reshape(-1, 1, 2)
    ang = np.array([0.0, 2 * np.pi / 3, 4 * np.pi / 3])
    unit = np.stack([np.cos(ang), np.sin(ang)], -1)  # clockwise on screen (y down): front faces
    small = corner + 4.0 * unit
    if kind == "wide":
        big = rng.uniform(100.0, SIDE - 100.0, (nbig, 1, 2)) + 58.0 * unit
    else:
        shift = rng.uniform(0.0, 12.0, (nbig, 1, 1))
        big = np.array([[8.0, 12.0], [8.0, 8.0], [1008.0, 1008.0]]) + shift
    (ax, ay), (bx, by) = (big[:, 1] - big[:, 0]).T, (big[:, 2] - big[:, 0]).T
    assert (ax * by > ay * bx).all()
    px = np.concatenate([small, big])
    w = np.concatenate([np.full(len(small), 2.0), rng.uniform(1.0, 1.5, nbig)])[:, None, None]
    ndc = np.stack([px[..., 0] / SIDE * 2.0 - 1.0, 1.0 - px[..., 1] / SIDE * 2.0], -1)
    pos = np.concatenate([ndc * w, np.broadcast_to(w, ndc.shape[:2] + (1,))], -1).reshape(-1, 3)
    tri = np.concatenate([np.arange(nsmall) % len(small), len(small) + np.arange(nbig)])
    idx = 3 * tri[:, None] + np.arange(3)
    nrm = np.tile(np.array([0.0, 0.0, -1.0], np.float32), (len(pos), 1))
    mesh = scenes.Mesh(pos.astype(np.float32), nrm, np.full((len(pos), 3), 0.5, np.float32),
                       np.zeros((len(pos), 2), np.float32), idx.astype(np.uint32))
    proj = np.array([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, scenes.STRESS_A, scenes.STRESS_B], [0, 0, 1, 0]], np.float32)
    view = scenes.View(SIDE, SIDE, np.eye(4, dtype=np.float32), proj, scenes.raster_matrix(SIDE, SIDE),
                       np.array([0.3, 0.5, -1.0], np.float32))
    return scenes.Scene(kind, mesh, view)


def big_triangles():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count - 2


def render(sc):
    r = R.Renderer()
    r.Initialize(SIDE, SIDE)
    R.configure(r, sc.view)
    r.RenderMesh(R.DeviceMesh.from_mesh(sc.mesh))
    out, stats = r.ReadOutputs(), r.Stats()
    r.close()
    return out, stats


@pytest.mark.parametrize("kind", ["wide", "thin"])
def test_fits_the_fixed_scratch(cuda_lib, kind):
    import torch
    nbig = big_triangles()
    sc = scene(kind, nbig, 65000)
    rc, (c1, d1, t1) = call_noalloc(cuda_lib, sc, torch.cuda.Stream())
    assert rc == 0, cuda_lib.edxr_last_error_string()
    (c0, d0, t0), _ = render(sc)
    seen = np.unique(t0)
    assert (seen < 65000).any() and ((seen >= 65000) & (seen < 65000 + nbig)).any()
    assert np.array_equal(t1, t0)
    assert np.array_equal(d1.view(np.uint32), d0.view(np.uint32))
    assert np.array_equal(c1.view(np.uint32), c0.view(np.uint32))


@pytest.mark.parametrize("kind", ["wide", "thin"])
def test_first_frame_is_not_rendered_again(cuda_lib, kind):
    nsmall = 120000
    _, stats = render(scene(kind, big_triangles(), nsmall))
    assert stats.bin_entries > 4 * nsmall
    assert stats.rerenders == 0
