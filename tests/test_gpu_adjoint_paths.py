"""The adjoint's two ways to sum per-vertex gradients (packed scratch array when
the pixels outnumber the vertices fourfold, else the caller's arrays directly)
and its spans of pixels (one to eight rows of 32 per warp, ragged ends, frames
that begin inside a span), against the FP64 reference; the arrays are added
to, and members that are NULL are skipped."""
import ctypes

import numpy as np
import pytest

from edxraster_gb300 import _lib
from edxraster_gb300 import renderer as R
from edxraster_gb300 import scenes

pytestmark = pytest.mark.gpu
REL_TOL = 1e-4  # gradient against FP64, relative L2 error per parameter group (as in test_gpu_adjoint.py)
NAMES = ("albedo", "normals", "positions", "light", "ks", "shininess")


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("nu,nviews,width,height", [
    (40, 1, 37, 29),     # one row a warp; fewer pixels than four times the vertices: added in place
    (64, 3, 61, 47),     # in place, frames begin inside spans
    (16, 5, 77, 51),     # packed
    (12, 40, 131, 97),   # packed, two rows a warp
    (12, 120, 129, 127),  # packed, eight rows a warp
])
def test_paths_match_fp64(cuda_lib, nu, nviews, width, height):
    import torch
    from oracle import adjoint_fp64
    mesh = scenes.torus(nu, max(8, nu // 2), 1.0, 0.35)
    rng = np.random.default_rng(nu)
    mesh.albedo = rng.uniform(0.1, 0.9, size=(mesh.nv, 3)).astype(np.float32)
    views = scenes.orbit_views(nviews, width, height, seed=nu + nviews)
    for v in views:
        v.light = views[0].light
    r = R.Renderer()
    r.Initialize(width, height)
    dm = R.DeviceMesh.from_mesh(mesh)
    r.RenderBatched([dm], views, width, height)
    ids = r.ReadBatchOutputs(0, nviews, width, height)[2]
    gen = torch.Generator(device="cuda").manual_seed(nu)
    gc = torch.randn((nviews, height, width, 4), dtype=torch.float32, device="cuda", generator=gen)
    abi = dm.abi()

    def run(skip=()):
        # arrays that already hold ones
        g = {k: torch.ones_like(getattr(dm, k)) for k in NAMES[:3]}
        g["light"], g["ks"], g["shininess"] = (torch.ones(n, device="cuda") for n in (3, 1, 1))
        torch.cuda.synchronize()
        grads = _lib.Grads(*[None if k in skip else g[k].data_ptr() for k in NAMES])
        _lib.check(r._lib.edxr_backward(r._h, ctypes.byref(abi), None, gc.data_ptr(), ctypes.byref(grads)))
        torch.cuda.synchronize()
        return {k: v.cpu().numpy().astype(np.float64) - 1.0 for k, v in g.items()}

    out = torch.empty_like(gc)
    _lib.check(r._lib.edxr_shade_visible(r._h, ctypes.byref(abi), None, out.data_ptr()))
    first, again, part = run(), run(), run(("normals", "ks"))
    r.close()
    ref = adjoint_fp64.reference_gradients(mesh, views[0].light, views[0].ks, views[0].shininess, views, ids,
                                           gc.cpu().numpy())
    covered = ids != 0xFFFFFFFF
    assert np.abs(out.cpu().numpy()[..., :3] - ref["color"]).max() <= 1e-5
    assert np.array_equal(out.cpu().numpy()[..., 3], covered.astype(np.float32))
    for got in (first, again):  # the scratch sums are zero again after a call
        errs = {k: rel(got[k].reshape(np.shape(ref[k])), ref[k]) for k in NAMES}
        assert all(e <= REL_TOL for e in errs.values()), errs
    assert not part["normals"].any() and not part["ks"].any()
    for k in ("albedo", "positions", "light", "shininess"):
        assert rel(part[k], first[k]) <= REL_TOL
