"""The reference Blinn-Phong shader's float pairs against its FP64 form, both on
the GPU: colours are diffuse + ks * (N.H)^s, and weights above 1e6 take FP64,
so twice the colour at K = 6e5 less the colour at 2 K is the diffuse term.

Tolerance: each colour is rounded to float once (2^-24 of it; the one at K
counts twice), the pairs may add a quarter of a rounding (2^-26), and the
diffuse term (the Lambertian shader, no larger than 1.2) is within the
pipeline's colour tolerance of 1e-5.

Scenes: a sphere, a terrain, and a ground triangle that starts in front of the
camera and ends 10^7 units away, where what the weights' errors are worth grows
with the far vertices' distance.
"""
import numpy as np
import pytest

from edxraster_gb300 import renderer as R
from edxraster_gb300 import scenes

pytestmark = pytest.mark.gpu
K = 6.0e5


def ground(width=160, height=90, far=1.0e7):
    """One triangle in the plane y = -1, the far vertex last; the light mirrors
    the line of sight at the bottom of the image, a little off."""
    pos = np.array([[0.0, -1.0, 0.3], [-far, -1.0, far], [far, -1.0, far]], np.float32)
    mesh = scenes.Mesh(pos, np.tile(np.array([0.0, 1.0, 0.0], np.float32), (3, 1)), np.full((3, 3), 0.5, np.float32),
                       np.zeros((3, 2), np.float32), np.array([[0, 1, 2]], np.uint32))
    view = scenes.View(width, height, np.eye(4, dtype=np.float32), scenes.perspective_lh(70.0, width / height, 0.1, 1e8),
                       scenes.raster_matrix(width, height), np.array([0.1, 1.0, 1.9], np.float32))
    return scenes.Scene("ground", mesh, view)


SCENES = {"sphere": lambda: scenes.sphere_scene(160, 90, seed=4), "terrain": lambda: scenes.terrain_scene(96, 160, 90, seed=5),
          "ground": ground}


def render(sc, shader, ks, shininess):
    sc.view.shader, sc.view.ks, sc.view.shininess = shader, ks, shininess
    r = R.Renderer()
    r.Initialize(sc.view.width, sc.view.height)
    R.configure(r, sc.view)
    r.RenderMesh(sc.mesh)
    color, _, tid = r.ReadOutputs()
    r.close()
    return color[..., 0].astype(np.float64), tid != 0xFFFFFFFF


@pytest.mark.parametrize("shininess", [1.0, 32.0, 200.0, 256.0, 2000.0, 2048.0, 2049.0, 65536.0])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_pairs_are_as_good_as_fp64(cuda_lib, name, sign, shininess):
    sc = SCENES[name]()
    diffuse, covered = render(sc, scenes.SHADER_LAMBERTIAN, 0.0, 1.0)
    once, _ = render(sc, scenes.SHADER_BLINN_PHONG_REFERENCE, sign * K, shininess)
    twice, _ = render(sc, scenes.SHADER_BLINN_PHONG_REFERENCE, sign * 2 * K, shininess)
    assert np.array_equal(np.isnan(once), np.isnan(twice))
    ok = covered & ~np.isnan(twice)
    off = np.abs(2 * once - twice - diffuse)[ok]
    bound = ((2.0 ** -24 + 2.0 ** -26) * (2 * np.abs(once) + np.abs(twice)) + 1e-5)[ok]
    if name == "ground" or shininess <= 32.0:
        assert (np.abs(twice[ok]) > 10.0).any()  # the specular term shows
    assert (off <= bound).all(), (off / bound).max()
