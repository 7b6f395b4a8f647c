"""BlinnPhongPixelShader as written (no clamp on N.H), shaded in float pairs
with FP64 for what leaves their plain range: within the pipeline's colour
tolerance (1e-5, as everywhere in these tests) of the oracle over exponents,
weights, back-lit pixels and normals of any length, with NaN where a negative
N.H has no power."""
import numpy as np
import pytest

from edxraster_gb300 import renderer as R
from edxraster_gb300 import scenes
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def check(sc):
    r = R.Renderer()
    r.Initialize(sc.view.width, sc.view.height)
    R.configure(r, sc.view)
    r.RenderMesh(sc.mesh)
    color, _, tid = r.ReadOutputs()
    r.close()
    o = pyoracle.render_oracle(sc.mesh, sc.view)
    assert np.array_equal(tid, o["id"])
    cov = tid != 0xFFFFFFFF
    got, want = color[cov, :3].astype(np.float64), np.asarray(o["color"], np.float64)[cov][:, :3]
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert ok.any() and np.abs(got[ok] - want[ok]).max() <= 1e-5


@pytest.mark.parametrize("ks,shininess", [(3.0, 200.0), (0.5, 32.0), (1.0, 0.0), (-2.0, 1.0), (3.0, 7.0), (2.0, 0.5),
                                          (2.0, 33.3)])
@pytest.mark.parametrize("scene", ["sphere", "terrain", "stress"])
def test_exponents_and_weights(cuda_lib, scene, ks, shininess):
    sc = {"sphere": lambda: scenes.sphere_scene(160, 90, seed=4), "terrain": lambda: scenes.terrain_scene(96, 160, 90, seed=5),
          "stress": lambda: scenes.stress_scene(3000, 160, 90, seed=6, max_area=2e3)}[scene]()
    sc.view.shader, sc.view.ks, sc.view.shininess = scenes.SHADER_BLINN_PHONG_REFERENCE, ks, shininess
    check(sc)


@pytest.mark.parametrize("scale", [1e-18, 1e-6, 1e12])
def test_normals_of_any_length(cuda_lib, scale):
    sc = scenes.terrain_scene(64, 96, 64, seed=2)
    sc.view.shader, sc.view.ks, sc.view.shininess = scenes.SHADER_BLINN_PHONG_REFERENCE, 3.0, 200.0
    sc.mesh.normals = (sc.mesh.normals * np.float32(scale)).astype(np.float32)
    check(sc)
