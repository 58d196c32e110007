"""Coverage of solid scenes, one beam walk per pixel, against the oracle's 16 rays, bit for bit: silhouettes
against the sky, a camera along an axis (directions that change sign within a pixel), one pixel and sizes
that are no multiple of a block's 16 x 8, and pixels wider than the scene's triangles."""
import numpy as np
import pytest

import oracle
from verion_gb300 import pack, scenes
from verion_gb300.backend import Renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (17, 9), (130, 75)])
@pytest.mark.parametrize("scene", ["spheres", "cornell", "cube", "far"])
def test_solid_coverage_matches_the_oracle(gpu_ctx, scene, size):
    if scene == "cornell":
        s = scenes.cornell()
    elif scene == "cube":
        s = scenes.white_furnace()
    else:
        s = scenes.many_spheres(spheres=4, sphere_n=15, grid=48, hdri=(64, 32))
        if scene == "far":
            s.camera = scenes.look_at((40.0, 90.0, 30.0), (0.0, 0.0, 0.0), fov=0.9)
    p = pack.pack(s)
    a = Renderer(gpu_ctx, p).render_aovs(*size)
    ad, oi, mi, cv = oracle.OracleScene(p).render_aovs(pack.camera_record(p.view, *size))
    assert np.array_equal(a.coverage, cv)
    assert np.array_equal(a.albedo, ad[:, :3]) and np.array_equal(a.depth, ad[:, 3])
    assert np.array_equal(a.object_id, oi) and np.array_equal(a.material_id, mi)
