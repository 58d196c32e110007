"""Coverage of solid scenes where the beam walk is given up and rays are traced one by one: pixels much larger than the
triangles, against the same 16 rays followed one after the other (a renderer whose material table holds an unused
translucent material takes that form) bit for bit, in one launch and in more than one; and their cost."""
import time

import numpy as np
import pytest

from verion_gb300 import pack, scene as sc, scenes
from verion_gb300.backend import Renderer

pytestmark = pytest.mark.gpu


def detailed(spheres=16, sphere_n=21, grid=160):
    return scenes.many_spheres(spheres=spheres, sphere_n=sphere_n, grid=grid, hdri=(64, 32))


def pair(ctx, s):
    solid = Renderer(ctx, pack.pack(s))
    s.add_material(sc.BaseBsdf(opacity=0.5))
    return solid, Renderer(ctx, pack.pack(s))


# One pixel, a block's 16 x 8 and one more, a long row and a long column, and ordinary small images.
@pytest.mark.parametrize("size", [(1, 1), (16, 8), (17, 9), (1023, 1), (1, 1023), (72, 44), (256, 144)])
@pytest.mark.parametrize("where", ["usual", "above", "axis"])
def test_large_pixels_match_the_layered_form(gpu_ctx, size, where):
    s = detailed()
    if where == "above":
        s.camera = scenes.look_at((40.0, 90.0, 30.0), (0.0, 0.0, 0.0), fov=0.9)
    if where == "axis":
        s.camera = scenes.camera_at_z(14.0)
    solid, layered = pair(gpu_ctx, s)
    want = layered.render_aovs(*size).coverage
    assert np.array_equal(solid.render_aovs(*size).coverage, want)
    assert min(size) < 44 or want.max() > 0.0


def test_more_tiles_than_one_launch_takes(gpu_ctx):
    # 256 x 257 tiles of 16 x 8; a launch takes 65,536.
    solid, layered = pair(gpu_ctx, detailed(4, 15, 48))
    size = (4096, 2056)
    assert np.array_equal(solid.render_aovs(*size).coverage, layered.render_aovs(*size).coverage)


def test_few_large_pixels_cost_no_more_than_many_small_ones(gpu_ctx):
    # 16x16 and 256x144 pixels of the 110k-triangle scene: 0.43 and 0.51 ms; the walk without a bound took 7.4 and 0.9.
    r = Renderer(gpu_ctx, pack.pack(detailed()))

    def seconds(*size):
        best = 1.0
        for _ in range(8):
            t = time.perf_counter()
            r.render_aovs(*size)
            best = min(best, time.perf_counter() - t)
        return best

    assert seconds(16, 16) < 2.5 * seconds(256, 144)
