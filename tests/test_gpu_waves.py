"""The streaming wavefront's waves against the oracle, bit for bit, at the sizes and in the forms where
their queues can go wrong: one pixel, a block of the resolve stage and one more, path and shadow rays in
one launch or each in its own, shading sorted or not, a slot's next sample started ahead of the adaptive
decision, and the tail taking over with shadow rays in flight."""
import pytest

from verion_gb300 import pack, scenes
from verion_gb300.backend import Integrator, Renderer
from verion_gb300.readback import Adaptive

from .test_gpu_parity import assert_same, oracle_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (16, 16), (257, 1), (33, 31)])
@pytest.mark.parametrize("form", ["merged", "separate", "unsorted", "tail"])
def test_waves_match_the_oracle(gpu_ctx, size, form):
    p = pack.pack(scenes.many_spheres(spheres=4, sphere_n=15, grid=48, hdri=(64, 32)))
    adaptive = Adaptive(threshold=0.05, min_spp=2)
    r = Renderer(gpu_ctx, p)
    r.set_integrator(Integrator.WAVEFRONT)
    r.set_max_depth(16)
    r.set_adaptive(adaptive)
    r.set_accum_precision(32)
    r.set_stage_timing(form == "separate")
    r.set_material_sort(form != "unsorted")
    r.set_stream_tail(100 if form == "tail" else 0)
    acc = r.new_accumulation(*size)
    for n in (1, 4, 3):
        r.accumulate(acc, n)
    ref = oracle_render(p, *size, 8, depth=16, adaptive=adaptive)
    assert_same(acc.sums(), ref.sums, f"{form} sums")
    assert_same(acc.raw_stats(), ref.stats, f"{form} adaptive statistics")


@pytest.mark.parametrize("size", [(1, 1), (16, 16), (257, 1), (33, 31)])
@pytest.mark.parametrize("form", ["merged", "separate", "tail"])
def test_split_waves_match_the_oracle(gpu_ctx, size, form):
    # The lighting split's parts and light slots: the deferred light sample carries its share of each.
    p = pack.pack(scenes.many_spheres(spheres=4, sphere_n=15, grid=48, hdri=(64, 32)))
    adaptive = Adaptive(threshold=0.05, min_spp=2)
    r = Renderer(gpu_ctx, p)
    r.set_integrator(Integrator.WAVEFRONT)
    r.set_max_depth(16)
    r.set_adaptive(adaptive)
    r.set_accum_precision(32)
    r.set_stage_timing(form == "separate")
    r.set_stream_tail(100 if form == "tail" else 0)
    acc = r.new_accumulation(*size, True)
    for n in (1, 4, 3):
        r.accumulate(acc, n)
    ref = oracle_render(p, *size, 8, depth=16, adaptive=adaptive, lighting=True)
    assert_same(acc.sums(), ref.sums, f"{form} sums")
    assert_same(acc.raw_lighting(), ref.lighting, f"{form} lighting split")
