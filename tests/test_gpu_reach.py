"""Kernels that small frames pass by: the waves of cached and of ReSTIR frames (with the default tail a frame of up to
262,144 pixels goes into one launch), and the refill of the block wavefront's slots (more pixels than its blocks hold
at a time)."""
import pytest

import oracle
from verion_gb300 import pack, scenes
from verion_gb300.backend import Cache, Integrator, Renderer
from verion_gb300.readback import Adaptive, Restir

from . import analytic
from .test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(48, 40), (65, 47)])
@pytest.mark.parametrize("form", ["waves", "unsorted", "tail"])
@pytest.mark.parametrize("scene", ["cornell", "zoo"])
def test_cached_waves_match_the_megakernel_cache(gpu_ctx, scene, form, size):
    # A cache that is not trained, one sample a frame: the same paths, queries and answers per pixel, bit for bit.
    p = pack.pack(scenes.cornell() if scene == "cornell" else analytic.feature_zoo())

    def run(integrator, tail):
        r = Renderer(gpu_ctx, p)
        r.set_integrator(integrator)
        cache = Cache(gpu_ctx, bounds=r.bounds(), seed=7)
        r.set_cache(cache, spread=0.01, train_paths=64, train_steps=0, train_batch=1024)
        r.set_cache_frame(1)
        r.set_stream_tail(tail)
        r.set_material_sort(form != "unsorted")
        acc = r.new_accumulation(*size)
        queries = 0
        for _ in range(3):
            r.accumulate(acc, 1)
            queries += acc.cache_stats().queries
        return acc.sums_f64(), queries

    want, wq = run(Integrator.MEGAKERNEL, 0)
    got, gq = run(Integrator.WAVEFRONT, 200 if form == "tail" else 0)
    assert gq == wq > 0
    assert_same(got, want, "sums")


def test_restir_waves_under_a_camera_pan_match_the_oracle(gpu_ctx):
    s = scenes.many_lights()
    p = pack.pack(s)
    w, h = 240, 135
    rs = Restir(di=True, gi=False, candidates=8, history=8)
    r = Renderer(gpu_ctx, p)
    r.set_accum_precision(32)
    r.set_integrator(Integrator.WAVEFRONT)
    r.set_stream_tail(0)
    r.set_restir(rs)
    acc = r.new_accumulation(w, h)
    o = oracle.OracleScene(p)
    ref = oracle.OracleAccumulation(w, h, restir=True)
    for k in range(4):
        eye = (0.3 * k, 6.0, 14.0)
        view = pack.View.new(scenes.look_at(eye, (0.0, 0.5, 0.0), fov=0.9))
        r.set_camera(view)
        r.accumulate(acc, 1)
        oracle.render(o, pack.base_params(p.info, view, (w, h), False, True, restir=rs), ref, 1)
        assert acc.last_waves() > 1
    assert_same(acc.sums(), ref.sums, "sums after the pan")


@pytest.mark.parametrize("scene", ["cornell", "zoo"])
@pytest.mark.parametrize("lighting", [False, True])
def test_refilled_slots_match_the_waves(gpu_ctx, scene, lighting):
    # 532,480 pixels; 152 blocks hold 3072 each, so most blocks' slots take a second pixel.
    p = pack.pack(scenes.cornell() if scene == "cornell" else analytic.feature_zoo())
    w, h = 1024, 520

    def run(integrator, tail):
        r = Renderer(gpu_ctx, p)
        r.set_integrator(integrator)
        r.set_stream_tail(tail)
        r.set_adaptive(Adaptive(threshold=0.05, min_spp=2))
        acc = r.new_accumulation(w, h, lighting)
        for n in (1, 3):
            r.accumulate(acc, n)
        return acc

    want = run(Integrator.WAVEFRONT, 0)
    assert want.last_waves() > 1
    for integrator, tail in ((Integrator.WAVEFRONT, 1 << 20), (Integrator.MEGAKERNEL, 0)):
        got = run(integrator, tail)
        assert_same(got.sums_f64(), want.sums_f64(), f"{integrator.name} sums")
        assert_same(got.raw_stats(), want.raw_stats(), f"{integrator.name} statistics")
        if lighting:
            assert_same(got.raw_lighting(), want.raw_lighting(), f"{integrator.name} lighting split")
