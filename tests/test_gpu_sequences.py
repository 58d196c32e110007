"""Sequences of calls that the entry points accept before an accumulation's first sample: options changed after a call
that added no sample, or that failed, give what a fresh accumulation with the later options gives, bit for bit."""
import time

import numpy as np
import pytest

from verion_gb300 import pack, scenes
from verion_gb300.backend import VG_ERR_TIMEOUT, Cache, Error, Integrator, Renderer
from verion_gb300.readback import Restir

from .test_gpu_parity import assert_same, oracle_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", [0, 1 << 18])
@pytest.mark.parametrize("first", ["no samples", "failed"])
def test_restir_switched_off_before_the_first_sample_of_a_split(gpu_ctx, first, tail):
    # The first call makes the wavefront's buffers without the deferred shadows' planes, the second needs them.
    p = pack.pack(scenes.many_spheres(spheres=4, sphere_n=15, grid=48, hdri=(64, 32)))
    w, h, spp = 65, 47, 3
    r = Renderer(gpu_ctx, p)
    r.set_integrator(Integrator.WAVEFRONT)
    r.set_accum_precision(32)
    r.set_stream_tail(tail)
    r.set_restir(Restir(di=True))
    acc = r.new_accumulation(w, h, True)
    if first == "failed":
        cache = Cache(gpu_ctx, bounds=r.bounds(), levels=2, log2_entries=8, base_resolution=4, max_resolution=8)
        r.set_cache(cache)
        with pytest.raises(Error):
            r.accumulate(acc, 1)  # (a cache takes neither the split nor ReSTIR)
        r.set_cache(None)
    else:
        r.accumulate(acc, 0)
    r.set_restir(None)
    r.accumulate(acc, spp)
    ref = oracle_render(p, w, h, spp, lighting=True)
    assert_same(acc.sums(), ref.sums, "sums")
    assert_same(acc.raw_lighting(), ref.lighting, "lighting split")


@pytest.mark.parametrize("form", ["megakernel", "one launch", "waves"])
def test_a_deadline_passed_returns_at_once_and_leaves_the_context_usable(gpu_ctx, form, monkeypatch):
    # The limit is far below what the call's GPU work takes, which ends by itself afterwards.
    p = pack.pack(scenes.many_spheres(spheres=16, sphere_n=21, grid=160, hdri=(64, 32)))
    r = Renderer(gpu_ctx, p)
    r.set_integrator(Integrator.MEGAKERNEL if form == "megakernel" else Integrator.WAVEFRONT)
    r.set_accum_precision(32)
    r.set_max_depth(16)
    w, h, spp = (960, 540, 64) if form == "waves" else (512, 512, 192)
    r.set_stream_tail(0 if form == "waves" else 1 << 18)
    small = r.new_accumulation(33, 31)
    r.accumulate(small, 2)
    want = small.sums()

    full = r.new_accumulation(w, h)
    r.accumulate(full, 1)
    t = time.perf_counter()
    r.accumulate(full, spp)
    ordinary = time.perf_counter() - t
    assert ordinary > 0.02
    monkeypatch.setenv("VG_TIMEOUT_S", "0.0001")
    t = time.perf_counter()
    with pytest.raises(Error) as e:
        r.accumulate(full, spp)
    passed = time.perf_counter() - t
    monkeypatch.delenv("VG_TIMEOUT_S")
    assert e.value.status == VG_ERR_TIMEOUT
    assert passed < ordinary / 2
    # With the abandoned work still in flight, calls that take the same pools give what they gave.
    for _ in range(3):
        acc = r.new_accumulation(33, 31)
        r.accumulate(acc, 2)
        assert np.array_equal(acc.sums(), want)


def test_tail_threshold_of_the_inline_form_stays_at_its_own_most(gpu_ctx):
    # A path per thread from at most 32,768 slots, whatever the block wavefront's threshold is set to.
    p = pack.pack(scenes.many_spheres(spheres=4, sphere_n=15, grid=48, hdri=(64, 32)))

    def waves(threshold):
        r = Renderer(gpu_ctx, p)
        r.set_integrator(Integrator.WAVEFRONT)
        r.set_deferred_shadows(False)
        if threshold is not None:
            r.set_stream_tail(threshold)
        acc = r.new_accumulation(320, 300)
        r.accumulate(acc, 2)
        return acc.last_waves()

    assert waves(1 << 18) == waves(None)


def test_autotune_tries_what_its_frame_reaches(gpu_ctx):
    p = pack.pack(scenes.many_spheres(spheres=4, sphere_n=15, grid=48, hdri=(64, 32)))
    r = Renderer(gpu_ctx, p)
    t = r.autotune(96, 54, 1, bvh=False)
    if t["deferred_shadows"] and t["stream_tail"] >= 96 * 54 and not t["graph_waves"]:
        # One launch: itself, shadows, three tails, the graph, two refills, two step counts.
        assert t["trials"] == 10
        assert t["dynamic_fetch"] and t["material_sort"] and not t["coop_triangles"]
    # ReSTIR GI traces its light samples inside shade: the threshold tried and reported is that form's.
    r = Renderer(gpu_ctx, p)
    r.set_restir(Restir(di=True, gi=True))
    assert r.autotune(96, 54, 1, bvh=False)["stream_tail"] in (0, 8192, 32768)
