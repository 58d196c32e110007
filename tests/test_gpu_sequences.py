"""Sequences of calls that the entry points accept before an accumulation's first sample: options changed after a call
that added no sample, or that failed, give what a fresh accumulation with the later options gives, bit for bit."""
import numpy as np
import pytest

from verion_gb300 import pack, scenes
from verion_gb300.backend import Cache, Error, Integrator, Renderer
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
