"""The cache's network over record counts around the encoding's and the scatter's edges (one record, a tile of 128
and one more or less, the last count of the four-thread encoding and the first of the other) against the CPU oracle."""
import numpy as np
import pytest

from oracle import nrc
from verion_gb300.backend import Cache

from .test_gpu_cache import BOX, SMALL, grid_of, records, table16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 131072, 131073])
def test_network_matches_the_oracle_over_record_counts(gpu_ctx, n):
    cache = Cache(gpu_ctx, bounds=BOX, **SMALL)
    g = grid_of(cache)
    rng = np.random.default_rng(n)
    m, gsize = cache.param_counts()
    mlp = rng.normal(0.0, (2.0 / 64.0) ** 0.5, m).astype(np.float32)
    cache.write_params(mlp, rng.uniform(-0.5, 0.5, gsize).astype(np.float32))
    rec = records(n, n + 1)
    got = cache.infer(rec)
    # A sample of rows: the first and last tile and some between.
    rows = np.unique(np.concatenate([np.arange(min(n, 130)), np.arange(max(0, n - 130), n), rng.integers(0, n, 64)]))
    want = nrc.predict(mlp, g, table16(cache, g), rec[rows])
    # One bf16 rounding flip of an activation (2^-8 of a value) may pass through each of four layers.
    assert np.max(np.abs(got[rows] - want)) <= 0.02 * max(1.0, np.max(np.abs(want)))
    if n <= 129:
        gm, gg, loss = cache.gradients(rec)
        lw, dws, gx = nrc.backward(nrc.layers(mlp), nrc.inputs(g, table16(cache, g), rec), rec[:, 16:19])
        assert abs(loss - lw) <= 0.02 * abs(lw) + 1e-6
        ref = nrc.grid_gradient(g, rec, gx[:, :2 * g.levels]).ravel()
        assert np.linalg.norm(gg - ref) <= 0.05 * np.linalg.norm(ref)
