"""The vertex stage's two ways of reading SH rows (staged through shared memory from 2^19 splats on, a row
per lane below) against the oracle, bit for bit: every SH degree, both sides of the limit, a last warp that
is not full, visible sets from one splat to all of them."""
import math

import numpy as np
import pytest

import oracle
from splatter_gb300 import Configuration, Renderer, Scene, camera, synthetic
from tests.helpers import oracle_cfg, oracle_uniforms

pytestmark = pytest.mark.gpu

LIMIT = 1 << 19


@pytest.mark.parametrize("covariance,rects", [(True, True), (False, False)])
@pytest.mark.parametrize("sh", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [LIMIT - 1, LIMIT, LIMIT + 37])
@pytest.mark.parametrize("seen", ["one", "some", "all"])
def test_records_equal_the_oracle(cuda, n, sh, seen, covariance, rects):
    import torch
    if seen != "some" and (n != LIMIT + 37 or not rects):
        pytest.skip("the visible set's extremes once per degree")
    config = Configuration(max_splat_count=n, spherical_harmonics_order=sh, use_covariance_for_scale=covariance,
                           use_unaligned_rectangles=rects, field_of_view_y=math.radians(60))
    rec = synthetic.clustered(n, seed=5, sh_order=3)
    if seen == "one":
        rec[:, 2] -= 1000.0
        rec[n // 2, 0:3] = 0.0
    elif seen == "all":
        rec[:, 0:3] *= 0.1
    cam = camera.look_at([0.0, 3.0, -16.0], [0.0, 0.0, 0.0])
    r = Renderer(config)
    s = Scene(r, n)
    s.load_chunk(rec)
    r.render_frame(s, cam, 320, 200)
    torch.cuda.synchronize()
    keys, idx, info = r.sorted_entries()
    got = r.records().cpu().numpy()
    visible = np.sort(idx.cpu().numpy().view(np.uint32))
    assert info.visible_count == {"one": 1, "some": info.visible_count, "all": n}[seen]
    want, _, _ = oracle.preprocess(oracle_uniforms(oracle, config, cam, 320, 200), oracle_cfg(oracle, config),
                                   oracle.load_transform(rec), visible)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(np.where(nan, 0.0, got).astype(np.float32).view(np.uint32),
                          np.where(nan, 0.0, want).astype(np.float32).view(np.uint32))
    s.close()
    r.close()
