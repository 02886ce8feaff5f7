"""The (tile, splat) pairs' emission against the oracle's frames, bit for bit, where its chunks can go wrong:
splats that cover the whole viewport beside splats of one tile or none, entry counts at the edges of the
binning kernel's tiles, lists of a few pairs and of hundreds per entry."""
import math

import numpy as np
import pytest

import oracle
from splatter_gb300 import Configuration, Renderer, Scene, synthetic
from tests.helpers import default_cam, oracle_cfg, oracle_uniforms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", ["none", "first", "some", "all"])
@pytest.mark.parametrize("n", [1, 127, 511, 512, 513, 1025, 20011])
def test_frames_equal_the_oracle(cuda, n, wide):
    import torch
    if wide == "all" and n > 2000:
        pytest.skip("a viewport-filling splat per entry is enough at small counts")
    rng = np.random.default_rng(n)
    rec = synthetic.plain_small(n, seed=n, sh_order=0)
    rec[:, 0:3] = rng.normal(0.0, 1.2, (n, 3))
    rec[rng.random(n) < 0.3, 0] += 4.0  # visible by the frustum's tolerance, outside the viewport or behind its edge
    big = {"none": np.zeros(n, bool), "first": np.arange(n) < max(1, n // 300), "some": rng.random(n) < 0.01,
           "all": np.ones(n, bool)}[wide]
    rec[big, 55:58] = rng.uniform(0.0, 1.0, (int(big.sum()), 3))
    rec[big, 54] = -4.0
    rec[big, 0:3] *= 0.3
    config = Configuration(max_splat_count=n, spherical_harmonics_order=0, field_of_view_y=math.radians(50))
    cam = default_cam(dist=6.0)
    w, h = 333, 207
    r = Renderer(config)
    s = Scene(r, n)
    s.load_chunk(rec)
    img = r.render_frame(s, cam, w, h)
    torch.cuda.synchronize()
    r.frame_info()
    ref, _ = oracle.render(oracle_uniforms(oracle, config, cam, w, h), oracle_cfg(oracle, config), oracle.load_transform(rec))
    assert np.array_equal(img.cpu().numpy(), ref)
    s.close()
    r.close()
