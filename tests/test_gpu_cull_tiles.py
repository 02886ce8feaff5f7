"""The compaction of the visible splats (keys and indices in index order, no depth sort) against the oracle at
the edges of its tiles and of the look-back's windows, on both sides of the limit between the two tile sizes,
with visible sets from none to all."""
import math

import numpy as np
import pytest

import oracle
from splatter_gb300 import Configuration, DepthSorting, Renderer, Scene, camera, synthetic
from tests.helpers import oracle_uniforms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 256 * 1024 + 1, 257 * 1024 + 5, (1 << 19) - 1, 1 << 19, (1 << 19) + 1,
                               256 * 2048 + 1, 513 * 2048 + 77])
@pytest.mark.parametrize("where", [0.0, 9.0, 100.0])
def test_visible_set(cuda, n, where):
    rec = synthetic.plain_small(n, seed=n % 97, sh_order=0)
    rec[:, 0] += where  # in view, half in view, out of view
    if where == 100.0:
        rec[n // 2, 0:3] = 0.0
    config = Configuration(max_splat_count=n, spherical_harmonics_order=0, depth_sorting=DepthSorting.NONE,
                           field_of_view_y=math.radians(60))
    cam = camera.look_at([0.0, 1.0, -12.0], [0.0, 0.0, 0.0])
    r = Renderer(config)
    s = Scene(r, n)
    s.load_chunk(rec)
    for _ in range(2):
        r.render_frame(s, cam, 64, 48)
        keys, idx, info = r.sorted_entries()
        okeys, oidx, v, _ = oracle.draw_list(oracle_uniforms(oracle, config, cam, 64, 48), int(config.depth_sorting),
                                             oracle.load_transform(rec)["center"])
        assert info.visible_count == v
        assert np.array_equal(idx.cpu().numpy().view(np.uint32), oidx)
        assert np.array_equal(keys.cpu().numpy().view(np.uint32), okeys)
    s.close()
    r.close()
