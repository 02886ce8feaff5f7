"""Lists of one, two, four and eight words per batch, and batches that end at such a number of records, against the
oracle bit for bit."""
import math

import pytest

import oracle
from splatter_gb300 import BlendMode, Configuration, Renderer, Scene
from tests.helpers import default_cam, oracle_cfg, oracle_uniforms
from tests.test_gpu_raster_lists import stack_of_splats

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rects", [True, False])
@pytest.mark.parametrize("blend", [BlendMode.UNORM8, BlendMode.FP32])
@pytest.mark.parametrize("pairs", [31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 288, 289, 320, 321, 384, 385])
def test_a_tile_of_exactly_so_many_records(cuda, pairs, blend, rects):
    import torch
    n, (w, h) = 1200, (16, 16)
    rec = stack_of_splats(n, seed=pairs)
    cam = default_cam(dist=4.0)
    # as many of the first splats as give the tile that many pairs
    lo, hi = 0, n
    while True:
        m = (lo + hi) // 2
        config = Configuration(max_splat_count=max(m, 1), spherical_harmonics_order=1, field_of_view_y=math.radians(50),
                               use_unaligned_rectangles=rects, blend_mode=blend)
        r = Renderer(config)
        s = Scene(r, m)
        s.load_chunk(rec[:m])
        img = r.render_frame(s, cam, w, h)
        torch.cuda.synchronize()
        got = r.frame_info().pair_count
        if got == pairs:
            break
        lo, hi = (m + 1, hi) if got < pairs else (lo, m)
        assert lo <= hi and hi - lo < n + 1
        s.close()
        r.close()
    ref, _ = oracle.render(oracle_uniforms(oracle, config, cam, w, h), oracle_cfg(oracle, config),
                           oracle.load_transform(rec[:m]))
    assert img.cpu().numpy().tobytes() == ref.tobytes()
    s.close()
    r.close()
