"""Frames whose vertex stage runs beside the depth sort against the same frames with the stages one after the other
(as they are while their times are taken): images, drawing order and records, frame after frame without a wait between,
on both sides of the sort's and the frame's limits, launched directly and from the renderer's graph."""
import math

import pytest

from splatter_gb300 import Configuration, DepthSorting, Renderer, Scene
from tests.helpers import default_cam

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 700, 4097, 65537, 786_432, 786_433, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("mode", [DepthSorting.GPU, DepthSorting.CPU])
def test_frames_equal_those_one_after_the_other(cuda, n, mode):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    rec = torch.randn((n, 62), generator=gen, device="cuda")
    rec[:, 6:54] *= 0.1
    rec[:, 55:58] = -5.0 + 0.3 * rec[:, 55:58]
    config = Configuration(max_splat_count=n, spherical_harmonics_order=2, depth_sorting=mode,
                           field_of_view_y=math.radians(60))
    cams = [default_cam(dist=d) for d in (6.0, 9.0, 6.5, 12.0)]
    size = (333, 257)
    results = []
    for apart in (True, False):
        r = Renderer(config)
        s = Scene(r, n)
        s.load_chunk_device(rec)
        r.set_profiling(apart)
        images = [r.render_frame(s, c, *size) for c in cams]  # direct, captured, replayed
        keys, idx, info = r.sorted_entries()
        results.append((images, keys, idx, r.records(), info.visible_count))
        s.close()
        r.close()
    (ia, ka, xa, ra, va), (ib, kb, xb, rb, vb) = results
    assert va == vb and va > 0
    assert all(torch.equal(a, b) for a, b in zip(ia, ib))
    assert torch.equal(ka, kb) and torch.equal(xa, xb)
    assert torch.equal(ra.view(torch.int32), rb.view(torch.int32))
