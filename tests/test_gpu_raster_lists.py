"""The rasteriser's per-pixel record lists against the oracle, bit for bit, where they can go wrong: batch
and list-word edges (31 ... 513 records on a tile), viewports that end inside a tile, needles and discs at
any angle (their column intervals per row), margins on both sides of the falloff's short path."""
import math

import numpy as np
import pytest

import oracle
from splatter_gb300 import BlendMode, Configuration, Renderer, Scene, synthetic
from tests.helpers import default_cam, oracle_cfg, oracle_uniforms

pytestmark = pytest.mark.gpu


def stack_of_splats(n, seed):
    """n splats around the view axis, so that one tile's list holds most of them: round ones of every size,
    needles and discs, opacities from below the 1/255 discard to nearly 1."""
    rng = np.random.default_rng(seed)
    rec = synthetic.plain_small(n, seed=seed, sh_order=1)
    rec[:, 0:3] = rng.normal(0.0, 0.4, (n, 3))
    rec[:, 55:58] = rng.uniform(-5.0, -0.5, (n, 1))
    kind = rng.integers(0, 3, n)
    rec[kind == 1, 55] += 3.0
    rec[kind == 2, 56:58] += 3.0
    rec[:, 54] = rng.uniform(-6.0, 4.0, n)
    return rec


@pytest.mark.parametrize("rects", [True, False])
@pytest.mark.parametrize("margin", [0.5, 2.0, 9.0, 9.5])
@pytest.mark.parametrize("n,size", [(1, (16, 16)), (31, (17, 15)), (32, (16, 16)), (33, (33, 31)), (255, (16, 16)),
                                    (256, (37, 29)), (257, (16, 16)), (513, (47, 33)), (3000, (61, 47))])
def test_lists_equal_the_oracle(cuda, n, size, margin, rects):
    import torch
    rec = stack_of_splats(n, seed=n)
    sc = oracle.load_transform(rec)
    w, h = size
    cam = default_cam(dist=4.0)
    for blend in (BlendMode.UNORM8, BlendMode.FP32):
        config = Configuration(max_splat_count=n, spherical_harmonics_order=1, ellipse_margin=margin,
                               use_unaligned_rectangles=rects, field_of_view_y=math.radians(50), blend_mode=blend)
        r = Renderer(config)
        s = Scene(r, n)
        s.load_chunk(rec)
        img = r.render_frame(s, cam, w, h)
        torch.cuda.synchronize()
        r.frame_info()
        ref, _ = oracle.render(oracle_uniforms(oracle, config, cam, w, h), oracle_cfg(oracle, config), sc)
        got = img.cpu().numpy()
        assert got.dtype == ref.dtype and got.tobytes() == ref.tobytes(), (blend, np.argwhere(got != ref)[:4].tolist())
        s.close()
        r.close()


@pytest.mark.parametrize("size", [(608, 384), (1328, 176), (1024, 1024), (272, 3856)])
def test_tile_order_covers_the_viewport(cuda, size):
    """Viewports at the edges of the tile order: 912 tiles (all resident, no order) and 913, one 4096-tile step
    and one tile more."""
    import torch
    n, (w, h) = 4000, size
    rec = stack_of_splats(n, seed=3)
    rec[:, 0:3] *= 4.0
    config = Configuration(max_splat_count=n, spherical_harmonics_order=1, field_of_view_y=math.radians(70))
    cam = default_cam(dist=4.0)
    r = Renderer(config)
    s = Scene(r, n)
    s.load_chunk(rec)
    img = r.render_frame(s, cam, w, h, out=torch.full((h, w, 4), 7, dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    ref, _ = oracle.render(oracle_uniforms(oracle, config, cam, w, h), oracle_cfg(oracle, config), oracle.load_transform(rec))
    assert np.array_equal(img.cpu().numpy(), ref)
    s.close()
    r.close()
