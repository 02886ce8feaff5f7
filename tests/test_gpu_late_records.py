"""Records of a tile's second and third batch, in the raster and its backward.  Small faint splats all over one tile, so
that its pixels are far from opaque after 256 records and every later record shows: in the oracle's image, which is the
renderer's bit for bit, and in the record gradients, each of which is compared by itself."""
import math

import numpy as np
import pytest

import oracle
from splatter_gb300 import BlendMode, Configuration, Renderer, Scene, camera, synthetic
from tests.helpers import oracle_cfg, oracle_uniforms
from tests.test_gpu_backward_lists import reference

W = H = 16
DIST, FOVY, MARGIN = 10.0, math.radians(50), 2.0
COUNTS = [257, 288, 289, 320, 321, 384, 385, 512, 513]  # one, two, four and eight list words in a later batch, and one record
CAM = camera.look_at([0.0, 0.0, -DIST], [0.0, 0.0, 0.0])


def faint_splats(n):
    """n records whose splats lie inside the tile, some three pixels across, at depths that are all different."""
    pitch = 2.0 * DIST * math.tan(FOVY / 2) / H  # of a pixel, at the splats
    rng = np.random.default_rng(n)
    rec = synthetic.plain_small(n, seed=n, sh_order=1)
    rec[:, 0:2] = rng.uniform(-6.0, 6.0, (n, 2)) * pitch
    rec[:, 2] = (rng.permutation(n) + 0.5) / n - 0.5
    rec[:, 54] = rng.uniform(-3.0, -2.0, n)  # opacities from 0.05 to 0.12
    rec[:, 55:58] = np.log(rng.uniform(0.4, 0.7, (n, 3)) * pitch)
    return rec


def config(n, rects, blend):
    return Configuration(max_splat_count=n, spherical_harmonics_order=1, field_of_view_y=FOVY, ellipse_margin=MARGIN,
                         use_unaligned_rectangles=rects, blend_mode=blend)


def scene_on_cpu(cfg, rec):
    """(splats, uniforms, configuration, the splats' indices in drawing order) of the oracle."""
    splats, u = oracle.load_transform(rec), oracle_uniforms(oracle, cfg, CAM, W, H)
    return splats, u, oracle_cfg(oracle, cfg), oracle.draw_list(u, int(cfg.depth_sorting), splats["center"])[1]


def far(got, want):
    """The entries (record, column) that are off by more than 1e-3 of themselves and of their column's scale: a record's
    gradients are float sums of the terms of some ten pixels, in which the difference of the final and the blended
    colours, of some 40 roundings of at most 2^-24, is the least exact value (some 1e-5 of its factors)."""
    scale = np.sqrt((want ** 2).mean(0))
    return ~(np.abs(got - want) <= 1e-3 * (np.abs(want) + scale))


def gradient_case(n, rects, records, order):
    """(dL/dimage, record gradients in 64 bits) of the frame with these records."""
    g = np.random.default_rng(n).normal(size=(H, W, 4)).astype(np.float32)
    want, gray = reference(records, order, g.astype(np.float64), W, H, FOVY, MARGIN, rects)
    g[gray] = 0.0
    return g, want


@pytest.mark.parametrize("rects", [True, False])
@pytest.mark.parametrize("blend", [BlendMode.UNORM8, BlendMode.FP32])
@pytest.mark.parametrize("n", [257, 385, 513])
def test_late_records_show_in_the_oracle(n, blend, rects):
    cfg = config(n, rects, blend)
    rec = faint_splats(n)
    splats, u, c, order = scene_on_cpu(cfg, rec)
    assert len(order) == n
    whole = oracle.render(u, c, splats)[0].tobytes()
    late = order[256:]
    seen = [oracle.render(u, c, oracle.load_transform(np.delete(rec, k, 0)))[0].tobytes() != whole for k in late]
    assert all(seen) if blend == BlendMode.FP32 else np.mean(seen) > 0.75


@pytest.mark.parametrize("rects", [True, False])
@pytest.mark.parametrize("n", [257, 513])
def test_a_lost_record_is_seen_in_the_gradients(n, rects):
    splats, u, c, order = scene_on_cpu(config(n, rects, BlendMode.FP32), faint_splats(n))
    records = oracle.preprocess(u, c, splats, np.arange(n, dtype=np.uint32))[0]
    want = gradient_case(n, rects, records, order)[1]
    assert not far(want.astype(np.float32), want).any()
    for k in range(n):
        lost = want.copy()
        lost[k] = 0.0
        assert far(lost, want)[k].any(), k


@pytest.mark.gpu
@pytest.mark.parametrize("rects", [True, False])
@pytest.mark.parametrize("blend", [BlendMode.UNORM8, BlendMode.FP32])
@pytest.mark.parametrize("n", COUNTS)
def test_image(cuda, n, blend, rects):
    import torch
    cfg = config(n, rects, blend)
    rec = faint_splats(n)
    r = Renderer(cfg)
    s = Scene(r, n)
    s.load_chunk(rec)
    img = r.render_frame(s, CAM, W, H)
    torch.cuda.synchronize()
    assert r.frame_info().pair_count == n
    splats, u, c, _ = scene_on_cpu(cfg, rec)
    assert img.cpu().numpy().tobytes() == oracle.render(u, c, splats)[0].tobytes()
    r.close()


@pytest.mark.gpu
@pytest.mark.parametrize("rects", [True, False])
@pytest.mark.parametrize("n", COUNTS)
def test_record_gradients(cuda, n, rects):
    import ctypes
    import torch
    from splatter_gb300._lib import check
    r = Renderer(config(n, rects, BlendMode.FP32))
    s = Scene(r, n)
    s.load_chunk(faint_splats(n))
    img = r.render_frame(s, CAM, W, H)
    torch.cuda.synchronize()
    idx, info = r.sorted_entries()[1:]
    assert info.visible_count == info.pair_count == n
    g, want = gradient_case(n, rects, r.records().cpu().numpy(), idx.cpu().numpy())  # all visible: slots are indices
    dev = dict(device="cuda", dtype=torch.float32)
    gi = torch.from_numpy(g).cuda()
    out = [torch.zeros(n, **dev) for _ in range(3)] + [torch.zeros((n, k), **dev) for k in (4, 4, 48)]
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    check(r._lib.spl_render_backward(r.handle, s.handle, ptr(img), ptr(gi), *(ptr(t) for t in out), stream))
    got = torch.empty((n, 10), **dev)
    check(r._lib.spl_renderer_copy_record_gradients(r.handle, ptr(got), n, stream))
    bad = far(got.cpu().numpy().astype(np.float64), want)
    assert not bad.any(), np.argwhere(bad)
    r.close()
