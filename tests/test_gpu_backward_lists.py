"""The raster backward's lists against a plain torch float64 evaluation of the same frame, record gradients of
every splat: batch and list-word edges (1 ... 513 records on a tile), viewports that end inside a tile, margins on
both sides of the falloff's short path, both rectangle kinds."""
import math

import numpy as np
import pytest

from splatter_gb300 import BlendMode, Configuration, Renderer, Scene
from tests.helpers import default_cam
from tests.test_gpu_raster_lists import stack_of_splats

pytestmark = pytest.mark.gpu


def reference(rec, order, image_grad, w, h, fov, margin, rects):
    """dL/drecord (n, 10) in float64 torch from the renderer's own records, in their drawing order; the
    renderer's gradients of A are against offsets from the pixel box's centre and of B at that centre."""
    import torch
    box = rec[:, [7, 11]].copy().view(np.uint32)
    lo, hi = box[:, 0], box[:, 1]
    n = rec.shape[0]
    ctr = np.stack([0.5 * ((lo & 0xFFFF) + (hi & 0xFFFF) + 1.0), 0.5 * ((lo >> 16) + (hi >> 16) + 1.0)], 1)
    drawn = (lo & 0xFFFF) <= (hi & 0xFFFF)
    rec = np.where(drawn[:, None] & np.isfinite(rec), rec, 0.0)
    q = torch.from_numpy(np.nan_to_num(rec.astype(np.float64)))
    lin, const = q[:, [0, 1, 3, 4]], q[:, [2, 5]]
    c = torch.from_numpy(np.where(drawn[:, None], ctr, 0.0))
    at_centre = torch.stack([const[:, 0] + lin[:, 0] * c[:, 0] + lin[:, 1] * c[:, 1],
                             const[:, 1] + lin[:, 2] * c[:, 0] + lin[:, 3] * c[:, 1]], 1)
    p = torch.cat([lin[:, :2], at_centre[:, :1], lin[:, 2:], at_centre[:, 1:], q[:, 6:7], q[:, 8:11]], 1)
    p.requires_grad_(True)
    psx, psy = 2.0 * math.tan(fov / 2) * (w / h) / w, -2.0 * math.tan(fov / 2) / h
    ys, xs = torch.meshgrid(torch.arange(h, dtype=torch.float64) + 0.5, torch.arange(w, dtype=torch.float64) + 0.5, indexing="ij")
    col, trans = [torch.zeros(h, w, dtype=torch.float64) for _ in range(3)], torch.ones(h, w, dtype=torch.float64)
    gray = torch.zeros(h, w, dtype=torch.bool)  # pixels within rounding of a decision
    live = torch.ones(h, w, dtype=torch.bool)
    for k in order:
        if not drawn[k]:
            continue
        a = p[k]
        dx, dy = xs - c[k, 0], ys - c[k, 1]
        u, v = a[0] * dx + a[1] * dy + a[2], a[3] * dx + a[4] * dy + a[5]
        inbox = (xs > (lo[k] & 0xFFFF)) & (xs < (hi[k] & 0xFFFF) + 1) & (ys > (lo[k] >> 16)) & (ys < (hi[k] >> 16) + 1)
        with torch.no_grad():
            if rects:
                far = torch.maximum(u.abs(), v.abs())
                edge, cover = (far - margin).abs() < 1e-4 * (1 + far), far <= margin
            else:  # the axis-aligned square in the view plane
                sx, sy = (psx * xs + q[k, 12]).abs(), (psy * ys + q[k, 13]).abs()
                far, side = torch.maximum(sx, sy), q[k, 14]
                edge, cover = (far - side).abs() < 1e-5, far <= side
        alpha = a[6] * torch.exp(-0.5 * (u * u + v * v))
        with torch.no_grad():
            gray |= live & inbox & (edge | (cover & ((alpha * 255 - 1).abs() < 1e-3)))
            use = live & inbox & cover & (alpha >= 1.0 / 255.0)
        alpha = torch.where(use, alpha, torch.zeros_like(alpha))
        for ch in range(3):
            col[ch] = col[ch] + (a[7 + ch] * alpha).clamp(0, 1) * trans
        trans = trans * (1 - alpha.clamp(max=1))
        with torch.no_grad():
            gray |= live & ((trans / 1e-4 - 1).abs() < 1e-3)
            live &= trans >= 1e-4
    img = torch.stack(col + [trans], -1) + 0.0 * p.sum()  # differentiable where nothing is drawn
    img.backward(torch.from_numpy(np.where(gray.numpy()[..., None], 0.0, image_grad)))
    return p.grad.numpy(), gray.numpy()


@pytest.mark.parametrize("rects", [True, False])
@pytest.mark.parametrize("margin", [2.0, 9.5])
@pytest.mark.parametrize("n,size", [(1, (16, 16)), (33, (19, 17)), (256, (16, 16)), (257, (33, 15)), (513, (16, 31))])
def test_record_gradients(cuda, n, size, margin, rects):
    import ctypes
    import torch
    from splatter_gb300._lib import check
    w, h = size
    config = Configuration(max_splat_count=n, spherical_harmonics_order=1, ellipse_margin=margin, blend_mode=BlendMode.FP32,
                           use_unaligned_rectangles=rects, field_of_view_y=math.radians(50))
    r = Renderer(config)
    s = Scene(r, n)
    s.load_chunk(stack_of_splats(n, seed=n + 7))
    img = r.render_frame(s, default_cam(dist=4.0), w, h)
    torch.cuda.synchronize()
    keys, idx, info = r.sorted_entries()
    visible = np.sort(idx.cpu().numpy())
    order = np.searchsorted(visible, idx.cpu().numpy())[:info.draw_count]
    rng = np.random.default_rng(n)
    g = rng.normal(size=(h, w, 4)).astype(np.float32)
    want, gray = reference(r.records().cpu().numpy(), order, g.astype(np.float64), w, h, config.field_of_view_y, margin,
                           rects)
    g[gray] = 0.0
    dev = dict(device="cuda", dtype=torch.float32)
    gi = torch.from_numpy(g).cuda()
    out = [torch.zeros(n, **dev) for _ in range(3)] + [torch.zeros((n, 4), **dev), torch.zeros((n, 4), **dev),
                                                       torch.zeros((n, 48), **dev)]
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    check(r._lib.spl_render_backward(r.handle, s.handle, ptr(img), ptr(gi), *(ptr(t) for t in out),
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = torch.empty((info.visible_count, 10), **dev)
    check(r._lib.spl_renderer_copy_record_gradients(r.handle, ptr(got), info.visible_count, ctypes.c_void_p(0)))
    torch.cuda.synchronize()
    got = got.cpu().numpy().astype(np.float64)
    # float32 sums of up to w h terms of the frame's size: a component's error against its column's scale
    scale = np.sqrt((want ** 2).mean(0)) + 1e-6
    assert np.abs(got - want).max(0).max() / scale.max() < 0.05
    assert (np.abs(got - want) <= 2e-3 * (np.abs(want) + scale)).mean() > 0.99
    r.close()
