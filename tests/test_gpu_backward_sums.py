"""How exactly the raster backward sums a record's gradients: the colour gradients of large splats that lie alone on
their pixels, whose terms are known bit for bit, against sums in 64 bits, and beside the error of the order that the
kernel's sums are meant to have: a tree over each group of 4x2 pixels, the groups' sums added to one float in any order.

The bound is 1.2 times that order's error.  A sum of N terms to a float one after another is off by an amount that grows
with the square root of N, so that groups of half the size would be off by 1.41 times as much; the 1,536 sums tell the
errors' root mean square to about 2%."""
import ctypes
import math

import numpy as np
import pytest

from splatter_gb300 import BlendMode, Configuration, Renderer, Scene, camera, synthetic
from splatter_gb300._lib import check

pytestmark = pytest.mark.gpu

SIDE, CELL, MARGIN, ROUNDS = 8, 64, 2.0, 8
DIST, FOVY = 10.0, math.radians(50)
F = np.float32


def splats():
    """SIDE x SIDE round splats, one in the middle of each cell of CELL pixels, some 30 pixels wide."""
    n, size = SIDE * SIDE, SIDE * CELL
    pitch = 2.0 * DIST * math.tan(FOVY / 2) / size  # of a pixel, at the splats
    rng = np.random.default_rng(0)
    rec = synthetic.plain_small(n, seed=0, sh_order=0)
    k = np.arange(n)
    rec[:, 0] = (CELL * (k % SIDE + 0.5) - size / 2 + rng.uniform(-2, 2, n)) * pitch
    rec[:, 1] = (CELL * (k // SIDE + 0.5) - size / 2 + rng.uniform(-2, 2, n)) * pitch
    rec[:, 2] = 0.0
    rec[:, 6:9] = rng.uniform(0.0, 0.5, (n, 3))
    rec[:, 54] = rng.uniform(1.0, 2.0, n)
    rec[:, 55:58] = np.log(rng.uniform(6.5, 8.0, (n, 1)) * pitch)
    rec[:, 58:62] = [1.0, 0.0, 0.0, 0.0]
    return rec


def fma(a, b, c):  # the product is exact in 64 bits
    return (np.float64(a) * np.float64(b) + np.float64(c)).astype(F)


def falloff(rec):
    """alpha of every pixel (0 where the record is not drawn) of one record, in the kernel's operations."""
    size = SIDE * CELL
    lo, hi = rec[[7, 11]].copy().view(np.uint32)
    x, y = np.meshgrid(np.arange(size, dtype=F) + F(0.5), np.arange(size, dtype=F) + F(0.5))
    u = fma(rec[1], y, fma(rec[0], x, rec[2]))
    v = fma(rec[4], y, fma(rec[3], x, rec[5]))
    box = (x > (lo & 0xFFFF)) & (x < (hi & 0xFFFF) + 1) & (y > (lo >> 16)) & (y < (hi >> 16) + 1)
    power = fma(u, u, (v * v).astype(F))
    alpha = rec[6] * np.exp(-0.5 * power.astype(np.float64)).astype(F)
    return np.where(box & (np.abs(u) <= F(MARGIN)) & (np.abs(v) <= F(MARGIN)) & (alpha >= F(1.0 / 255.0)), alpha, F(0.0))


def group_sums(terms):
    """The sums of the 4x2-pixel groups of an image, each in the kernel's order: over columns and rows of lane
    index 4 row + column by exchanges with lane ^ 4, ^ 2, ^ 1."""
    h, w = terms.shape
    lanes = terms.reshape(h // 2, 2, w // 4, 4).transpose(0, 2, 1, 3).reshape(-1, 8)
    for d in (4, 2, 1):
        lanes = lanes[:, :d] + lanes[:, d:2 * d]
    return lanes[:, 0]


def test_sums_are_as_exact_as_the_order_of_4x2_groups(cuda):
    import torch
    n, size = SIDE * SIDE, SIDE * CELL
    config = Configuration(max_splat_count=n, spherical_harmonics_order=0, ellipse_margin=MARGIN, field_of_view_y=FOVY,
                           blend_mode=BlendMode.FP32)
    r = Renderer(config)
    s = Scene(r, n)
    s.load_chunk(splats())
    img = r.render_frame(s, camera.look_at([0.0, 0.0, -DIST], [0.0, 0.0, 0.0]), size, size)
    torch.cuda.synchronize()
    info = r.frame_info()
    assert info.visible_count == n
    alpha = [falloff(rec) for rec in r.records().cpu().numpy()]
    assert (sum((a > 0).astype(int) for a in alpha) <= 1).all()  # alone on their pixels: each meets T = 1
    assert min((group_sums(a) > 0).sum() for a in alpha) > 80
    dev = dict(device="cuda", dtype=torch.float32)
    out = [torch.zeros(n, **dev) for _ in range(3)] + [torch.zeros((n, 4), **dev), torch.zeros((n, 4), **dev),
                                                       torch.zeros((n, 48), **dev)]
    got = torch.empty((n, 10), **dev)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(1)
    off, order_off = [], []
    for _ in range(ROUNDS):
        weight = rng.uniform(0.5, 2.0, 3).astype(F)
        g = torch.zeros((size, size, 4), **dev)
        g[..., :3] = torch.from_numpy(weight).cuda()
        check(r._lib.spl_render_backward(r.handle, s.handle, ptr(img), ptr(g), *(ptr(t) for t in out), stream))
        check(r._lib.spl_renderer_copy_record_gradients(r.handle, ptr(got), n, stream))
        have = got.cpu().numpy().astype(np.float64)
        for k in range(n):
            for c in range(3):
                terms = weight[c] * alpha[k]
                exact = terms.astype(np.float64).sum()
                sums = group_sums(terms)
                sums = rng.permutation(sums[sums != 0])
                off.append(have[k, 7 + c] / exact - 1)
                order_off.append(float(np.cumsum(sums, dtype=F)[-1]) / exact - 1)
    rms = lambda v: float(np.sqrt(np.mean(np.square(v))))  # noqa: E731
    print("error of the sums %.3g, of the order %.3g" % (rms(off), rms(order_off)))
    assert rms(off) <= 1.2 * rms(order_off)
    r.close()
