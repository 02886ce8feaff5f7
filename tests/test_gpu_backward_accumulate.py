"""Gradients added in place, exactly: each splat lies on one group of 2x2 pixels alone, so that its record's gradients
are one addition each, and the loss of a view given twice has gradients that are twice the single view's bit for bit
(once: the same).  Every SH degree, the last, partial piece of a row among them; needles and round splats."""
import math

import pytest

from splatter_gb300 import BlendMode, Configuration, Renderer, camera
from splatter_gb300.autograd import render_raw, render_raw_views

pytestmark = pytest.mark.gpu

DIST, FOVY = 10.0, math.radians(50)


def lattice(side, size):
    """side^2 splats whose centres lie on the corners between the four pixels of every other group, 2 sigma = 0.6 pixel
    wide across; every third one a needle along the view."""
    import torch
    pitch = 2.0 * DIST * math.tan(FOVY / 2) / size  # of a pixel, at the splats
    k = torch.arange(side * side)
    px = 4.0 * torch.stack([k % side, k // side], 1) + 1.0 - size / 2
    gen = torch.Generator().manual_seed(side)
    means = torch.cat([px * pitch, torch.zeros(side * side, 1)], 1)
    quats = torch.tensor([[1.0, 0.0, 0.0, 0.0]]).repeat(side * side, 1)
    logs = math.log(0.3 * pitch) + torch.zeros(side * side, 3)
    logs[::3, 2] -= 4.0
    sh = 0.2 * torch.randn(side * side, 48, generator=gen)
    sh[:, :3] += 1.0
    return [t.float().contiguous() for t in (means, quats, logs, torch.rand(side * side, generator=gen) + 0.5, sh)]


@pytest.mark.parametrize("sh_order", [0, 1, 2, 3])
@pytest.mark.parametrize("side", [1, 6, 23])
def test_accumulated_gradients_are_exact(cuda, side, sh_order):
    import torch
    size = 4 * side + (4 * side) % 2
    params = lattice(side, size)
    n = side * side
    config = Configuration(max_splat_count=n, max_pair_count=64 * n + 1024, spherical_harmonics_order=sh_order,
                           blend_mode=BlendMode.FP32, field_of_view_y=FOVY)
    cam = camera.look_at([0.0, 0.0, -DIST], [0.0, 0.0, 0.0])
    weight = torch.rand((size, size, 3), device="cuda", generator=torch.Generator("cuda").manual_seed(n)) - 0.3
    rs = [Renderer(config) for _ in range(2)]

    def grads(render):
        leaves = [t.cuda().requires_grad_(True) for t in params]
        (render(leaves)[..., :3] * weight).sum().backward()
        return [t.grad for t in leaves]
    single = grads(lambda p: render_raw(*p, rs[0], cam, size, size))
    once = grads(lambda p: render_raw_views(*p, rs, [cam], size, size))
    twice = grads(lambda p: render_raw_views(*p, rs, [cam, cam], size, size))
    assert float((single[0].abs().sum(1) > 0).float().mean()) > 0.9
    for a, b, c in zip(single, once, twice):
        assert torch.equal(a, b) and torch.equal(2.0 * a, c)
    for r in rs:
        r.close()
