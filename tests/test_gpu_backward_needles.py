"""The sweep of needles and discs in double, 32 to a block and a warp for each part of their gradients: scenes of
needles and discs alone, as many as fill a block, a round of the grid and more.  The same scene with its splats in
another order is the same image, while every splat takes another place in the blocks: its gradients are the same.
Bar: 5e-6 of each array's largest gradient, the order of the raster backward's float atomics (the bar of the repeated
needle gradients, whose noise it bounds)."""
import math

import pytest

from splatter_gb300 import BlendMode, Configuration, Renderer, camera
from splatter_gb300.autograd import render_raw

pytestmark = pytest.mark.gpu

CELL = 16  # pixels


def splats(n, side):
    """Raw parameters of n splats in the cells of a side x side grid, seen head on at distance 10."""
    import torch
    gen = torch.Generator().manual_seed(n)
    k = torch.arange(n)
    pitch = 2.0 * 10.0 * math.tan(math.radians(25)) / side
    xy = (torch.stack([k % side, k // side], 1) + 0.5 - side / 2) * pitch
    depth = (torch.randperm(n, generator=gen) + 0.5) / n - 0.5  # no two the same
    means = torch.cat([xy, depth[:, None]], 1)
    quats = torch.randn(n, 4, generator=gen)
    quats = quats / quats.norm(dim=1, keepdim=True) * (0.9 + 0.2 * torch.rand(n, 1, generator=gen))
    logs = math.log(pitch / 12) + torch.tensor([[0.0, -3.7, -3.9]]).repeat(n, 1)  # needles: ratio 40 and 49
    logs[1::2] = math.log(pitch / 12) + torch.tensor([0.0, 0.1, -4.0])  # discs
    logits = torch.rand(n, generator=gen) + 0.5
    sh = 0.2 * torch.randn(n, 48, generator=gen)
    sh[:, :3] += 1.0
    return [t.float().contiguous() for t in (means, quats, logs, logits, sh)]


def gradients(params, side, cov, sh_order):
    import torch
    n = params[0].shape[0]
    r = Renderer(Configuration(max_splat_count=n, max_pair_count=64 * n + 1024, spherical_harmonics_order=sh_order,
                               blend_mode=BlendMode.FP32, use_covariance_for_scale=cov, field_of_view_y=math.radians(50)))
    leaves = [t.cuda().requires_grad_(True) for t in params]
    w = side * CELL
    img = render_raw(*leaves, r, camera.look_at([0.0, 0.0, -10.0], [0.0, 0.0, 0.0]), w, w)
    y, x = torch.meshgrid(torch.arange(w, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    weight = torch.stack([torch.sin(0.31 * x + 0.17 * y), torch.cos(0.23 * x - 0.29 * y), torch.sin(0.37 * y)], -1)
    (img[..., :3] * weight).sum().backward()
    r.close()
    return [t.grad for t in leaves]


@pytest.mark.parametrize("cov,sh_order", [(True, 3), (False, 0)])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 97, "round", "round + 1", "two rounds"])
def test_needles_alone(cuda, n, cov, sh_order):
    import torch
    one_round = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    n = {"round": one_round, "round + 1": one_round + 1, "two rounds": 2 * one_round + 33}.get(n, n)
    side = math.ceil(math.sqrt(n))
    params = splats(n, side)
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(7))
    one, other = gradients(params, side, cov, sh_order), gradients([t[perm].contiguous() for t in params], side, cov, sh_order)
    # a needle thinner than a pixel may lie between the pixels' centres and not be drawn
    assert float((one[0].abs().sum(1) > 0).float().mean()) > 0.5 or n < 31
    for a, b in zip(one, other):
        assert bool(torch.isfinite(a).all())
        assert float((a[perm.cuda()] - b).abs().max()) <= 5e-6 * float(a.abs().max())
