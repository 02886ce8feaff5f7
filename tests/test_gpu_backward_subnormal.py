"""Gradients below the smallest normal float, added in place: the same bits as stored ones, and twice those after a
second addition.  Each splat lies on one pixel group alone, so that its record's gradients are one addition each."""
import ctypes

import numpy as np
import pytest

from splatter_gb300 import BlendMode, Configuration, Renderer, camera
from splatter_gb300._lib import check
from splatter_gb300.autograd import _planes, _ptr, _WrappedScene, activate_native
from tests.test_gpu_backward_accumulate import DIST, FOVY, lattice

pytestmark = pytest.mark.gpu


def test_subnormal_gradients_are_kept(cuda):
    import torch
    side, size = 6, 24
    n = side * side
    means, quats, logs, logits, sh = (t.cuda() for t in lattice(side, size))
    xyz, rot, sa = activate_native(means, quats, logs, logits)
    r = Renderer(Configuration(max_splat_count=n, max_pair_count=64 * n + 1024, spherical_harmonics_order=3,
                               blend_mode=BlendMode.FP32, field_of_view_y=FOVY))
    scene = _WrappedScene(r, n, _planes(xyz), _ptr(rot), _ptr(sa), _ptr(sh), (xyz, rot, sa, sh))
    img = r.render_frame(scene, camera.look_at([0.0, 0.0, -DIST], [0.0, 0.0, 0.0]), size, size)
    weight = torch.rand((size, size, 4), device="cuda", generator=torch.Generator("cuda").manual_seed(1)) - 0.3
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def zeros():
        return [torch.zeros(n, device="cuda") for _ in range(3)] + [torch.zeros((n, k), device="cuda") for k in (4, 4, 48)]

    def add(call, grad, into):
        check(call(r.handle, scene.handle, _ptr(img), _ptr(grad), *(_ptr(t) for t in into), stream))
        return [t.cpu().numpy() for t in into]
    seen = np.zeros(6, int)
    for exponent in (-130, -126, -122, -118, -114, -110):
        grad = weight * 2.0 ** exponent
        stored = add(r._lib.spl_render_backward, grad, zeros())
        arrays = zeros()
        once = add(r._lib.spl_render_backward_accumulate, grad, arrays)
        twice = add(r._lib.spl_render_backward_accumulate, grad, arrays)
        for k, (a, b, c) in enumerate(zip(stored, once, twice)):
            seen[k] += ((a != 0) & (np.abs(a) < np.finfo(np.float32).tiny)).sum()
            assert np.array_equal(a, b) and np.array_equal(a + a, c)
    assert (seen > 0).all()
    r.close()
