"""Differentiable rendering: torch.autograd.Function over the hand-written backward kernels.

`render_splats` takes the splat parameters the renderer uses (centres, rotations as given, scales,
opacities, SH) and returns the float4 image of an fp32-blend frame; its backward calls
spl_render_backward (raster backward + vertex-stage backward on the GPU).  `render_raw` applies the
file loader's activations first (Scene::load_chunk, scene.rs:225-250: rotor normalisation, exp of the
log-scales clamped to mean +- 5, sigmoid of the opacity logit) with the loader's own arithmetic on the
GPU (spl_activate_splats) and chains its backward there too (spl_activate_splats_backward), so
gradients reach the raw parameters a training loop optimises without torch elementwise kernels per
frame.  `render_raw_views` renders several views of the same raw parameters in one autograd node and
sums their gradients in place on the GPU (spl_render_backward_accumulate).  `l2_image_loss` is the
L2 loss of such frames against RGB targets, one pass each way (spl_l2_image_loss).  `activate` is
the same transform written in torch (a reference).  Depth order, culling and the 1/255 discard are
constants of the frame (no gradient), as in any splat rasteriser.
"""
import ctypes

import numpy as np

from . import _lib
from ._lib import check
from .renderer import BlendMode, Renderer, _stream_ptr

__all__ = ["render_splats", "render_raw", "render_raw_views", "activate", "activate_native", "l2_image_loss"]


# A pass over a small scene is bound by the host: a view, an allocation or a launch of torch costs 5 to 20 us there,
# about what a kernel of this library takes on 20k splats.  So the arrays that only this library sees are parts of
# one tensor, addressed by their offsets, and the stream is looked up once a pass (a step of fitting 20k splats at
# 256x192: 641 us with a tensor per array, 581 us so).
def _ptr(t):
    return t.data_ptr()


def _planes(t):
    """The addresses of t[0], t[1] and t[2], without the views; an IndexError where one of them is missing."""
    p, row = t.data_ptr(), t.element_size() * t.stride(0)
    if t.shape[0] < 3:
        raise IndexError(f"three planes expected, got {t.shape[0]}")
    return p, p + row, p + 2 * row


class _Splats:
    """n activated splats, or their gradients, in one tensor of 11 n floats: rotation (n, 4), scale and opacity
    (n, 4), centre planes (3, n).  Every part starts on a 16-byte boundary."""

    def __init__(self, data, n):
        self.data, self.n = data, n
        self.rot = data.data_ptr()
        self.scale_alpha = self.rot + 16 * n
        x = self.rot + 32 * n
        self.planes = (x, x + 4 * n, x + 8 * n)


class _WrappedScene:
    """A scene over device arrays (spl_scene_wrap): n splats whose x, y, z, rotation, scale_alpha and sh start at
    the addresses given.  Keeps the tensors in `keep`, which hold the arrays, alive."""

    def __init__(self, renderer, n, planes, rot, scale_alpha, sh, keep):
        self._lib = _lib.load()
        self._keep = keep
        h = ctypes.c_void_p()
        check(self._lib.spl_scene_wrap(renderer.handle, n, *planes, rot, scale_alpha, sh, ctypes.byref(h)))
        self._h = h

    @property
    def handle(self):
        return self._h

    def close(self):
        if getattr(self, "_h", None):
            self._lib.spl_scene_destroy(self._h)
            self._h = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def _import_torch():
    import torch
    return torch


class _RenderSplats:  # built lazily so that importing the package does not import torch
    fn = None

    @classmethod
    def get(cls):
        if cls.fn is None:
            torch = _import_torch()

            class RenderSplats(torch.autograd.Function):
                @staticmethod
                def forward(ctx, xyz, rot, scale_alpha, sh, renderer, camera_to_world, width, height):
                    xyz = xyz.contiguous()
                    rot = rot.contiguous()
                    scale_alpha = scale_alpha.contiguous()
                    sh = sh.contiguous()
                    n = rot.shape[0]
                    scene = _WrappedScene(renderer, n, _planes(xyz), _ptr(rot), _ptr(scale_alpha), _ptr(sh),
                                          (xyz, rot, scale_alpha, sh))
                    img = renderer.render_frame(scene, camera_to_world, width, height)
                    ctx.renderer = renderer
                    ctx.scene = scene
                    ctx.cam = np.ascontiguousarray(np.asarray(camera_to_world, np.float32).reshape(16))
                    ctx.size = (width, height)
                    ctx.save_for_backward(img)
                    renderer._last_frame_key = (id(scene), ctx.cam.tobytes(), width, height)
                    return img

                @staticmethod
                def backward(ctx, grad_img):
                    (img,) = ctx.saved_tensors
                    _frame_ready(ctx)
                    r = ctx.renderer
                    xyz, rot, sa, sh = ctx.scene._keep
                    gxyz = torch.zeros_like(xyz)
                    grot = torch.zeros_like(rot)
                    gsa = torch.zeros_like(sa)
                    gsh = torch.zeros_like(sh)
                    g = grad_img.contiguous().float()
                    check(r._lib.spl_render_backward(r.handle, ctx.scene.handle, _ptr(img), _ptr(g),
                                                     *_planes(gxyz), _ptr(grot), _ptr(gsa), _ptr(gsh),
                                                     _stream_ptr(None)))
                    return gxyz, grot, gsa, gsh, None, None, None, None

            cls.fn = RenderSplats
        return cls.fn


def _ensure_frame(r, scene, cam, w, h):
    """Re-renders (scene, cam) on renderer r if r has rendered another frame since: the backward
    reuses the renderer's frame state (sorted pairs, records, tile ranges)."""
    key = (id(scene), cam.tobytes(), w, h)
    if getattr(r, "_last_frame_key", None) != key:
        r.render_frame(scene, cam, w, h)  # deterministic: the same frame again
        r._last_frame_key = key


def _frame_ready(ctx):
    """Re-renders the frame of this autograd node if the renderer has rendered another one since."""
    _ensure_frame(ctx.renderer, ctx.scene, ctx.cam, *ctx.size)


def _activated_scene(torch, means, quats, log_scales, logits, sh, stream):
    """Activates the parameters (contiguous) on `stream`; returns wrap(renderer), the scene of the result."""
    n = quats.shape[0]
    splats = _Splats(torch.empty(11 * n, device=quats.device, dtype=torch.float32), n)
    check(_lib.load().spl_activate_splats(n, _ptr(means), _ptr(quats), _ptr(log_scales), _ptr(logits), *splats.planes,
                                          splats.rot, splats.scale_alpha, stream.cuda_stream))
    return lambda r: _WrappedScene(r, n, splats.planes, splats.rot, splats.scale_alpha, _ptr(sh), (splats, sh))


def _activation_grads(torch, quats, log_scales, splats, grads, st):
    """The gradients of means, quaternions, log-scales and logits from those of the activated splats."""
    n = splats.n
    f32 = dict(device=quats.device, dtype=torch.float32)
    g_means, g_quats = torch.empty((n, 3), **f32), torch.empty((n, 4), **f32)
    g_logs, g_logits = torch.empty((n, 3), **f32), torch.empty((n,), **f32)
    check(_lib.load().spl_activate_splats_backward(n, _ptr(quats), _ptr(log_scales), splats.rot, splats.scale_alpha,
                                                   *grads.planes, grads.rot, grads.scale_alpha, _ptr(g_means),
                                                   _ptr(g_quats), _ptr(g_logs), _ptr(g_logits), st))
    return g_means, g_quats, g_logs, g_logits


class _RenderRaw:  # built lazily, like _RenderSplats
    fn = None

    @classmethod
    def get(cls):
        if cls.fn is None:
            torch = _import_torch()

            class RenderRaw(torch.autograd.Function):
                @staticmethod
                def forward(ctx, means, quats, log_scales, logits, sh, renderer, camera_to_world, width, height):
                    means, quats, log_scales, logits, sh = (t.contiguous() for t in (means, quats, log_scales, logits,
                                                                                      sh))
                    st = torch.cuda.current_stream()
                    scene = _activated_scene(torch, means, quats, log_scales, logits, sh, st)(renderer)
                    img = renderer.render_frame(scene, camera_to_world, width, height, stream=st)
                    ctx.renderer = renderer
                    ctx.scene = scene
                    ctx.cam = np.ascontiguousarray(np.asarray(camera_to_world, np.float32).reshape(16))
                    ctx.size = (width, height)
                    ctx.save_for_backward(img, quats, log_scales)
                    renderer._last_frame_key = (id(scene), ctx.cam.tobytes(), width, height)
                    return img

                @staticmethod
                def backward(ctx, grad_img):
                    img, quats, log_scales = ctx.saved_tensors
                    _frame_ready(ctx)
                    r = ctx.renderer
                    splats, sh = ctx.scene._keep
                    grads = _Splats(torch.zeros_like(splats.data), splats.n)
                    gsh = torch.zeros_like(sh)
                    g = grad_img.contiguous().float()
                    st = _stream_ptr(None)
                    check(r._lib.spl_render_backward(r.handle, ctx.scene.handle, _ptr(img), _ptr(g), *grads.planes,
                                                     grads.rot, grads.scale_alpha, _ptr(gsh), st))
                    return *_activation_grads(torch, quats, log_scales, splats, grads, st), gsh, None, None, None, None

            cls.fn = RenderRaw
        return cls.fn


class _RenderRawViews:  # built lazily, like _RenderSplats
    fn = None

    @classmethod
    def get(cls):
        if cls.fn is None:
            torch = _import_torch()

            class RenderRawViews(torch.autograd.Function):
                @staticmethod
                def forward(ctx, means, quats, log_scales, logits, sh, renderers, cameras, width, height):
                    means, quats, log_scales, logits, sh = (t.contiguous() for t in (means, quats, log_scales, logits,
                                                                                      sh))
                    st = torch.cuda.current_stream()
                    wrap = _activated_scene(torch, means, quats, log_scales, logits, sh, st)
                    out = torch.empty((len(cameras), height, width, 4), device=quats.device, dtype=torch.float32)
                    scenes, views = {}, []
                    for v, cam in enumerate(cameras):
                        r = renderers[v % len(renderers)]
                        if id(r) not in scenes:
                            scenes[id(r)] = wrap(r)
                        scene = scenes[id(r)]
                        c = np.ascontiguousarray(np.asarray(cam, np.float32).reshape(16))
                        r.render_frame(scene, c, width, height, out=out[v], stream=st)
                        r._last_frame_key = (id(scene), c.tobytes(), width, height)
                        views.append((r, scene, c))
                    ctx.views = views
                    ctx.size = (width, height)
                    ctx.save_for_backward(out, quats, log_scales)
                    return out

                @staticmethod
                def backward(ctx, grad_out):
                    out, quats, log_scales = ctx.saved_tensors
                    w, h = ctx.size
                    splats, sh = ctx.views[0][1]._keep
                    grads = _Splats(torch.zeros_like(splats.data), splats.n)
                    gsh = torch.zeros_like(sh)
                    g = grad_out.contiguous().float()
                    st = _stream_ptr(None)
                    # the views in order, each adding its gradients in place
                    for v, (r, scene, c) in enumerate(ctx.views):
                        _ensure_frame(r, scene, c, w, h)
                        check(r._lib.spl_render_backward_accumulate(
                            r.handle, scene.handle, _ptr(out) + 4 * out.stride(0) * v, _ptr(g) + 4 * g.stride(0) * v,
                            *grads.planes, grads.rot, grads.scale_alpha, _ptr(gsh), st))
                    return *_activation_grads(torch, quats, log_scales, splats, grads, st), gsh, None, None, None, None

            cls.fn = RenderRawViews
        return cls.fn


def render_splats(xyz, rotation, scale_alpha, sh, renderer: Renderer, camera_to_world, width, height):
    """Differentiable frame.  xyz: (3, N) centre planes; rotation: (N, 4) scalar first; scale_alpha:
    (N, 4) scale xyz + opacity; sh: (N, 48).  Returns (H, W, 4) float32 (r, g, b, T)."""
    if renderer.config.blend_mode != BlendMode.FP32:
        raise ValueError("render_splats needs a renderer with blend_mode FP32")
    return _RenderSplats.get().apply(xyz, rotation, scale_alpha, sh, renderer, camera_to_world, width, height)


def activate_native(means, quats, log_scales, opacity_logits):
    """The loader's activations on the GPU (spl_activate_splats, no autograd): (xyz planes (3, N),
    rotation (N, 4), scale_alpha (N, 4)), bit for bit the arrays of a scene loaded from records."""
    torch = _import_torch()
    means, quats, log_scales, opacity_logits = (t.detach().contiguous() for t in (means, quats, log_scales,
                                                                                  opacity_logits))
    n = quats.shape[0]
    f32 = dict(device=quats.device, dtype=torch.float32)
    xyz, rot, sa = torch.empty((3, n), **f32), torch.empty((n, 4), **f32), torch.empty((n, 4), **f32)
    check(_lib.load().spl_activate_splats(n, _ptr(means), _ptr(quats), _ptr(log_scales), _ptr(opacity_logits),
                                          *_planes(xyz), _ptr(rot), _ptr(sa),
                                          _stream_ptr(None)))
    return xyz, rot, sa


def activate(means, quats, log_scales, opacity_logits):
    """The loader's activations (scene.rs:225-250) in torch: (xyz planes, rotation, scale_alpha)."""
    torch = _import_torch()
    rot = quats * (1.0 / torch.sqrt((quats * quats).sum(-1, keepdim=True)))
    avg = log_scales.sum(-1, keepdim=True) / 3.0
    ls = torch.minimum(torch.maximum(log_scales, avg - 5.0), avg + 5.0)
    scale = torch.exp(ls)
    alpha = torch.sigmoid(opacity_logits)
    return means.t(), rot, torch.cat([scale, alpha[:, None]], 1)


def render_raw(means, quats, log_scales, opacity_logits, sh, renderer, camera_to_world, width, height):
    """Differentiable frame from raw parameters: means (N, 3), quaternions (N, 4, scalar first),
    log-scales (N, 3), opacity logits (N,), SH (N, 48), all float32 CUDA tensors.  The frame equals the
    frame of a scene loaded from the same file records; gradients reach every raw parameter."""
    if renderer.config.blend_mode != BlendMode.FP32:
        raise ValueError("render_raw needs a renderer with blend_mode FP32")
    for t, shape in ((means, 3), (quats, 4), (log_scales, 3), (sh, 48)):
        if t.dim() != 2 or t.shape[1] != shape or t.dtype.itemsize != 4 or not t.is_cuda:
            raise ValueError("render_raw: float32 CUDA tensors (N, 3), (N, 4), (N, 3), (N,), (N, 48) expected")
    return _RenderRaw.get().apply(means, quats, log_scales, opacity_logits, sh, renderer, camera_to_world, width,
                                  height)


def render_raw_views(means, quats, log_scales, opacity_logits, sh, renderers, cameras, width, height):
    """render_raw over several views of the same parameters in one autograd node: returns
    (len(cameras), H, W, 4) float32.  The backward adds every view's gradients into one set of arrays
    in place (spl_render_backward_accumulate), view after view, and chains the loader's activations
    once, instead of a gradient array per view that autograd zeroes and sums.  `renderers`: one
    Renderer, or a sequence used round robin over the views; a renderer keeps the frame state of the
    last view it rendered, so with fewer renderers than views the backward renders the other views
    again (same frames).  Gradients equal the per-view render_raw gradients summed over the views, to
    rounding: the raster backward sums with float atomics, and the activations' chain rule is
    applied to the sum instead of to each view."""
    if isinstance(renderers, Renderer):
        renderers = [renderers]
    renderers = list(renderers)
    cameras = list(cameras)
    if not renderers or not cameras:
        raise ValueError("render_raw_views: at least one renderer and one camera")
    if any(r.config.blend_mode != BlendMode.FP32 for r in renderers):
        raise ValueError("render_raw_views needs renderers with blend_mode FP32")
    for t, shape in ((means, 3), (quats, 4), (log_scales, 3), (sh, 48)):
        if t.dim() != 2 or t.shape[1] != shape or t.dtype.itemsize != 4 or not t.is_cuda:
            raise ValueError("render_raw_views: float32 CUDA tensors (N, 3), (N, 4), (N, 3), (N,), (N, 48) expected")
    return _RenderRawViews.get().apply(means, quats, log_scales, opacity_logits, sh, renderers, cameras, width,
                                       height)


class _L2ImageLoss:  # built lazily, like _RenderSplats
    fn = None

    @classmethod
    def get(cls):
        if cls.fn is None:
            torch = _import_torch()

            class L2ImageLoss(torch.autograd.Function):
                @staticmethod
                def forward(ctx, images, targets):
                    images, targets = images.contiguous(), targets.contiguous()
                    pixels = images.numel() // 4
                    lib = _lib.load()
                    partial = torch.empty(int(lib.spl_l2_image_loss_partials(pixels)), device=images.device,
                                          dtype=torch.float32)
                    check(lib.spl_l2_image_loss(_ptr(images), _ptr(targets), pixels, _ptr(partial), _stream_ptr(None)))
                    ctx.save_for_backward(images, targets)
                    return partial.sum()

                @staticmethod
                def backward(ctx, grad_loss):
                    images, targets = ctx.saved_tensors
                    grad = torch.empty_like(images)
                    scale = grad_loss.detach().to(torch.float32).contiguous()
                    check(_lib.load().spl_l2_image_loss_backward(_ptr(images), _ptr(targets), images.numel() // 4,
                                                                 _ptr(scale), _ptr(grad), _stream_ptr(None)))
                    return grad, None

            cls.fn = L2ImageLoss
        return cls.fn


def l2_image_loss(images, targets):
    """sum over pixels and RGB of (images[..., :3] - targets)^2 for float4 frames (..., 4) (r, g, b, T),
    such as render_raw_views returns, against float32 RGB targets (..., 3): the value of
    ((images[..., :3] - targets) ** 2).sum() (summed in another order) with the same gradient bit for
    bit, (2 (image - target) * upstream, 0), each way in one pass over the frames."""
    if images.dim() < 1 or images.shape[-1] != 4 or targets.shape[-1] != 3 or images.shape[:-1] != targets.shape[:-1]:
        raise ValueError("l2_image_loss: images (..., 4) and targets (..., 3) with the same leading shape expected")
    torch = _import_torch()
    if images.dtype != torch.float32 or targets.dtype != torch.float32 or not images.is_cuda or not targets.is_cuda:
        raise ValueError("l2_image_loss: float32 CUDA tensors expected")
    return _L2ImageLoss.get().apply(images, targets)
