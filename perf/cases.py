"""The calls whose time and results stand for this package's use, as cases that a timing program runs.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call: a renderer, a resident scene, a camera, targets
    run(state)           one pass through the public entry points, and its outputs
    work(case)           the bytes and operations that one pass cannot do without
    exact(case, seed)    the same outputs in 64 bits, in plain torch, for the cases whose outputs are floats

Scenes are the two kinds of the benchmark configurations: one object (positions ~ N(0, 2^2), seen from
distance 8) and clusters in a 40^3 box (seen from an orbit inside it or a fly-through around it).
"""
import math

import numpy as np
import torch

from splatter_gb300 import BlendMode, Configuration, DepthSorting, Renderer, Scene
from splatter_gb300.autograd import l2_image_loss, render_raw, render_raw_views
from splatter_gb300.serving import Server

FOV = math.radians(60.0)
MARGIN, CULL_TOL = 2.0, 1.1
VIEWPORTS = ((512, 512), (1280, 720), (1920, 1080))


def _frame(name, n, w, h, scene, sh=3, sorting="GPU", covariance=True, rects=True, blend="UNORM8"):
    return {"name": name, "kind": "frame", "n": n, "w": w, "h": h, "scene": scene, "sh": sh, "sorting": sorting,
            "covariance": covariance, "rects": rects, "blend": blend}


def listed():
    return [
        # a thumbnail of a few splats: the launches of a frame and little else
        _frame("thumb_2k_128x96", 2048, 128, 96, "object"),
        # one scanned object in a small window, colours without view dependence
        _frame("object_100k_640x480", 100_000, 640, 480, "object", sh=0),
        # a viewer inside a room-sized scene at full HD
        _frame("room_1m_1080p", 1_000_000, 1920, 1080, "orbit"),
        # an odd-sized offline frame in the float target: axis-aligned squares, the CPU rule's depth keys
        _frame("squares_350k_1237x723", 349_999, 1237, 723, "orbit", sh=2, sorting="CPU", rects=False, blend="FP32"),
        # a fly-through of a large capture, full HD and 4K
        _frame("fly_6m_1080p", 6_000_000, 1920, 1080, "fly"),
        _frame("fly_6m_2160p", 6_000_000, 3840, 2160, "fly"),
        # a step of fitting a small object to one photograph: frame, loss, gradients of every parameter
        {"name": "fit_20k_256x192", "kind": "fit", "n": 20_000, "w": 256, "h": 192, "views": 1, "scene": "object"},
        # a step of training a full scene on a batch of eight photographs
        {"name": "train_1m_1024x1024_8v", "kind": "fit", "n": 1_000_000, "w": 1024, "h": 1024, "views": 8,
         "scene": "orbit"},
        # a service holding several scenes that answers a burst of requests of mixed scenes and viewports
        {"name": "serve_8_scenes_24_requests", "kind": "serve", "scenes": 8, "lo": 200_000, "hi": 1_500_000,
         "requests": 24},
        # the viewer while a file loads: the next 32768 records from the host, then the frame
        {"name": "loading_1m_1080p", "kind": "loading", "n": 1_000_000, "chunk": 32768, "w": 1920, "h": 1080},
        # the depth sort as a call of its own, at the size of a full frame's visible keys
        {"name": "sort_3500k", "kind": "sort", "n": 3_500_000, "bits": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 5 + ["fit"] * 2 + ["serve", "loading", "sort"])
    if kind == "frame":
        n, w = _log(rng, 2000, 6_000_000), _log(rng, 120, 3840)
        if n < 50_000:
            w = min(w, 1920)
        h = max(90, min(2160, int(w * rng.uniform(0.5, 1.0))))
        scene = rng.choice(["object", "orbit"]) if n <= 1_000_000 else "fly"
        c = _frame("", n, w, h, scene, rng.randint(0, 3), rng.choice(["GPU", "GPU", "GPU_INDIRECT_DRAW", "CPU", "NONE"]),
                   rng.random() < 0.8, rng.random() < 0.8, rng.choice(["UNORM8", "UNORM8", "FP32"]))
        c.pop("name")
        return c
    if kind == "fit":
        n, w = _log(rng, 5000, 1_000_000), _log(rng, 150, 1024)
        return {"kind": kind, "n": n, "w": w, "h": int(w * rng.uniform(0.6, 1.0)), "views": rng.randint(1, 8),
                "scene": rng.choice(["object", "orbit"]) if n <= 200_000 else "orbit"}
    if kind == "serve":
        lo = _log(rng, 50_000, 300_000)
        return {"kind": kind, "scenes": rng.randint(2, 8), "lo": lo, "hi": _log(rng, 2 * lo, 1_500_000),
                "requests": rng.randint(8, 24)}
    if kind == "loading":
        n, w = _log(rng, 100_000, 1_000_000), _log(rng, 400, 1920)
        return {"kind": kind, "n": n, "chunk": _log(rng, 4096, 65536), "w": w, "h": int(w * rng.uniform(0.5, 0.75))}
    return {"kind": "sort", "n": _log(rng, 1000, 6_000_000), "bits": rng.choice([8, 16, 24, 32, 32])}


# ---- inputs ------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _records(n, scene, sh, seed):
    """(n, 62) float32 file records: centre, normal, 48 SH coefficients, opacity logit, log-scales, rotation."""
    g, f32 = _generator(seed), dict(device="cuda", dtype=torch.float32)
    rec = torch.zeros((n, 62), **f32)
    if scene == "object":
        rec[:, 0:3] = 2.0 * torch.randn((n, 3), generator=g, **f32)
    else:  # 64 clusters (sigma 0.5-3) and 20% uniform background in a 40^3 box, in random order
        nb = n // 5
        centre = 40.0 * (torch.rand((64, 3), generator=g, **f32) - 0.5)
        sigma = 0.5 + 2.5 * torch.rand(64, generator=g, **f32)
        which = torch.randint(0, 64, (n,), generator=g, device="cuda")
        p = centre[which] + sigma[which, None] * torch.randn((n, 3), generator=g, **f32)
        p[:nb] = 40.0 * (torch.rand((nb, 3), generator=g, **f32) - 0.5)
        rec[:, 0:3] = p[torch.randperm(n, generator=g, device="cuda")]
    rec[:, 6:9] = 0.3 * torch.randn((n, 3), generator=g, **f32)
    if sh:
        k = 3 * (sh + 1) ** 2
        rec[:, 9:6 + k] = 0.05 * torch.randn((n, k - 3), generator=g, **f32)
    rec[:, 54] = 1.5 * torch.randn(n, generator=g, **f32)
    rec[:, 55:58] = -4.0 + 0.5 * torch.randn((n, 3), generator=g, **f32)
    q = torch.randn((n, 4), generator=g, **f32)
    rec[:, 58:62] = q / q.norm(dim=1, keepdim=True)
    return rec


def _look_at(eye, target):
    """Camera-to-world matrix, column-major float32[16]: right, up, forward, position."""
    f = target - eye
    f = f / np.linalg.norm(f)
    r = np.cross([0.0, 1.0, 0.0], f)
    r = r / np.linalg.norm(r)
    m = np.zeros((4, 4))
    m[0, :3], m[1, :3], m[2, :3], m[3, :3], m[3, 3] = r, np.cross(f, r), f, eye, 1.0
    return m.reshape(16).astype(np.float32)


def _poses(scene, count, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        az, el = rng.uniform(0, 2 * math.pi), rng.uniform(-math.pi / 6, math.pi / 6)
        radius = {"object": 8.0, "orbit": rng.uniform(6, 12), "fly": rng.uniform(18, 32)}[scene]
        eye = radius * np.array([math.cos(el) * math.cos(az), math.sin(el), math.cos(el) * math.sin(az)])
        out.append(_look_at(eye, rng.uniform(-3, 3, 3) if scene == "fly" else np.zeros(3)))
    return out


def _config(case):
    return Configuration(depth_sorting=DepthSorting[case["sorting"]], use_covariance_for_scale=case["covariance"],
                         use_unaligned_rectangles=case["rects"], spherical_harmonics_order=case["sh"],
                         max_splat_count=case["n"], frustum_culling_tolerance=CULL_TOL, ellipse_margin=MARGIN,
                         field_of_view_y=FOV, blend_mode=BlendMode[case["blend"]])


def _photos(views, w, h, seed):
    """Smooth seeded RGB images in [0, 1], (views, h, w, 3)."""
    small = torch.rand((views, 3, 12, 16), generator=_generator(seed), device="cuda")
    big = torch.nn.functional.interpolate(small, (h, w), mode="bilinear", align_corners=False)
    return big.permute(0, 2, 3, 1).contiguous()


def _fit_inputs(case, seed):
    rec = _records(case["n"], case["scene"], 3, seed)
    params = [rec[:, a:b].contiguous() for a, b in ((0, 3), (58, 62), (55, 58), (54, 55), (6, 54))]
    params[3] = params[3].reshape(-1)
    return params, _poses(case["scene"], case["views"], seed), _photos(case["views"], case["w"], case["h"], seed + 1)


def _fit_config(case):
    return dict(case, sorting="GPU", covariance=True, rects=True, sh=3, blend="FP32")


def _sort_inputs(case, seed):
    keys = torch.randint(0, 1 << case["bits"], (case["n"],), generator=_generator(seed), device="cuda")
    values = torch.randperm(case["n"], generator=_generator(seed + 1), device="cuda")
    return keys, values


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "loading"):
        if kind == "loading":
            case = dict(case, scene="orbit", sh=3, sorting="GPU", covariance=True, rects=True, blend="UNORM8")
        renderer = Renderer(_config(case))
        scene = Scene(renderer, case["n"])
        scene.load_chunk_device(_records(case["n"], case["scene"], case["sh"], seed))
        state = dict(case, renderer=renderer, scene=scene, camera=_poses(case["scene"], 1, seed)[0])
        if kind == "loading":
            count = min(case["chunk"], case["n"])
            state["start"] = (case["n"] - count) // 2
            state["records"] = _records(count, "orbit", 3, seed + 1).cpu().numpy()
        return state
    if kind == "fit":
        params, poses, photos = _fit_inputs(case, seed)
        renderers = [Renderer(_config(_fit_config(case))) for _ in poses]
        return dict(case, params=[p.requires_grad_(True) for p in params], poses=poses, photos=photos,
                    renderers=renderers)
    if kind == "serve":
        rng = np.random.default_rng(seed)
        sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["scenes"])).astype(int)
        sizes[0], sizes[-1] = case["hi"], case["lo"]
        server = Server(Configuration(max_splat_count=case["hi"], spherical_harmonics_order=3, field_of_view_y=FOV),
                        slots=8, max_width=1920, max_height=1080)
        ids = [server.add_scene(_records(int(n), "orbit", 3, seed + i)) for i, n in enumerate(sizes)]
        poses = _poses("orbit", case["requests"], seed)
        requests = []
        for k in range(case["requests"]):
            w, h = VIEWPORTS[k % len(VIEWPORTS)]
            requests.append((ids[rng.integers(len(ids))], poses[k], w, h, server.output_buffer(w, h)))
        return dict(case, server=server, queue=requests)
    keys, values = _sort_inputs(case, seed)
    keys = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32)
    renderer = Renderer(Configuration(max_splat_count=case["n"], max_pair_count=1024))
    return dict(case, renderer=renderer, keys=keys, values=values.to(torch.int32))


# ---- one pass ----------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "frame":
        return state["renderer"].render_frame(state["scene"], state["camera"], state["w"], state["h"])
    if kind == "loading":
        state["scene"].load_chunk(state["records"], state["start"])
        return state["renderer"].render_frame(state["scene"], state["camera"], state["w"], state["h"])
    if kind == "fit":
        params, w, h = state["params"], state["w"], state["h"]
        for p in params:
            p.grad = None
        if state["views"] == 1:
            image = render_raw(*params, state["renderers"][0], state["poses"][0], w, h)[None]
        else:
            image = render_raw_views(*params, state["renderers"], state["poses"], w, h)
        loss = l2_image_loss(image, state["photos"])
        loss.backward()
        return [image.detach(), loss.detach()] + [p.grad for p in params]
    if kind == "serve":
        for scene, camera, w, h, out in state["queue"]:
            state["server"].submit(scene, camera, w, h, out)
        state["server"].wait_all(len(state["queue"]))
        return [r[4] for r in state["queue"]]
    return list(state["renderer"].sort_pairs(state["keys"], state["values"], key_bits=state["bits"]))


# ---- the work of one pass ----------------------------------------------------------------------------
def _frame_work(n, w, h, sh, pixel_bytes, scene):
    """Every centre is read; a visible splat's rotation, scale, opacity and used SH coefficients too; the
    image is written.  About 500 operations per visible splat (cone, axes, colour) and 60 per blended
    pixel, of which a splat has some eight at full HD, in proportion to the viewport's height squared."""
    visible = n * {"object": 0.95, "orbit": 0.4, "fly": 0.6}[scene]
    blended = visible * 8.0 * (h / 1080.0) ** 2
    return {"bytes": 12.0 * n + visible * (32 + 12 * (sh + 1) ** 2) + float(pixel_bytes) * w * h,
            "flops": 15.0 * n + 500.0 * visible + 60.0 * blended}


def work(case):
    kind = case["kind"]
    if kind == "frame":
        return _frame_work(case["n"], case["w"], case["h"], case["sh"], 4 if case["blend"] == "UNORM8" else 16,
                           case["scene"])
    if kind == "loading":
        f = _frame_work(case["n"], case["w"], case["h"], 3, 4, "orbit")
        count = min(case["chunk"], case["n"])
        return {"bytes": f["bytes"] + count * (248 + 236), "flops": f["flops"] + 60.0 * count}
    if kind == "fit":
        # the parameters and targets are read, the images and the parameters' gradients written, once;
        # the backward's operations are about twice the frame's
        n, pixels = case["n"], case["views"] * case["w"] * case["h"]
        f = _frame_work(n, case["w"], case["h"], 3, 16, case["scene"])
        return {"bytes": 2.0 * 236 * n + (12.0 + 16.0) * pixels, "flops": 3.0 * case["views"] * f["flops"]}
    if kind == "serve":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])  # of a log-uniform size
        f = [_frame_work(mean, w, h, 3, 4, "orbit") for w, h in VIEWPORTS]
        return {k: case["requests"] * sum(x[k] for x in f) / len(f) for k in ("bytes", "flops")}
    return {"bytes": 16.0 * case["n"], "flops": 0.0}


# ---- the same in 64 bits -----------------------------------------------------------------------------
def _view_matrices(camera, w, h):
    """World-to-camera and view-projection matrices in float32 (rows), and the view plane's half extents.
    The depth keys and the visible set are defined in 32 bits, so their matrix is formed in 32 bits."""
    one = np.float32(1.0)
    c = camera.reshape(4, 4)  # rows: right, up, forward, position
    view = np.zeros((4, 4), np.float32)
    view[:3, :3], view[3, 3] = c[:3, :3], one
    for r in range(3):
        view[r, 3] = -((c[r, 0] * c[3, 0] + c[r, 1] * c[3, 1]) + c[r, 2] * c[3, 2])
    vh = np.float32(math.tan(float(np.float32(FOV) * np.float32(0.5))))
    vw = (np.float32(w) / np.float32(h)) * vh
    near, far = one, np.float32(1000.0)
    den = one / (near - far)
    proj = np.zeros((4, 4), np.float32)
    proj[0, 0], proj[1, 1], proj[2, 2], proj[2, 3], proj[3, 2] = one / vw, one / vh, -far * den, near * far * den, one
    vp = np.zeros((4, 4), np.float32)
    for i in range(4):
        for r in range(4):
            vp[r, i] = ((proj[r, 0] * view[0, i] + proj[r, 1] * view[1, i]) + proj[r, 2] * view[2, i]) + \
                proj[r, 3] * view[3, i]
    return view, vp, vw, vh


def _draw_order(centre, vp, sorting):
    """Indices of the drawn splats in drawing order, by the 32-bit frustum test and depth keys."""
    x, y, z = (t.contiguous() for t in centre.float().unbind(1))
    m = [[float(v) for v in row] for row in vp]
    hx, hy, hz, hw = (((m[r][0] * x + m[r][1] * y) + m[r][2] * z) + m[r][3] for r in range(4))
    if sorting == "CPU":
        rw = 1.0 / hw
        cx, cy, cz = hx * rw, hy * rw, hz * rw
    else:
        den = hw + 1e-7
        cx, cy, cz = hx / den, hy / den, hz / den
    seen = (cx.abs() < CULL_TOL) & (cy.abs() < CULL_TOL) & ((cz - 0.5).abs() < 0.5)
    if sorting == "CPU":
        key = cz.view(torch.int32).long()
    else:
        def word(v):  # truncation that saturates below at 0; NaN never passes the frustum test
            return v.clamp(min=0.0).nan_to_num().double().clamp(max=4294967295.0).long()
        key = ((word(cz * 65535.0) << 16) & 0xFFFFFFFF) | ((word((cx * 0.5 + 0.5) * 255.0) << 8) & 0xFFFFFFFF) | \
            word((cy * 0.5 + 0.5) * 255.0)
        if sorting == "GPU":
            seen &= key != 0xFFFFFFFF
        elif sorting == "GPU_INDIRECT_DRAW":
            seen &= (key >> 24) != 0xFF
    idx = seen.nonzero().reshape(-1)
    if sorting != "NONE":
        idx = idx[torch.sort(key[idx], stable=True).indices]
    return idx


SH_BASIS = (0.28209479177387814, -0.4886025119029199, 0.4886025119029199, -0.4886025119029199, 1.0925484305920792,
            -1.0925484305920792, 0.31539156525252005, -1.0925484305920792, 0.5462742152960396, -0.5900435899266435,
            2.890611442640554, -0.4570457994644658, 0.3731763325901154, -0.4570457994644658, 1.445305721320277,
            -0.5900435899266435)


def _colour(sh, d, order):
    x, y, z = d.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    one = torch.ones_like(x)
    terms = [one, y, z, x, x * y, y * z, 2 * zz - xx - yy, x * z, xx - yy, y * (3 * xx - yy), x * y * z,
             y * (4 * zz - xx - yy), z * (2 * zz - 3 * xx - 3 * yy), x * (4 * zz - xx - yy), z * (xx - yy),
             x * (xx - 3 * yy)]
    k = (order + 1) ** 2
    basis = torch.stack([c * t for c, t in zip(SH_BASIS[:k], terms[:k])], 1)
    return 0.5 + (basis[:, :, None] * sh.reshape(-1, 16, 3)[:, :k]).sum(1)


def _image64(centre, quat, scale, opacity, sh, camera, w, h, case):
    """(h, w, 4) float64 image (r, g, b, transmittance) of activated float64 parameters; differentiable."""
    f64 = dict(device="cuda", dtype=torch.float64)
    view, vp, vw, vh = _view_matrices(camera, w, h)
    idx = _draw_order(centre.detach(), vp, case["sorting"])
    vw, vh = float(vw), float(vh)
    p, q, s, a, coef = (t[idx] for t in (centre, quat, scale, opacity, sh))
    cam = torch.tensor(camera.reshape(4, 4), **f64)
    eye, axes = cam[3, :3], cam[:3, :3]  # rows: the camera's axes in the world
    # the rotation's matrix, column i the i-th axis as the path has it
    e, i, j, k = (math.sqrt(2.0) * t for t in q.unbind(1))
    rot = torch.stack([1 - j * j - k * k, i * j + k * e, i * k - j * e, i * j - k * e, 1 - i * i - k * k, j * k + i * e,
                       i * k + j * e, j * k - i * e, 1 - i * i - j * j], 1).reshape(-1, 3, 3).transpose(1, 2)
    # cone of rays that touch the ellipsoid: M = T2 ((1 - |l|^2) I + l l^T) T2^T, T2 = axes (rot / scale)
    t = rot / s[:, None, :]
    l = ((eye - p)[:, None, :] @ t)[:, 0]
    inner = (1.0 - (l * l).sum(1))[:, None, None] * torch.eye(3, **f64) + l[:, :, None] * l[:, None, :]
    t2 = axes @ t
    m = t2 @ inner @ t2.transpose(1, 2)
    xx, xy, xz, yy, yz, zz = m[:, 0, 0], m[:, 0, 1], m[:, 0, 2], m[:, 1, 1], m[:, 1, 2], m[:, 2, 2]
    disc = xx * yy - xy * xy
    t0, t1 = (xy * yz - yy * xz) / disc, (xy * xz - xx * yz) / disc
    diff = xx - yy
    rc = 0.5 * torch.sqrt(diff * diff / (diff * diff + 4 * xy * xy))
    rj, rk = torch.sqrt((0.5 - rc).clamp(min=1e-34)), -torch.sqrt(0.5 + rc) * torch.sign(xy) * torch.sign(diff)
    flip = torch.where((xy < 0) | (diff < 0), -1.0, 1.0)
    rj, rk = rj * flip, rk * flip
    rj, rk = torch.where(diff < 0, -rk, rj), torch.where(diff < 0, rj, rk)
    if case["covariance"]:
        v = (p - eye) @ axes.T
        vx, vy, vz = (v[:, 0] / v[:, 2]).clamp(-1, 1), (v[:, 1] / v[:, 2]).clamp(-1, 1), v[:, 2]
        zero = torch.zeros_like(vz)
        jac = torch.stack([torch.stack([1 / vz, zero, -vx / vz], 1), torch.stack([zero, 1 / vz, -vy / vz], 1)], 1)
        half = jac @ axes @ (rot * s[:, None, :])
        cov = half @ half.transpose(1, 2)
        cxx, cxy, cyy = cov[:, 0, 0], cov[:, 0, 1], cov[:, 1, 1]
        b = torch.sqrt((cxx - cyy) ** 2 + 4 * cxy * cxy)
        ax0, ax1 = torch.sqrt(0.5 * (cxx + cyy + b)), torch.sqrt((0.5 * (cxx + cyy - b)).clamp(min=1e-300))
    else:
        d = 2 * xy * rj * rk
        f = zz - (xx * t0 * t0 + yy * t1 * t1 + 2 * xy * t0 * t1)
        ax0 = torch.sqrt((f / (xx * rk * rk + yy * rj * rj - d)).abs())
        ax1 = torch.sqrt((f / (xx * rj * rj + yy * rk * rk + d)).abs())
    bias = 0.2 * vw / w
    sa, sb = bias + ax0, bias + ax1
    ux, uy, wx, wy = rk * sa, -rj * sa, rj * sb, rk * sb  # the rectangle's half axes
    det = ux * wy - uy * wx
    direction = p - eye
    rgb = _colour(coef, direction / direction.norm(dim=1, keepdim=True), case["sh"])
    # pixels of each splat's box
    psx, psy = 2 * vw / w, 2 * vh / h
    with torch.no_grad():
        if case["rects"]:
            ex, ey = MARGIN * (ux.abs() + wx.abs()), MARGIN * (uy.abs() + wy.abs())
        else:
            ex = ey = MARGIN * torch.sqrt(torch.maximum(ux * ux + uy * uy, wx * wx + wy * wy))
        px, py = (t0 + vw) / psx, (vh - t1) / psy
        x0, x1 = torch.ceil(px - ex / psx - 0.5), torch.floor(px + ex / psx - 0.5)
        y0, y1 = torch.ceil(py - ey / psy - 0.5), torch.floor(py + ey / psy - 0.5)
        ok = torch.isfinite(x0 + x1 + y0 + y1 + det) & (det != 0) & (a >= 1.0 / 255.0)
        x0, x1 = x0.nan_to_num().clamp(0, w), x1.nan_to_num().clamp(-1, w - 1)
        y0, y1 = y0.nan_to_num().clamp(0, h), y1.nan_to_num().clamp(-1, h - 1)
        bw, bh = (x1 - x0 + 1).clamp(min=0).long(), (y1 - y0 + 1).clamp(min=0).long()
        count = torch.where(ok, bw * bh, torch.zeros_like(bw))
        who = torch.repeat_interleave(torch.arange(len(idx), device="cuda"), count)
        at = torch.arange(len(who), device="cuda") - (count.cumsum(0) - count)[who]
        gx, gy = x0[who].long() + at % bw[who], y0[who].long() + at // bw[who]

    def falloff(who, gx, gy):
        dx, dy = (gx + 0.5) * psx - vw - t0[who], vh - (gy + 0.5) * psy - t1[who]
        u, v = (wy[who] * dx - wx[who] * dy) / det[who], (ux[who] * dy - uy[who] * dx) / det[who]
        inside = (u.abs() <= MARGIN) & (v.abs() <= MARGIN) if case["rects"] else \
            (dx.abs() <= ex[who]) & (dy.abs() <= ex[who])
        return inside, a[who] * torch.exp(-0.5 * (u * u + v * v))

    with torch.no_grad():  # blended pixels, by pixel and then in drawing order
        inside, alpha = falloff(who, gx, gy)
        keep = inside & (alpha >= 1.0 / 255.0)
        who, gx, gy = who[keep], gx[keep], gy[keep]
        pixel, by = torch.sort(gy * w + gx, stable=True)
        who, gx, gy = who[by], gx[by], gy[by]
        first = torch.searchsorted(pixel, pixel)

    def before(alpha):  # log of the transmittance in front of each entry
        sums = torch.cat([torch.zeros(1, **f64), torch.log1p(-alpha.clamp(0, 1 - 1e-12)).cumsum(0)])
        return sums[:-1] - sums[first]

    with torch.no_grad():  # a pixel stops once its transmittance falls below 1e-4
        keep = before(falloff(who, gx, gy)[1]) >= math.log(1e-4)
        who, gx, gy, pixel = who[keep], gx[keep], gy[keep], pixel[keep]
        first = torch.searchsorted(pixel, pixel)
    alpha = falloff(who, gx, gy)[1].clamp(max=1.0)
    weight = torch.exp(before(alpha))
    image = torch.zeros((h * w, 3), **f64).index_add(0, pixel, (rgb[who] * alpha[:, None]).clamp(0, 1) * weight[:, None])
    left = torch.zeros(h * w, **f64).index_add(0, pixel, torch.log1p(-alpha.clamp(max=1 - 1e-12)))
    return torch.cat([image, torch.exp(left)[:, None]], 1).reshape(h, w, 4)


def _activate64(centre, quat, logs, logit):
    mean = logs.mean(1, keepdim=True)
    clamped = torch.minimum(torch.maximum(logs, mean - 5.0), mean + 5.0)
    return centre, quat / quat.norm(dim=1, keepdim=True), torch.exp(clamped), torch.sigmoid(logit)


def exact(case, seed):
    if case["kind"] == "sort":
        keys, values = _sort_inputs(case, seed)
        order = torch.sort(keys, stable=True).indices
        keys = keys[order]
        return [torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32), values[order].to(torch.int32)]
    if case["kind"] == "frame" and case["blend"] == "FP32" and case["n"] <= 2_000_000:
        rec = _records(case["n"], case["scene"], case["sh"], seed).double()
        p = _activate64(rec[:, 0:3], rec[:, 58:62], rec[:, 55:58], rec[:, 54])
        camera = _poses(case["scene"], 1, seed)[0]
        with torch.no_grad():
            return _image64(*p, rec[:, 6:54], camera, case["w"], case["h"], case)
    if case["kind"] == "fit":
        params, poses, photos = _fit_inputs(case, seed)
        params = [p.double().requires_grad_(True) for p in params]
        images, loss = [], 0.0
        for camera, photo in zip(poses, photos):  # one view at a time: its gradients are added to the others'
            image = _image64(*_activate64(*params[:4]), params[4], camera, case["w"], case["h"], _fit_config(case))
            one = ((image[..., :3] - photo.double()) ** 2).sum()
            one.backward()
            images.append(image.detach())
            loss = loss + one.detach()
        return [torch.stack(images), loss] + [p.grad for p in params]
    return None
