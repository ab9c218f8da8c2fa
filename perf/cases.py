"""The work that programs have this library do, as measurable cases.

A case is one of six kinds of call:

step    the training step: render, loss, adjoint, parameter chain and Adam over
        one or several views (SplatTrainer.accumulate + apply, the two halves
        of a step, so that the gradients can be returned); with `scenes` > 1
        independent scenes of uneven sizes in one batch, with `frame_width`
        8-bit camera frames staged from page-locked host memory one step ahead
device  a host framework's call on its own tensors: one view's forward and
        adjoint (pxs_render_and_accumulate_device)
host    the same call on host arrays (render_and_accumulate)
render  a view of a trained cloud (pxs_trainer_render) into page-locked memory
loss    the photometric loss and its gradient on a framework's images
        (pxs_photometric_loss_static)
adam    the optimiser step on a framework's tensors (pxs_adam_device)

exact() restates each in 64 bits with plain torch, where that is quick enough.
"""
import ctypes as ct
import math

import numpy as np
import torch

import parallax_b200 as px
from parallax_b200.data_parallel import device_tensors

REST = {0: 0, 1: 3, 2: 8, 3: 15}
C0 = 0.28209479177387814
SCENE_SIZES = ((320, 240), (640, 480), (1280, 720))


def listed():
    return [
        # the smallest training call there is, as an engine's SplatBackend makes
        # it: 4k gaussians SH3, 128x128, host arrays in and out (latency counts)
        dict(name="host_4k_128", kind="host", n=4000, sh=3, width=128, height=128, ssim=0.2),
        # one step at the size the CPU trainer can still do: 20k gaussians SH0,
        # one 320x240 view (launches count)
        dict(name="step_20k_320", kind="step", n=20000, sh=0, views=1, width=320, height=240,
             scenes=1, frame_width=0),
        # a few small views of ragged size and a cloud of ragged count
        dict(name="step_37k_ragged", kind="step", n=37813, sh=1, views=3, width=637, height=423,
             scenes=1, frame_width=0),
        # the phone-shape step: one 1280x720 view, SH3, the count that a run
        # from 200k gaussians has after densification
        dict(name="step_152k_720p", kind="step", n=151721, sh=3, views=1, width=1280, height=720,
             scenes=1, frame_width=0),
        # four views a step whose 8-bit frames arrive wider than the views and
        # are downscaled on the device
        dict(name="step_100k_frames", kind="step", n=100000, sh=2, views=4, width=1280,
             height=720, scenes=1, frame_width=1920),
        # many independent scans trained together, sizes far apart
        dict(name="step_10_scenes", kind="step", n=150000, sh=3, views=4, width=1280, height=720,
             scenes=10, frame_width=0),
        # the full-size batch: 1M gaussians SH3, 8 views of 1920x1440
        dict(name="step_1m_8views", kind="step", n=1000000, sh=3, views=8, width=1920,
             height=1440, scenes=1, frame_width=0),
        # a framework's own training loop, L1 only, an odd view on a background
        dict(name="device_60k_odd", kind="device", n=60001, sh=2, width=801, height=603,
             ssim=0.0),
        # looking at a trained cloud
        dict(name="render_300k", kind="render", n=300000, sh=3, width=1600, height=1200),
        # scoring a batch of images, odd sizes
        dict(name="loss_4x719p", kind="loss", views=4, width=1279, height=719, ssim=0.2),
        # the optimiser alone at an odd count (counts are odd after densification)
        dict(name="adam_333k", kind="adam", n=333333, sh=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "device", "host", "render", "loss",
                       "adam"])
    sh = rng.choice([0, 1, 2, 3, 3, 3])
    width = _log(rng, 128, 1920)
    height = max(96, int(width * rng.choice([0.5625, 0.75, 0.75, 1.0, 1.3333])))
    if kind == "step":
        scenes = rng.choice([1, 1, 1, 1, _log(rng, 2, 12)])
        n = _log(rng, 3000, 800000 if scenes == 1 else 100000)
        # at most the pixels of four of the largest views
        views = min(rng.choice([1, 1, 2, 4, 6]), max(1, 11_000_000 // (width * height)))
        if scenes > 1:
            views, width, height = min(views, 4), 1280, 720
        frame = rng.choice([0, 0, width, int(width * 1.5)]) if scenes == 1 else 0
        return dict(kind=kind, n=n, sh=sh, views=views, width=width, height=height,
                    scenes=scenes, frame_width=frame)
    if kind == "device":
        return dict(kind=kind, n=_log(rng, 3000, 600000), sh=sh, width=width, height=height,
                    ssim=rng.choice([0.0, 0.2, 0.2]))
    if kind == "host":
        return dict(kind=kind, n=_log(rng, 2000, 40000), sh=sh, width=min(width, 640),
                    height=min(height, 480), ssim=0.2)
    if kind == "render":
        return dict(kind=kind, n=_log(rng, 3000, 800000), sh=sh, width=width, height=height)
    if kind == "loss":
        return dict(kind=kind, views=rng.choice([1, 2, 4, 8]), width=width, height=height,
                    ssim=rng.choice([0.2, 0.2, 0.5, 0.0]))
    return dict(kind=kind, n=_log(rng, 3000, 1000000), sh=sh)


# ------------------------------------------------------------------ inputs


def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    return g


def _cloud(seed, salt, n, sh):
    """Parameters (P x n float32, component-major): positions in a cube, sizes
    log-normal, any orientation, opacities around one half, grey colours."""
    g = _generator(seed, salt)

    def normal(rows):
        return torch.randn(rows, n, generator=g, device="cuda")

    q = normal(4)
    return torch.cat([
        torch.rand(3, n, generator=g, device="cuda") * 2 - 1,
        -4.0 + 0.5 * normal(3),
        q / q.norm(dim=0, keepdim=True),
        normal(1),
        0.1 / C0 * normal(3),
        0.1 * normal(3 * REST[sh]),
    ]).contiguous()


def _images(seed, salt, count, width, height):
    """Photograph-like 8-bit images (count, H, W, 3): smooth shapes with detail."""
    g = _generator(seed, salt)
    out = torch.zeros(count, 3, height, width, device="cuda")
    for cells, gain in ((6, 0.35), (40, 0.12)):
        coarse = torch.rand(count, 3, cells, cells, generator=g, device="cuda") - 0.5
        out += gain * torch.nn.functional.interpolate(coarse, size=(height, width),
                                                      mode="bicubic", align_corners=False)
    out += 0.4 + 0.02 * torch.randn(count, 3, height, width, generator=g, device="cuda")
    return (out.clamp(0, 1) * 255).round().to(torch.uint8).permute(0, 2, 3, 1).contiguous()


def _poses(seed, count, width, height):
    """(K, R, t) of cameras around the cloud, looking at its middle."""
    rs = np.random.default_rng(seed + 17)
    f = width * 0.5 / math.tan(math.radians(60.0) * 0.5)
    K = (f, f, width * 0.5 - 0.5, height * 0.5 - 0.5)
    spin = rs.uniform(0.0, 2.0 * math.pi)
    poses = []
    for i in range(count):
        y = 0.9 - 1.8 * (i + 0.5) / count
        r, a = math.sqrt(1.0 - y * y), math.pi * (3.0 - math.sqrt(5.0)) * i + spin
        eye = 3.0 * np.array([r * math.cos(a), y, r * math.sin(a)])
        forward = -eye / np.linalg.norm(eye)
        right = np.cross(forward, [0.0, 1.0, 0.0])
        right /= np.linalg.norm(right)
        R = np.stack([right, np.cross(forward, right), forward])
        poses.append((K, R, -R @ eye))
    return poses


def _views(poses, width, height):
    return [px.SplatView(K, width, height, R, t) for K, R, t in poses]


def _scene_shapes(case):
    """(gaussians, width, height) of each scene: counts spread over the
    logarithm up to `n`, not in order of size, at three frame sizes."""
    if case["scenes"] == 1:
        return [(case["n"], case["width"], case["height"])]
    low = math.log(max(1000, case["n"] // 30))
    shapes = []
    for s in range(case["scenes"]):
        at = (s * 7 % case["scenes"] + 0.5) / case["scenes"]
        n = int(math.exp(low + at * (math.log(case["n"]) - low)))
        shapes.append((n,) + SCENE_SIZES[s % 3])
    return shapes


def _options(background=(0.0, 0.0, 0.0), sh=0):
    return px.RasterOptions(background=background, sh_degree=sh)


BACKGROUND = (0.2, 0.3, 0.1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _prepare_step(case, seed)
    w, h = case.get("width", 0), case.get("height", 0)
    if kind == "adam":
        n, rows = case["n"], 14 + 3 * REST[case["sh"]]
        g = _generator(seed, 3)
        grads = 1e-4 * torch.randn(rows, n, generator=g, device="cuda")
        m = 1e-4 * torch.randn(rows, n, generator=g, device="cuda")
        v = 1e-8 * torch.rand(rows, n, generator=g, device="cuda")
        # small rates, as late in a run: repeated passes do the same work
        lr = (ct.c_float * 6)(5.3e-6, 5e-7, 1e-7, 5e-6, 2.5e-7, 1.25e-8)
        return dict(kind=kind, ctx=px.Context(0), params=_cloud(seed, 1, n, case["sh"]), grads=grads,
                    m=m, v=v, n=n, rest=REST[case["sh"]], lr=lr)
    if kind == "loss":
        a = _images(seed, 4, case["views"], w, h).float() / 255
        noise = torch.randn(a.shape, generator=_generator(seed, 5), device="cuda")
        b = (a + 0.05 * noise).clamp(0, 1)  # the rendering: near its photograph
        return dict(kind=kind, rendered=b, target=a, grad=torch.empty_like(a),
                    per_view=torch.empty(case["views"], device="cuda"),
                    loss=torch.empty(1, device="cuda"), views=case["views"], width=w, height=h,
                    ssim=case["ssim"], error=ct.create_string_buffer(256))
    params = _cloud(seed, 1, case["n"], case["sh"])
    rest = REST[case["sh"]]
    view = _views(_poses(seed, 1, w, h), w, h)[0]
    if kind == "render":
        config = px.TrainConfig(iterations=1 << 30, sh_degree=case["sh"], sh_increase_interval=0,
                                densify_from_iteration=(1 << 30) + 1,
                                densify_until_iteration=1 << 30)
        trainer = px.SplatTrainer(px.GaussianCloud(params.cpu().numpy(), case["sh"], rest), [],
                                  config)
        return dict(kind=kind, trainer=trainer, camera=view.camera(),
                    options=_options(BACKGROUND, case["sh"]),
                    rgb=torch.empty(h, w, 3, pin_memory=True),
                    transmittance=torch.empty(h, w, pin_memory=True))
    target = (_images(seed, 2, 1, w, h)[0].float() / 255).contiguous()
    if kind == "host":
        return dict(kind=kind, ctx=px.Context(0), camera=view.camera(), ssim=case["ssim"],
                    cloud=px.GaussianCloud(params.cpu().numpy(), case["sh"], rest),
                    options=_options(BACKGROUND, case["sh"]),
                    target=target.cpu().numpy().reshape(-1))
    ctx, stream = px.Context(0), torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)  # the framework's stream
    cloud = px._abi.Cloud(params.data_ptr(), case["n"], rest, case["sh"])
    grads = torch.zeros_like(params)
    screen = torch.zeros(case["n"], device="cuda")
    visible = torch.zeros(case["n"], dtype=torch.int32, device="cuda")
    gradients = px._abi.Gradients(grads.data_ptr(), screen.data_ptr(), visible.data_ptr())
    return dict(kind=kind, ctx=ctx, params=params, cloud=cloud, camera=view.camera(),
                options=_options(BACKGROUND, case["sh"]), target=target, ssim=case["ssim"],
                grads=grads, screen=screen, visible=visible, gradients=gradients,
                stream=stream, loss=torch.zeros(1, device="cuda"))


def _prepare_step(case, seed):
    sh, rest = case["sh"], REST[case["sh"]]
    # rates as late in a run and smaller: repeated passes stay at one point of
    # the training and do the same work
    config = px.TrainConfig(
        iterations=1 << 30, sh_degree=sh, sh_increase_interval=0,
        position_lr_initial=1.6e-6, position_lr_final=1.6e-6, dc_lr=2.5e-7, opacity_lr=5e-6,
        scale_lr=5e-7, rotation_lr=1e-7, densify_from_iteration=(1 << 30) + 1,
        densify_until_iteration=1 << 30, opacity_reset_interval=0)
    # with staged frames two groups of views take turns: one trains while the
    # other's frames are copied
    groups = 2 if case["frame_width"] else 1
    count = case["views"] * groups
    clouds, scene_views = [], []
    for s, (n, w, h) in enumerate(_scene_shapes(case)):
        clouds.append(px.GaussianCloud(_cloud(seed, 100 + s, n, sh).cpu().numpy(), sh, rest))
        images = (_images(seed, 200 + s, count, w, h).float() / 255).cpu().numpy()
        scene_views.append(list(zip(_views(_poses(seed + s, count, w, h), w, h), images)))
    if len(clouds) == 1:
        trainer = px.SplatTrainer(clouds[0], scene_views[0], config)
    else:
        trainer = px.SplatTrainer.from_scenes(clouds, scene_views, config)
    total = sum(c.count for c in clouds)
    block = device_tensors([trainer.reduction_block() + ("float32",)])[0]
    state = dict(kind="step", trainer=trainer, block=block, total=total, rows=14 + 3 * rest,
                 stream=torch.cuda.ExternalStream(trainer.stream()), turn=0,
                 ids=[list(range(g * case["views"], (g + 1) * case["views"]))
                      for g in range(groups)], frames=None)
    if len(clouds) > 1:
        state["ids"] = [list(range(case["views"] * len(clouds)))]
    if case["frame_width"]:
        fw = case["frame_width"]
        fh = int(round(case["height"] * fw / case["width"]))
        pinned = torch.empty(count, fh, fw, 3, dtype=torch.uint8, pin_memory=True)
        pinned.copy_(_images(seed, 300, count, fw, fh))
        state["frames"] = [[pinned[i].numpy() for i in ids] for ids in state["ids"]]
        state["sizes"] = [(fw, fh)] * case["views"]
        state["pinned"] = pinned
    return state


# -------------------------------------------------------------------- runs


def run(s):
    kind, lib = s["kind"], px.lib()
    if kind == "step":
        trainer, k = s["trainer"], s["turn"]
        if s["frames"]:
            s["turn"] = 1 - k
            trainer.stage_images(s["ids"][1 - k], s["frames"][1 - k], s["sizes"])
        loss = trainer.accumulate(s["ids"][k])
        with torch.cuda.stream(s["stream"]):
            got = s["block"].clone()
        trainer.apply(loss)
        n, rows = s["total"], s["rows"]
        return {"loss": loss, "gradients": got[: rows * n].view(rows, n),
                "screen": got[rows * n: (rows + 1) * n],
                "visible": got[(rows + 1) * n: (rows + 2) * n]}
    if kind == "device":
        with torch.cuda.stream(s["stream"]):
            s["grads"].zero_()
            s["screen"].zero_()
            s["visible"].zero_()
        s["ctx"].check(lib.pxs_render_and_accumulate_device(
            s["ctx"].handle, ct.byref(s["cloud"]), ct.byref(s["camera"]), ct.byref(s["options"]),
            s["target"].data_ptr(), s["ssim"], ct.byref(s["gradients"]), s["loss"].data_ptr()))
        return {"loss": s["loss"], "gradients": s["grads"], "screen": s["screen"],
                "visible": s["visible"]}
    if kind == "host":
        grads = px.SplatGradients.zeros(s["cloud"])
        loss = px.render_and_accumulate(s["cloud"], s["camera"], s["options"], s["target"],
                                        s["ssim"], grads, s["ctx"])
        return {"loss": loss, "gradients": grads.params, "screen": grads.screen_gradient,
                "visible": grads.visible_count}
    if kind == "render":
        t = s["trainer"]
        t._check(lib.pxs_trainer_render(t.handle, ct.byref(s["camera"]), ct.byref(s["options"]),
                                        s["rgb"].data_ptr(), s["transmittance"].data_ptr()))
        return {"rgb": s["rgb"], "transmittance": s["transmittance"]}
    if kind == "loss":
        status = lib.pxs_photometric_loss_static(
            s["rendered"].data_ptr(), s["target"].data_ptr(), s["width"], s["height"],
            s["views"], s["ssim"], s["grad"].data_ptr(), s["per_view"].data_ptr(),
            s["loss"].data_ptr(), torch.cuda.current_stream().cuda_stream, s["error"], 256)
        if status:
            raise RuntimeError(s["error"].value.decode())
        return {"loss": s["loss"], "per_view": s["per_view"], "gradient": s["grad"]}
    s["ctx"].check(lib.pxs_adam_device(
        s["ctx"].handle, s["params"].data_ptr(), s["grads"].data_ptr(), s["m"].data_ptr(),
        s["v"].data_ptr(), s["n"], s["rest"], s["lr"], 0.9, 0.999, 1e-15, 0.5, 0.25, 0))
    return {"params": s["params"], "m": s["m"], "v": s["v"]}


# -------------------------------------------------------------------- work


def work(case):
    """Inputs read and outputs written once, and the arithmetic of what the
    pixels cannot do without: about 100 operations for each splat that a pixel
    takes in the forward pass and its adjoint together (17 + 10 and 17 + 58),
    two 11-tap blurs each way of the loss's four and three planes per channel."""
    kind, sh = case["kind"], case.get("sh", 0)
    rows = 14 + 3 * REST[sh]
    blur = 3 * 7 * 2 * 2 * 11
    if kind == "adam":
        return {"bytes": 28.0 * rows * case["n"], "flops": 16.0 * rows * case["n"]}
    if kind == "loss":
        pixels = case["views"] * case["width"] * case["height"]
        return {"bytes": 36.0 * pixels, "flops": (blur if case["ssim"] > 0 else 12.0) * pixels}
    nbytes = flops = 0.0
    if kind == "step":
        for n, w, h in _scene_shapes(case):
            pixels = case["views"] * w * h
            nbytes += 28.0 * rows * n + 4.0 * rows * n + 12.0 * pixels
            flops += 102.0 * _taken(n, case["views"], w, h) + blur * pixels + 16.0 * rows * n
        if case["frame_width"]:
            nbytes += 3.0 * case["views"] * case["height"] * case["frame_width"] ** 2 / case["width"]
        return {"bytes": nbytes, "flops": flops}
    w, h = case["width"], case["height"]
    taken = _taken(case["n"], 1, w, h)
    if kind == "render":
        return {"bytes": 4.0 * rows * case["n"] + 16.0 * w * h, "flops": 27.0 * taken}
    return {"bytes": 8.0 * rows * case["n"] + 12.0 * w * h,
            "flops": 102.0 * taken + (blur if case["ssim"] > 0 else 12.0) * w * h}


def _taken(n, views, w, h):
    """About how many splats the pixels take: a splat of the usual size covers
    4 pi sigma^2 pixels, and a pixel is full after about 70."""
    sigma = 0.02 * w / (2 * math.tan(math.radians(30))) / 3.0
    return views * min(70.0 * w * h, n * 4 * math.pi * (sigma * sigma + 0.3))


# ----------------------------------------------------------- 64-bit restatement


def exact(case, seed):
    kind = case["kind"]
    if kind == "adam":
        return _exact_adam(prepare(case, seed))
    if kind == "loss":
        s = prepare(case, seed)
        per_view, grads = [], []
        for k in range(case["views"]):
            r = s["rendered"][k].double().requires_grad_()
            value = _loss64(r, s["target"][k].double(), case["ssim"])
            value.backward()
            per_view.append(value.detach())
            grads.append(r.grad)
        per_view = torch.stack(per_view)
        return {"loss": per_view.mean().reshape(1), "per_view": per_view,
                "gradient": torch.stack(grads)}
    tiles = case.get("views", 1) * (-(-case["width"] // 16)) * (-(-case["height"] // 16))
    if case.get("scenes", 1) > 1 or tiles > (8000 if kind == "render" else 4000):
        return None  # too slow in 64 bits
    salt = 100 if kind == "step" else 1
    params = _cloud(seed, salt, case["n"], case["sh"]).double().requires_grad_()
    w, h = case["width"], case["height"]
    count = case.get("views", 1) * (2 if case.get("frame_width") else 1)
    poses = _poses(seed, count, w, h)[: case.get("views", 1)]
    background = (0.0, 0.0, 0.0) if kind == "step" else BACKGROUND
    if kind == "render":
        rgb, transmittance = _render64(params.detach(), case["sh"], poses[0], w, h, background)
        return {"rgb": rgb, "transmittance": transmittance}
    images = _images(seed, 200 if kind == "step" else 2, count, w, h).float() / 255
    losses = []
    for pose, target in zip(poses, images):
        losses.append(_render64(params, case["sh"], pose, w, h, background, target.double(),
                                case.get("ssim", 0.2)))
    loss = sum(losses) / len(losses)
    if kind == "device":
        loss = torch.tensor([loss])
    return {"loss": loss, "gradients": params.grad, "screen": None, "visible": None}


def _exact_adam(s):
    p, g, m, v = (s[k].double() for k in ("params", "grads", "m", "v"))
    b1, b2 = float(np.float32(0.9)), float(np.float32(0.999))
    rate = torch.empty(p.shape[0], 1, dtype=torch.float64, device=p.device)
    for lo, hi, k in ((0, 3, 0), (3, 6, 1), (6, 10, 2), (10, 11, 3), (11, 14, 4),
                      (14, p.shape[0], 5)):
        rate[lo:hi] = float(s["lr"][k])
    m = b1 * m + (1 - b1) * g
    v = b2 * v + (1 - b2) * g * g
    p = p - rate * (m / 0.5) / ((v / 0.25).sqrt() + 1e-15)
    p[6:10] = p[6:10] / p[6:10].norm(dim=0, keepdim=True)
    return {"params": p, "m": m, "v": v}


def _blur64(x):
    """11 taps of a 1.5-pixel Gaussian along both axes of (..., H, W), zero outside."""
    k = torch.exp(-0.5 * torch.arange(-5, 6, dtype=torch.float64) ** 2 / 2.25)
    k = (k / k.sum()).tolist()
    for axis in (-1, -2):
        pad = (5, 5, 0, 0) if axis == -1 else (0, 0, 5, 5)
        y, size = torch.nn.functional.pad(x, pad), x.shape[axis]
        x = sum(k[i] * y.narrow(axis, i, size) for i in range(11))
    return x


def _loss64(rendered, target, weight):
    l1 = (rendered - target).abs().mean()
    if weight <= 0:
        return l1
    x, y = rendered.permute(2, 0, 1), target.permute(2, 0, 1)
    mx, my = _blur64(x), _blur64(y)
    vx, vy, c = _blur64(x * x) - mx * mx, _blur64(y * y) - my * my, _blur64(x * y) - mx * my
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    ssim = (2 * mx * my + c1) * (2 * c + c2) / ((mx * mx + my * my + c1) * (vx + vy + c2))
    return (1 - weight) * l1 + weight * (1 - ssim.mean())


def _sh64(degree, d):
    x, y, z = d
    xx, yy, zz = x * x, y * y, z * z
    basis = []
    if degree > 0:
        basis += [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if degree > 1:
        basis += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
                  0.31539156525252005 * (2 * zz - xx - yy), -1.0925484305920792 * x * z,
                  0.5462742152960396 * (xx - yy)]
    if degree > 2:
        basis += [-0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z,
                  -0.4570457994644658 * y * (4 * zz - xx - yy),
                  0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
                  -0.4570457994644658 * x * (4 * zz - xx - yy),
                  1.445305721320277 * z * (xx - yy), -0.5900435899266435 * x * (xx - 3 * yy)]
    return basis


def _project64(p, sh, pose, w, h):
    """Screen means (2), conics (3), colours (3), opacity, depth, radius and determinant."""
    K, R, t = pose

    def f32(v):
        return torch.as_tensor(np.asarray(v, np.float32).astype(np.float64), device=p.device)

    fx, fy, cx, cy = (float(np.float32(v)) for v in K)
    lim = [1.3 * float(np.float32(0.5 * w / K[0])), 1.3 * float(np.float32(0.5 * h / K[1]))]
    W, centre = f32(R), f32(-R.T @ t)
    q = p[6:10] / p[6:10].norm(dim=0, keepdim=True)
    qw, x, y, z = q
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - qw * z), 2 * (x * z + qw * y),
                       2 * (x * y + qw * z), 1 - 2 * (x * x + z * z), 2 * (y * z - qw * x),
                       2 * (x * z - qw * y), 2 * (y * z + qw * x),
                       1 - 2 * (x * x + y * y)]).view(3, 3, -1)
    M = rot * torch.exp(p[3:6])[None]
    pc = W @ p[0:3] + f32(t)[:, None]
    depth = pc[2]
    u = [(pc[i] / depth).clamp(-lim[i], lim[i]) for i in (0, 1)]
    zero = torch.zeros_like(depth)
    J = torch.stack([torch.stack([fx / depth, zero, -fx * u[0] / depth]),
                     torch.stack([zero, fy / depth, -fy * u[1] / depth])])
    A = torch.einsum("ijn,jk,kln->iln", J, W, M)
    cov = torch.einsum("ikn,jkn->ijn", A, A)
    a, b, c = cov[0, 0] + 0.3, cov[0, 1], cov[1, 1] + 0.3
    det = a * c - b * b
    mean = torch.stack([fx * pc[0] / depth + cx, fy * pc[1] / depth + cy])
    mid = 0.5 * (a + c)
    radius = 3 * (mid + (mid * mid - det).clamp(min=0).sqrt()).clamp(min=1e-6).sqrt().detach()
    off = p[0:3] - centre[:, None]
    colour = 0.5 + C0 * p[11:14]
    for k, value in enumerate(_sh64(sh, off / off.norm(dim=0, keepdim=True))):
        colour = colour + value * p[14 + k:: REST[sh]][:3]
    return (mean, torch.stack([c / det, -b / det, a / det]), colour.clamp(min=0),
            torch.sigmoid(p[10]), depth.detach(), radius, det.detach())


def _render64(params, sh, pose, w, h, background, target=None, weight=0.2):
    """The image and transmittance, or with a target the loss, its gradient added
    to params.grad. Tiles of 16x16 pixels take the splats whose 3-sigma box
    touches them, near to far."""
    with torch.no_grad():
        mean, _, _, opacity, depth, radius, det = _project64(params, sh, pose, w, h)
        seen = ((depth >= 0.01) & (det > 1e-12) & (mean[0] + radius >= 0) & (mean[0] - radius < w)
                & (mean[1] + radius >= 0) & (mean[1] - radius < h) & (opacity >= 1 / 255))
        index = seen.nonzero()[:, 0]
        index = index[depth[index].argsort(stable=True)]
    projected = _project64(params[:, index], sh, pose, w, h)
    leaves = [x.detach() for x in projected[:4]]
    mean, radius = leaves[0], projected[5]
    lo = ((mean - radius) / 16).floor()
    hi = ((mean + radius) / 16).floor()
    back = torch.tensor(background, dtype=torch.float64, device=params.device)
    tiles = [(tx, ty) for ty in range(-(-h // 16)) for tx in range(-(-w // 16))]

    def members():
        for ty in range(-(-h // 16)):
            row = ((lo[1] <= ty) & (hi[1] >= ty)).nonzero()[:, 0]
            first, last = lo[0][row], hi[0][row]
            for tx in range(-(-w // 16)):
                yield row[(first <= tx) & (last >= tx)]

    def tile(tx, ty, ids, values):
        xs = torch.arange(tx * 16, min(w, tx * 16 + 16), device=params.device) + 0.5
        ys = torch.arange(ty * 16, min(h, ty * 16 + 16), device=params.device) + 0.5
        m, conic, colour, opacity = (v[..., ids] for v in values)
        dx = (xs[None, :, None] - m[0]).expand(len(ys), -1, -1)
        dy = (ys[:, None, None] - m[1]).expand(-1, len(xs), -1)
        power = -0.5 * (conic[0] * dx * dx + conic[2] * dy * dy) - conic[1] * dx * dy
        alpha = (opacity * torch.exp(power)).clamp(max=0.99)
        alpha = torch.where((power > 0) | (alpha < 1 / 255), torch.zeros_like(alpha), alpha)
        log_after = torch.log1p(-alpha).cumsum(-1)
        before = torch.exp(torch.nn.functional.pad(log_after, (1, 0))[..., :-1])
        alpha = torch.where(before >= 1e-4, alpha, torch.zeros_like(alpha))
        left = torch.exp(torch.log1p(-alpha).sum(-1))
        return (alpha * before) @ colour.T + left[..., None] * back, left

    rgb = torch.empty(h, w, 3, dtype=torch.float64, device=params.device)
    left = torch.empty(h, w, dtype=torch.float64, device=params.device)
    lists = list(members())
    with torch.no_grad():
        for (tx, ty), ids in zip(tiles, lists):
            box = (slice(ty * 16, ty * 16 + 16), slice(tx * 16, tx * 16 + 16))
            rgb[box], left[box] = tile(tx, ty, ids, leaves)
    if target is None:
        return rgb, left
    rgb.requires_grad_()
    loss = _loss64(rgb, target, weight)
    loss.backward()
    for v in leaves:
        v.requires_grad_()
    for (tx, ty), ids in zip(tiles, lists):
        if len(ids):
            box = (slice(ty * 16, ty * 16 + 16), slice(tx * 16, tx * 16 + 16))
            (tile(tx, ty, ids, leaves)[0] * rgb.grad[box]).sum().backward()
    torch.autograd.backward(projected[:4], [v.grad for v in leaves])
    return loss.item()
