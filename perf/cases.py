"""What a user of this framework has it do, as cases that can be timed and compared.

Each case is a dict of plain values; ``prepare`` makes what a user's program
holds before the call (scene, cameras, photos, a ``Trainer``), ``run`` is one
pass through the public entry points, ``work`` the bytes and operations the
pass cannot do without and ``exact`` its outputs in 64 bits, evaluated with
plain torch from the definitions alone.

Kinds of pass:
  render     one view of a trainer's Gaussians as RGB floats (evaluation)
  preview    ``cpu::rasterize``'s framebuffer of a trainer's Gaussians
  drop_in    the stateless ``render_and_backward`` on host arrays
  gradients  one render + loss + backward over the step's views, gradients left
             on the device (what a rank does before the all-reduce), then, with
             ``adam``, the optimiser step on them
  training   several ``Trainer.step`` calls and the Gaussians read back (the
             work between two checkpoints); ``host_targets`` takes each step's
             photos from page-locked host memory
  loss       the photometric loss and its gradient on caller-owned device images

The learning rates are those of late training (a hundredth of the defaults),
so the scene, and with it the work, stays the same over many passes. Scenes
follow the repository's benchmark configurations: means uniform in a cube,
quaternions normalised, SH degree 3. The photos are smooth random images with
sensor noise, so the first gradients are those of a scene that has yet to fit.
"""
import ctypes
import math

import numpy as np
import torch

from rgsplat_b200 import Camera, Context, LossConfig, TrainConfig, Trainer, render_and_backward
from rgsplat_b200 import _lib
from rgsplat_b200.dp import CudaArray

LATE = dict(lr_position=1.6e-6, lr_rotation=1e-5, lr_scale=5e-5, lr_opacity=5e-4, lr_sh_dc=2.5e-5, lr_sh_rest=1.25e-6)
LAMBDA = 0.2
DEFAULTS = dict(kind="", n=0, extent=1.0, distance=4.0, focal=1.171875, log_scale=-4.0, log_scale_sigma=0.5, opacity=0.0,
                sizes="256x256", cams=1, views=1, steps=1, batched=False, host_targets=False, adam=False, exact_loss=False,
                batch=256, bg=0.0, srgb8=False)


def _case(name, **kw):
    c = dict(DEFAULTS)
    c.update(kw)
    if name:
        c["name"] = name
    return c


HEADLINE = dict(extent=2.0, distance=5.0, focal=1.25, sizes="1600x1064,1280x720,960x540", batch=128)


def listed():
    return [
        # the smallest call: one small view of a small scene, where latency and launches count
        _case("render_10k_256", kind="render", n=10_000, sizes="256x256"),
        # one iteration's gradients of the smallest benchmark scene, per-view launches
        _case("gradients_10k_256", kind="gradients", n=10_000, sizes="256x256"),
        # a program that calls the reference's free function with its own arrays
        _case("drop_in_50k_512", kind="drop_in", n=50_000, sizes="512x512"),
        # the reference's training loop: one view an iteration, on a NeRF-synthetic-sized scene
        _case("training_200k_800", kind="training", n=200_000, extent=2.0, distance=5.0, focal=1.25, sizes="800x800", cams=8,
              steps=20),
        # photos streamed from host memory, four views a step
        _case("training_200k_host_targets", kind="training", n=200_000, extent=2.0, distance=5.0, focal=1.25, sizes="800x800",
              cams=8, views=4, steps=10, batched=True, host_targets=True),
        # odd sizes, a white background (full tile lists) and the reference's exact loss arithmetic
        _case("gradients_97k_odd_white", kind="gradients", n=97_003, extent=2.0, distance=5.0, focal=1.25, sizes="1277x719",
              cams=3, views=3, batched=True, bg=1.0, exact_loss=True),
        # the benchmark's step as a data-parallel rank runs it: gradients, then Adam
        _case("gradients_1M_8views", kind="gradients", n=1_000_000, cams=8, views=8, batched=True, adam=True, **HEADLINE),
        # the benchmark's training step, Adam fused into the pass
        _case("training_1M_8views", kind="training", n=1_000_000, cams=16, views=8, steps=20, batched=True, **HEADLINE),
        # the largest benchmark scene (3M anisotropic Gaussians, full HD): one of two ranks' share of its
        # sixteen views, past one launch's pair budget
        _case("gradients_3M_8views_hd", kind="gradients", n=3_000_000, extent=2.0, distance=5.0, focal=1.0, log_scale=-3.5,
              log_scale_sigma=1.0, opacity=1.0, sizes="1920x1080", cams=8, views=8, batched=True, adam=True, batch=128),
        # a live preview of a scene in training, as display bytes
        _case("preview_1M_1600_bytes", kind="preview", n=1_000_000, extent=2.0, distance=5.0, focal=1.25, sizes="1600x1064",
              srgb8=True),
        # the loss alone, for a program with its own renderer
        _case("loss_1600x1064", kind="loss", sizes="1600x1064"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "preview", "drop_in", "gradients", "gradients", "training", "training", "loss"])
    w = _log_int(rng, 150, 1600)
    h = max(64, int(w * rng.uniform(0.5, 1.0)))
    if kind == "loss":
        return _case("", kind=kind, sizes="%dx%d" % (w, h))
    # the stateless call copies every array both ways: smaller scenes use it
    n = _log_int(rng, 5_000, 100_000 if kind == "drop_in" else 1_000_000)
    wide = dict(extent=2.0, distance=5.0, focal=rng.choice([1.0, 1.25]))
    c = _case("", kind=kind, n=n, sizes="%dx%d" % (w, h), **(wide if n > 60_000 or rng.random() < 0.5 else {}))
    c["batch"] = rng.choice([128, 256])
    c["bg"] = rng.choice([0.0, 0.0, 0.0, 1.0])
    if kind == "preview":
        c["srgb8"] = rng.random() < 0.5
    if kind in ("gradients", "training"):
        c["views"] = rng.choice([1, 1, 2, 3, 4, 6, 8])
        c["batched"] = c["views"] > 1 or rng.random() < 0.3
        c["cams"] = c["views"] + (4 if kind == "training" else 0)
        c["exact_loss"] = rng.random() < 0.2
        if c["views"] > 1 and rng.random() < 0.5:
            c["sizes"] += ",%dx%d" % (max(64, w * 3 // 4), max(64, h * 2 // 3))
        if kind == "training":
            # no more than the listed training of the benchmark scene
            most = min(60e6 / (c["views"] * w * h), 6e7 / (c["views"] * n))
            c["steps"] = max(1, min(rng.choice([5, 10, 20]), int(most)))
            c["host_targets"] = c["batched"] and rng.random() < 0.3
        else:
            c["adam"] = rng.random() < 0.5
    return c


# ---- inputs -----------------------------------------------------------------
def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]


def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed * 1_000_003 + 17)


def _scene(case, seed):
    """(N, 59) float32 records on the GPU."""
    g, n = _gen(seed), case["n"]
    out = torch.empty(n, 59, device="cuda")
    out[:, :3] = (torch.rand(n, 3, device="cuda", generator=g) * 2 - 1) * case["extent"]
    out[:, 3] = torch.randn(n, device="cuda", generator=g) + case["opacity"]
    q = torch.randn(n, 4, device="cuda", generator=g)
    out[:, 4:8] = q / q.norm(dim=1, keepdim=True).clamp_min(1e-12)
    out[:, 8:11] = torch.randn(n, 3, device="cuda", generator=g) * case["log_scale_sigma"] + case["log_scale"]
    sh = torch.randn(n, 48, device="cuda", generator=g) * 0.05
    sh[:, ::16] *= 6.0
    out[:, 11:] = sh
    return out


def _cameras(case, seed):
    """Cameras on a sphere around the origin (OpenCV axes), turned by the seed; sizes cycle."""
    cams, sizes = [], _sizes(case)
    turn = np.random.default_rng(seed).uniform(0.0, 2.0 * math.pi)
    for i in range(case["cams"]):
        y = 1.0 - 2.0 * (i + 0.5) / case["cams"]
        r, th = math.sqrt(max(0.0, 1.0 - y * y)), math.pi * (3.0 - math.sqrt(5.0)) * i + turn
        eye = case["distance"] * np.array([math.cos(th) * r, math.sin(th) * r, y])
        fwd = -eye / np.linalg.norm(eye)
        up = np.array([0.0, 0.0, 1.0]) if abs(fwd[2]) < 0.999 else np.array([0.0, 1.0, 0.0])
        right = np.cross(fwd, up)
        right /= np.linalg.norm(right)
        c2w = np.eye(4, dtype=np.float32)
        c2w[:3, 0], c2w[:3, 1], c2w[:3, 2], c2w[:3, 3] = right, np.cross(fwd, right), fwd, eye
        w, h = sizes[i % len(sizes)]
        cams.append((w, h, case["focal"] * w, c2w))
    return cams


def _photo(w, h, g):
    """(h, w, 4) float32 RGBA on the GPU: two octaves of smooth colour and sensor noise."""
    img = torch.full((1, 3, h, w), 0.45, device="cuda")
    for cells, amp in ((6, 0.25), (40, 0.1)):
        grid = torch.randn(1, 3, cells, cells, device="cuda", generator=g) * amp
        img += torch.nn.functional.interpolate(grid, size=(h, w), mode="bicubic", align_corners=False)
    img += torch.randn(1, 3, h, w, device="cuda", generator=g) * 0.01
    out = torch.ones(h, w, 4, device="cuda")
    out[..., :3] = img.clamp(0.02, 0.98)[0].permute(1, 2, 0)
    return out


def _photos(case, cams, seed):
    g = _gen(seed + 7919)
    return [_photo(w, h, g) for w, h, _, _ in cams]


def _loss_images(case, seed):
    w, h = _sizes(case)[0]
    g = _gen(seed)
    target = _photo(w, h, g)
    # a render that is close to the photo but not there yet
    rendered = (0.9 * target[..., :3] + 0.1 * _photo(w, h, g)[..., :3]).contiguous()
    return rendered, target


def prepare(case, seed):
    if case["kind"] == "loss":
        rendered, target = _loss_images(case, seed)
        lib = _lib.load()
        return {"case": case, "lib": lib, "rendered": rendered, "target": target, "loss": torch.zeros(1, device="cuda"),
                "dl": torch.zeros_like(rendered), "err": ctypes.create_string_buffer(256)}
    cams = _cameras(case, seed)
    cameras = [Camera(w, h, f, f, w / 2.0, h / 2.0, c2w) for w, h, f, c2w in cams]
    scene = _scene(case, seed).cpu().numpy()
    s = {"case": case, "bg": (case["bg"],) * 3, "loss_cfg": LossConfig(LAMBDA), "train_cfg": TrainConfig(**LATE), "at": 0}
    if case["kind"] == "drop_in":
        s.update(ctx=Context(batch=case["batch"]), scene=scene, camera=cameras[0], target=_photos(case, cams, seed)[0].cpu().numpy())
        return s
    trainer = Trainer(scene, cameras, batch=case["batch"], exact_loss=case["exact_loss"])
    s["trainer"] = trainer
    if case["kind"] in ("gradients", "training"):
        photos = _photos(case, cams, seed)
        if case["host_targets"]:
            s["photos"] = [torch.empty(p.shape, pin_memory=True).copy_(p) for p in photos]
        else:
            for i, p in enumerate(photos):
                trainer.set_target(i, p.cpu().numpy())
    return s


# ---- one pass ---------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "loss":
        w, h = _sizes(case)[0]
        rc = state["lib"].rgs_photometric_loss_grad_noalloc(
            0, state["rendered"].data_ptr(), state["target"].data_ptr(), w, h, LAMBDA, state["loss"].data_ptr(),
            state["dl"].data_ptr(), torch.cuda.current_stream().cuda_stream, state["err"], len(state["err"]))
        if rc:
            raise RuntimeError(state["err"].value.decode())
        return {"loss": state["loss"], "dl": state["dl"]}
    bg = state["bg"]
    if kind == "drop_in":
        loss, grads = render_and_backward(state["scene"], state["camera"], state["target"], bg=bg, cfg=state["loss_cfg"],
                                          ctx=state["ctx"])
        return {"loss": loss, "grads": grads}
    trainer = state["trainer"]
    if kind == "render":
        return {"image": trainer.render(0, bg=bg)}
    if kind == "preview":
        return {"image": trainer.rasterize(0, bg=bg, srgb8=case["srgb8"])}
    mode = Trainer.BATCHED if case["batched"] else Trainer.PLAIN
    if kind == "gradients":
        losses = trainer.backward(list(range(case["views"])), bg=bg, loss_cfg=state["loss_cfg"], mode=mode)
        ptr, nbytes, stride = trainer.grad_buffer()
        buffer = CudaArray(ptr, nbytes)
        buffer.owner = trainer  # the tensor holds its source, and with it the trainer whose memory it is
        planes = torch.as_tensor(buffer, device="cuda")[: 15 * stride * 4].view(15, stride, 4)[:, : case["n"]]
        if case["adam"]:
            trainer.apply_adam(state["train_cfg"], denom_increment=case["views"])
        return {"losses": losses, "grads": planes}
    losses = []
    for _ in range(case["steps"]):
        views = [(state["at"] + v) % case["cams"] for v in range(case["views"])]
        state["at"] = (state["at"] + case["views"]) % case["cams"]
        if case["host_targets"]:
            losses.append(trainer.step_host_targets(views, [state["photos"][v].data_ptr() for v in views], bg=bg,
                                                    loss_cfg=state["loss_cfg"], train_cfg=state["train_cfg"]))
        else:
            losses.append(trainer.step(views, bg=bg, loss_cfg=state["loss_cfg"], train_cfg=state["train_cfg"], mode=mode))
    return {"losses": np.stack(losses), "gaussians": trainer.gaussians()}


# ---- the work a pass cannot do without --------------------------------------
def work(case):
    sizes = _sizes(case)
    if case["kind"] == "loss":
        px = sizes[0][0] * sizes[0][1]
        # ten separable 11-tap blurs of three channels
        return {"bytes": px * (12.0 + 16.0 + 12.0), "flops": px * 3 * 10 * 2 * 21.0}
    views = [sizes[v % len(sizes)] for v in range(case["views"])]
    if case["kind"] == "training":
        views = [sizes[v % case["cams"] % len(sizes)] for v in range(case["views"] * case["steps"])]
    n, steps = case["n"], case["steps"]
    px = float(sum(w * h for w, h in views))
    # pixels a splat reaches (alpha >= 1/255) on the average and from the middle of the scene, and the
    # splats a pixel can take before its transmittance is spent (about forty at these opacities)
    pairs = 0.0
    for w, h in views:
        sigma = max(0.6, math.exp(case["log_scale"] + case["log_scale_sigma"] ** 2 / 2) * case["focal"] * w / case["distance"])
        pairs += min(n * 2 * math.pi * math.log(255 * 0.5) * sigma * sigma, w * h * 40.0)
    backward = case["kind"] in ("drop_in", "gradients", "training")
    flops = pairs * (21.0 + (47.0 if backward else 0.0)) + (px * 3 * 10 * 2 * 21.0 if backward else 0.0)
    if case["kind"] == "render":
        return {"bytes": n * 236.0 + px * 12, "flops": flops}
    if case["kind"] == "preview":
        return {"bytes": n * 236.0 + px * (4 if case["srgb8"] else 16), "flops": flops}
    if case["kind"] == "drop_in":
        return {"bytes": n * (236.0 + 240.0) + px * 16, "flops": flops}
    if case["kind"] == "gradients":
        # parameters in, gradients out; with Adam both moments in and out, parameters out
        return {"bytes": n * (236.0 + 240.0 + (5 * 236.0 + 16 if case["adam"] else 0.0)) + px * 16, "flops": flops}
    return {"bytes": steps * n * (6 * 236.0 + 16) + n * 236.0 + px * 16, "flops": flops}


# ---- 64-bit values ----------------------------------------------------------
def _loss64(x, y, lam):
    """(1 - lam) L1 + lam (1 - SSIM) of (h, w, 3) images: 11 taps, sigma 1.5, zero padding."""
    k = torch.exp(-0.5 * (torch.arange(11, device=x.device, dtype=torch.float64) - 5) ** 2 / 2.25)
    k = (k / k.sum()).view(1, 1, 1, 11)

    def blur(a):
        a = torch.nn.functional.conv2d(a, k, padding=(0, 5))
        return torch.nn.functional.conv2d(a, k.transpose(2, 3), padding=(5, 0))

    a, b = x.permute(2, 0, 1)[:, None], y.permute(2, 0, 1)[:, None]
    ma, mb = blur(a), blur(b)
    va, vb, vab = blur(a * a) - ma * ma, blur(b * b) - mb * mb, blur(a * b) - ma * mb
    ssim = ((2 * ma * mb + 1e-4) * (2 * vab + 9e-4)) / ((ma * ma + mb * mb + 1e-4) * (va + vb + 9e-4))
    d = x - y
    return (1 - lam) * torch.where(d >= 0, d, -d).mean() + lam * (1 - ssim.mean())  # derivative +1 at 0


def _sh_basis(d):
    x, y, z = d.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    return torch.stack([
        torch.full_like(x, 0.28209479177387814), -0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x,
        1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * zz - xx - yy),
        -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy), -0.5900435899266435 * y * (3 * xx - yy),
        2.890611442640554 * x * y * z, -0.4570457994644658 * y * (4 * zz - xx - yy),
        0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy), -0.4570457994644658 * x * (4 * zz - xx - yy),
        1.445305721320277 * z * (xx - yy), -0.5900435899266435 * x * (xx - 3 * yy)], dim=1)


def _project64(p, cam):
    """Splats of one view from the parameters: (attributes (V, 9), depth, tile rectangles, kept indices)."""
    w, h, f, c2w = cam
    f = float(np.float32(f))
    m = torch.from_numpy(np.linalg.inv(c2w.astype(np.float64)).astype(np.float32).astype(np.float64)).cuda()
    eye = torch.from_numpy(c2w[:3, 3].astype(np.float64)).cuda()
    pc = p["pos"] @ m[:3, :3].T + m[:3, 3]
    op = torch.sigmoid(p["logit"])
    tz = pc[:, 2]
    sx, sy = f * pc[:, 0] / tz + w / 2.0, f * pc[:, 1] / tz + h / 2.0
    ok = (op >= 1 / 255) & (tz > 0.001) & (sx >= -128) & (sx <= w + 128) & (sy >= -128) & (sy <= h + 128)
    keep = ok.nonzero()[:, 0]
    pc, op, sx, sy = pc[keep], op[keep], sx[keep], sy[keep]
    tx, ty, tz = pc.unbind(1)
    qw, qx, qy, qz = p["rot"][keep].unbind(1)
    rot = torch.stack([1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy - qw * qz), 2 * (qx * qz + qw * qy),
                       2 * (qx * qy + qw * qz), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz - qw * qx),
                       2 * (qx * qz - qw * qy), 2 * (qy * qz + qw * qx), 1 - 2 * (qx * qx + qy * qy)], dim=1).view(-1, 3, 3)
    rs = rot * p["log_scale"][keep].exp()[:, None, :]
    z = torch.zeros_like(tz)
    jac = torch.stack([f / tz, z, -f * tx / (tz * tz), z, f / tz, -f * ty / (tz * tz)], dim=1).view(-1, 2, 3)
    t = jac @ m[:3, :3] @ rs
    cov = t @ t.transpose(1, 2)
    a, b, c = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
    det = a * c - b * b
    d = eye - p["pos"][keep]
    d = d / d.norm(dim=1, keepdim=True)
    col = (0.5 + torch.einsum("nk,nck->nc", _sh_basis(d), p["sh"][keep].view(-1, 3, 16))).clamp(0, 1)
    attr = torch.cat([torch.stack([sx, sy, c / det, -b / det, a / det], dim=1), col, op[:, None]], dim=1)
    with torch.no_grad():
        disc = torch.sqrt((a - c) ** 2 * 0.25 + b * b)
        r = 3 * torch.sqrt(torch.clamp((a + c) * 0.5 + disc, min=0))
        x0, y0 = (sx - r).trunc().clamp_min(0).long(), (sy - r).trunc().clamp_min(0).long()
        x1, y1 = ((sx + r).trunc().long() + 1).clamp_max(w), ((sy + r).trunc().long() + 1).clamp_max(h)
        good = (det.abs() >= 1e-8) & (x0 < x1) & (y0 < y1)
        rect = torch.stack([x0 // 16, y0 // 16, (x1 + 15) // 16, (y1 + 15) // 16], dim=1)
    return attr[good], tz[good], rect[good], keep[good]


def _tile_lists(depth, rect, tiles_x, tiles):
    """Per-tile splat indices in depth order: (entries, start of each tile, length of each tile)."""
    order = torch.argsort(depth, stable=True)
    r = rect[order]
    wide, cnt = r[:, 2] - r[:, 0], (r[:, 2] - r[:, 0]) * (r[:, 3] - r[:, 1])
    who = torch.repeat_interleave(torch.arange(len(order), device="cuda"), cnt)
    at = torch.arange(len(who), device="cuda") - (cnt.cumsum(0) - cnt)[who]
    tile = (r[who, 1] + at // wide[who]) * tiles_x + r[who, 0] + at % wide[who]
    by = torch.argsort(tile, stable=True)
    length = torch.bincount(tile, minlength=tiles)
    return order[who[by]], length.cumsum(0) - length, length


def _blend64(attr, lists, w, h, bg, start, dl=None):
    """Composites the tiles front to back. Without ``dl``: the (h, w, 3) image and
    the final transmittance; with it, the gradient of sum(image * dl) by attribute."""
    entries, first, length = lists
    tiles_x = (w + 15) // 16
    entries = torch.cat([entries, torch.tensor([len(attr)], device="cuda")])
    attr = torch.cat([attr, torch.zeros(1, 9, device="cuda", dtype=torch.float64)])
    image = torch.zeros(h, w, 3, device="cuda", dtype=torch.float64)
    left = torch.ones(h, w, device="cuda", dtype=torch.float64)
    grad = torch.zeros_like(attr)
    ids = torch.argsort(length)
    ids = ids[int((length == 0).sum()):]
    lens = length[ids].cpu().numpy()
    px = torch.arange(256, device="cuda")
    i = 0
    while i < len(ids):
        j = i + 1
        while j < len(ids) and (j + 1 - i) * int(lens[j]) * 256 <= 12_000_000:
            j += 1
        t, most = ids[i:j], int(lens[j - 1])
        k = torch.arange(most, device="cuda")
        idx = entries[torch.where(k < length[t][:, None], first[t][:, None] + k, len(entries) - 1)]
        x, y = (t % tiles_x)[:, None] * 16 + px % 16, (t // tiles_x)[:, None] * 16 + px // 16
        inside = (x < w) & (y < h)
        with torch.set_grad_enabled(dl is not None):
            a = attr[idx].detach().requires_grad_(dl is not None)
            dx = x[..., None] + 0.5 - a[:, None, :, 0]
            dy = y[..., None] + 0.5 - a[:, None, :, 1]
            power = -0.5 * (a[:, None, :, 2] * dx * dx + 2 * a[:, None, :, 3] * dx * dy + a[:, None, :, 4] * dy * dy)
            alpha = (a[:, None, :, 8] * power.clamp_max(0).exp()).clamp_max(0.99)
            alpha = torch.where((power > 0) | (alpha < 1 / 255), torch.zeros_like(alpha), alpha)
            log = torch.log1p(-alpha)
            before = (log.cumsum(2) - log).exp()
            live = before >= 1e-4
            weight = torch.where(live, alpha * before, torch.zeros_like(alpha))
            end = torch.where(live, log, torch.zeros_like(log)).sum(2).exp()
            rgb = weight @ a[:, :, 5:8] + (bg if start else end[..., None] * bg)
            if dl is not None:
                up = torch.zeros_like(rgb)
                up[inside] = dl[y[inside], x[inside]]
                g, = torch.autograd.grad(rgb, a, up)
                grad.index_add_(0, idx.reshape(-1), g.reshape(-1, 9))
        if dl is None:
            image[y[inside], x[inside]] = rgb[inside]
            left[y[inside], x[inside]] = end[inside]
        i = j
    return grad[:-1] if dl is not None else (image, left)


def exact(case, seed):
    if case["kind"] == "loss":
        rendered, target = _loss_images(case, seed)
        x = rendered.double().requires_grad_(True)
        loss = _loss64(x, target[..., :3].double(), LAMBDA)
        dl, = torch.autograd.grad(loss, x)
        return {"loss": loss.detach().view(1), "dl": dl}
    sizes = _sizes(case)
    px = sum(w * h for w, h in (sizes[v % len(sizes)] for v in range(case["views"])))
    # several steps, display bytes and the large scenes have no value here (too slow, or not numbers)
    if case["kind"] == "training" or case["srgb8"] or px > 3_000_000 or case["n"] * case["views"] > 400_000:
        return None
    cams, scene = _cameras(case, seed), _scene(case, seed).double()
    bg = torch.full((3,), case["bg"], device="cuda", dtype=torch.float64)
    # the rotation's gradient is by the normalised quaternion
    q = scene[:, 4:8] / scene[:, 4:8].norm(dim=1, keepdim=True)
    p = {"pos": scene[:, :3], "logit": scene[:, 3], "rot": q, "log_scale": scene[:, 8:11], "sh": scene[:, 11:]}
    p = {k: v.clone().requires_grad_(True) for k, v in p.items()}
    total = {k: torch.zeros_like(v) for k, v in p.items()}
    screen = torch.zeros(case["n"], device="cuda", dtype=torch.float64)
    photos = _photos(case, cams, seed) if case["kind"] in ("gradients", "drop_in") else None
    losses = []
    for v in range(case["views"]):
        w, h = cams[v][:2]
        attr, depth, rect, keep = _project64(p, cams[v])
        tiles_x = (w + 15) // 16
        lists = _tile_lists(depth.detach(), rect, tiles_x, tiles_x * ((h + 15) // 16))
        image, left = _blend64(attr.detach(), lists, w, h, bg, case["kind"] == "preview")
        if case["kind"] == "render":
            return {"image": image}
        if case["kind"] == "preview":
            return {"image": torch.cat([image, 1 - left[..., None]], dim=2)}
        x = image.requires_grad_(True)
        loss = _loss64(x, photos[v][..., :3].double(), LAMBDA)
        dl, = torch.autograd.grad(loss, x)
        losses.append(float(loss.detach()))
        g = _blend64(attr.detach(), lists, w, h, bg, False, dl)
        screen[keep] += g[:, :2].norm(dim=1)
        for k, d in zip(p, torch.autograd.grad(attr, list(p.values()), g)):
            total[k] += d
    if case["kind"] == "drop_in":
        grads = torch.cat([total["pos"], total["rot"], total["log_scale"], total["logit"][:, None], total["sh"], screen[:, None]], 1)
        return {"loss": losses[0], "grads": grads}
    flat = torch.cat([total["pos"], total["logit"][:, None], total["rot"], total["log_scale"], screen[:, None], total["sh"]], 1)
    return {"losses": np.array(losses), "grads": flat.view(-1, 15, 4).transpose(0, 1)}
