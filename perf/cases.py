"""The performance cases of the framework: what its users have it render,
denoise and train, each through the public entry points, from the smallest
interactive frame to the precision workload's batched passes.

Scenes are the seeded phantoms of volview_gb300.scene (the head/neck phantom
with 120 labels and the small/torso body), built here on the GPU so that a
case's inputs are ready in a fraction of a second; the renderer takes them
from host memory, as a viewer hands over a CT. Every pass starts a new view
(`reset_view`), so that a pass does not depend on the ones before it.
"""
import ctypes as C
import math

import numpy as np
import torch

from volview_gb300 import abi, learned_denoiser, scene
from volview_gb300 import renderer as R

# Bytes a path must read and write (events of the head/neck default view times
# the element bytes of each: 698 MB per 1024 x 1024 paths), and its operations
# (26 flight iterations, 1.2 vertices).
PATH_BYTES, PATH_FLOPS = 666, 4000


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # The smallest call: one interactive frame of the small phantom at
        # 256 x 256 after a camera move, shown (latency and launches).
        dict(name="frame_small", kind="frame", body="torso", nx=128, ny=128, nz=128, w=256, h=256),
        # The ordinary viewer frame: a head/neck CT at 1024 x 1024.
        dict(name="frame_head", kind="frame", body="head", nx=512, ny=512, nz=400, w=1024, h=1024),
        # Offscreen rendering as the reference does it: `frames` records and a
        # tone-mapped image, a ragged CT and image.
        dict(name="offscreen_ragged", kind="offscreen", body="head", nx=251, ny=243, nz=187, w=643, h=479, frames=8),
        # Batched accumulation of a head/neck view: 16 frames in one call.
        dict(name="batch_head", kind="batch", body="head", nx=512, ny=512, nz=400, w=1024, h=1024, frames=16,
             light_map=0, density=0, kahan=0),
        # The same under an HDR light map (importance sampling, a second shadow ray).
        dict(name="batch_light_map", kind="batch", body="head", nx=256, ny=256, nz=200, w=601, h=433, frames=16,
             light_map=1024, density=0, kahan=0),
        # The largest: the precision workload, a 512 x 512 x 800 torso at
        # 1920 x 1080, FP16 density and compensated sums, 64 frames.
        dict(name="batch_torso_fp16", kind="batch", body="torso", nx=512, ny=512, nz=800, w=1920, h=1080, frames=64,
             light_map=0, density=1, kahan=1),
        # Serving: one batched pass over four requests (views) of two resident volumes.
        dict(name="serve_mix", kind="serve", body="head", nx=256, ny=256, nz=256, w=512, h=512, frames=8, requests=4),
        # Labels switched off and on again in the viewer: masks and majorants
        # of the whole volume are rebuilt, then a frame is shown.
        dict(name="relabel_head", kind="relabel", body="head", nx=512, ny=512, nz=400, w=768, h=768),
        # The real-time ray marcher while the camera orbits.
        dict(name="march_head", kind="march", body="head", nx=512, ny=512, nz=400, w=1024, h=1024),
        # The ray marcher while a clip plane is dragged: the occlusion and
        # shadow volumes follow every position.
        dict(name="cut_ragged", kind="cut", body="head", nx=301, ny=255, nz=203, w=511, h=387),
        # The learned denoiser on a 1024 x 1024 image.
        dict(name="unet_1024", kind="unet", n=1, w=1024, h=1024),
        # One training step's loss and gradients on a batch of four 256 x 256 crops.
        dict(name="train_256", kind="train", n=4, w=256, h=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "offscreen", "batch", "batch", "batch", "serve", "relabel", "march", "cut",
                       "unet", "train"])
    if kind == "unet":
        return dict(kind=kind, n=rng.randint(1, 2), w=256 * rng.randint(1, 4), h=16 * rng.randint(4, 64))
    if kind == "train":
        return dict(kind=kind, n=rng.randint(1, 6), w=256, h=16 * rng.randint(8, 16))
    body = rng.choice(["head", "head", "torso"])
    c = dict(kind=kind, body=body, nx=_log_int(rng, 100, 512), ny=_log_int(rng, 100, 512), nz=_log_int(rng, 100, 400),
             w=_log_int(rng, 200, 1280), h=_log_int(rng, 200, 1080))
    if kind == "offscreen":
        c["frames"] = rng.randint(2, 12)
    if kind == "batch":
        c.update(frames=_log_int(rng, 2, 32), light_map=rng.choice([0, 0, 512]), density=rng.randint(0, 3),
                 kahan=rng.randint(0, 1))
    if kind == "serve":
        c.update(frames=rng.randint(1, 12), requests=rng.randint(2, 6), w=_log_int(rng, 200, 640),
                 h=_log_int(rng, 200, 640))
    if kind == "cut":
        c.update(w=_log_int(rng, 200, 640), h=_log_int(rng, 200, 640))
    return c


# -------------------------------------------------------------------- phantoms
def _slabs(nz, step=48):
    return [(z, min(z + step, nz)) for z in range(0, nz, step)]


def _head(dims, spacing, seed):
    """scene.head_neck_phantom's recipe on the GPU: HU and labels (z, y, x)."""
    X, Y, Z = dims
    sx, sy, sz = spacing
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    hu = torch.empty((Z, Y, X), dtype=torch.int16, device="cuda")
    lab = torch.zeros((Z, Y, X), dtype=torch.uint8, device="cuda")
    ext = Z * sz
    cz, rz = 0.72 * ext, 0.27 * ext
    ys = ((torch.arange(Y, device="cuda") - (Y - 1) / 2) * sy)[None, :, None]
    xs = ((torch.arange(X, device="cuda") - (X - 1) / 2) * sx)[None, None, :]
    tubes = [(rng.uniform(0, 2 * math.pi), rng.uniform(15, 45), rng.uniform(3, 12), rng.uniform(1, 3),
              rng.uniform(1.5, 4), rng.uniform(0.55, 0.95)) for _ in range(30)]
    organs = [(58, 0, -25, 0.35, 18, 8, 14, 60), (59, 0, -40, 0.55, 22, 20, 16, 70), (60, -40, 5, 0.58, 12, 18, 20, 35),
              (61, 40, 5, 0.58, 12, 18, 20, 35), (119, -30, -70, 0.74, 11, 11, 11, 15),
              (120, 30, -70, 0.74, 11, 11, 11, 15)]
    sector = ((torch.atan2(ys, xs) + math.pi) / (2 * math.pi) * 8).int() % 8
    for z0, z1 in _slabs(Z):
        zs = ((torch.arange(z0, z1, device="cuda") + 0.5) * sz)[:, None, None]
        noise = torch.randn((z1 - z0, Y, X), generator=gen, device="cuda")
        h = torch.full((z1 - z0, Y, X), -1000.0, device="cuda")
        lb = lab[z0:z1]

        def put(mask, label, mean, sd):
            torch.where(mask, mean + sd * noise, h, out=h)
            if torch.is_tensor(label):
                torch.where(mask, label, lb, out=lb)
            else:
                lb.masked_fill_(mask, label)

        head = (xs / 74) ** 2 + (ys / 92) ** 2 + ((zs - cz) / rz) ** 2
        inner = (xs / 68) ** 2 + (ys / 86) ** 2 + ((zs - cz) / (rz - 6)) ** 2
        neck = ((xs / 55) ** 2 + ((ys - 8) / 50) ** 2 <= 1) & (zs < cz)
        band = (zs / (cz - 0.6 * rz) * 8).int().clamp(max=7)
        put((head <= 1) | neck, (62 + (band * 8 + sector).clamp(max=56)).to(torch.uint8), 40, 40)
        put((head <= 1) & (inner > 1) & (zs > cz - 0.6 * rz), 1, 1000, 80)
        put(inner <= 1, 56, 30, 20)
        put(((xs / 9) ** 2 + ((ys + 12) / 8) ** 2 <= 1) & (zs < cz - 20), 57, -900, 30)
        vert = (zs / 10).int().clamp(max=23)
        spine = ((xs / 13) ** 2 + ((ys - 22) / 11) ** 2 <= 1) | ((xs / 4) ** 2 + ((ys - 40) / 9) ** 2 <= 1)
        put(spine & (zs < cz - 0.4 * rz) & (zs % 10 < 7.5) & (zs < 240), (2 + vert).to(torch.uint8).expand_as(lb), 700, 80)
        t = zs / ext
        for v, (a, r0, amp, f, r, top) in enumerate(tubes):
            px = r0 * math.cos(a) + amp * torch.sin(2 * math.pi * f * t + v)
            py = r0 * math.sin(a) * 0.8 + amp * torch.cos(2 * math.pi * f * t * 0.7 + 2 * v)
            put(((xs - px) ** 2 + (ys - py) ** 2 <= r * r) & (t <= top), 26 + v, 400, 50)
        for label, ox, oy, oz, rx, ry, rzz, mean in organs:
            put(((xs - ox) / rx) ** 2 + ((ys - oy) / ry) ** 2 + ((zs - oz * ext) / rzz) ** 2 <= 1, label, mean, 20)
        hu[z0:z1] = h.round().clamp(-32768, 32767).to(torch.int16)
    return hu, lab


def _torso(dims, seed):
    """scene.torso_phantom's recipe on the GPU."""
    X, Y, Z = dims
    sx, sy, sz = X / 128, Y / 128, Z / 128
    gen = torch.Generator(device="cuda").manual_seed(seed)
    hu = torch.empty((Z, Y, X), dtype=torch.int16, device="cuda")
    lab = torch.zeros((Z, Y, X), dtype=torch.uint8, device="cuda")
    c = (X / 2 - 0.5, Y / 2 - 0.5, Z / 2 - 0.5)
    hc = c[2] + 31 * sz
    xs = torch.arange(X, device="cuda", dtype=torch.float32)[None, None, :] - c[0]
    ys = torch.arange(Y, device="cuda", dtype=torch.float32)[None, :, None] - c[1]
    for z0, z1 in _slabs(Z):
        zs = torch.arange(z0, z1, device="cuda", dtype=torch.float32)[:, None, None]
        noise = torch.randn((z1 - z0, Y, X), generator=gen, device="cuda")
        h = torch.full((z1 - z0, Y, X), -1000.0, device="cuda")
        lb = lab[z0:z1]

        def ell(dx, zc, rx, ry, rz):
            return ((xs - dx) / rx) ** 2 + (ys / ry) ** 2 + ((zs - zc) / rz) ** 2

        def put(mask, label, mean, sd):
            torch.where(mask, mean + sd * noise, h, out=h)
            if torch.is_tensor(label):
                torch.where(mask, label, lb, out=lb)
            else:
                lb.masked_fill_(mask, label)

        slab = ((zs - (c[2] - 58 * sz)) / (116 * sz) * 3).int().clamp(0, 2)
        region = (5 + slab * 2 + (xs >= 0).int()).to(torch.uint8).expand_as(lb)
        put(ell(0, c[2], 50 * sx, 40 * sy, 58 * sz) <= 1, region, 0, 40)
        out, inn = ell(0, hc, 34 * sx, 38 * sy, 26 * sz), ell(0, hc, 30 * sx, 34 * sy, 22 * sz)
        put(inn <= 1, 4, 20, 20)
        put((out <= 1) & (inn > 1), 1, 1000, 80)
        for k, dx in enumerate((-20 * sx, 20 * sx)):
            put(ell(dx, c[2] - 14 * sz, 14 * sx, 18 * sy, 24 * sz) <= 1, 2 + k, -800, 50)
        hu[z0:z1] = h.round().clamp(-32768, 32767).to(torch.int16)
    return hu, lab


def _soft(lab, spacing, factor):
    """scene.soft_grid's nodes on the GPU: own label, the nearest other label
    within 3 mm and the distance to it (x 16 x 4 / 3), not overridden."""
    g = lab[::factor, ::factor, ::factor].contiguous()
    s = [spacing[2] * factor, spacing[1] * factor, spacing[0] * factor]
    reach = [min(2, int(3.0 / q)) for q in s]
    best = torch.full(g.shape, 3.0, device="cuda")
    second = torch.zeros_like(g)
    pad = torch.nn.functional.pad(g[None, None].float(), [reach[2]] * 2 + [reach[1]] * 2 + [reach[0]] * 2,
                                  mode="replicate")[0, 0].to(torch.uint8)
    for dz in range(-reach[0], reach[0] + 1):
        for dy in range(-reach[1], reach[1] + 1):
            for dx in range(-reach[2], reach[2] + 1):
                d = math.sqrt((dz * s[0]) ** 2 + (dy * s[1]) ** 2 + (dx * s[2]) ** 2)
                if d == 0.0 or d > 3.0:
                    continue
                o = pad[reach[0] + dz:reach[0] + dz + g.shape[0], reach[1] + dy:reach[1] + dy + g.shape[1],
                        reach[2] + dx:reach[2] + dx + g.shape[2]]
                nearer = (o != g) & (best > d - 0.5 * min(s))
                best.masked_fill_(nearer, max(d - 0.5 * min(s), 0.0))
                torch.where(nearer, o, second, out=second)
    out = torch.zeros(g.shape + (4,), dtype=torch.uint8, device="cuda")
    out[..., 0] = g
    out[..., 1] = second
    out[..., 2] = (best * (64.0 / 3.0)).clamp(max=254).to(torch.uint8)
    return out.cpu().numpy()


# ------------------------------------------------------------------- renderers
class Scene:
    """A volume on a renderer, as a viewer keeps it, destroyed with the state."""

    def __init__(self, case, seed, precision=None):
        dims = (case["nx"], case["ny"], case["nz"])
        if case["body"] == "head":
            spacing = (256.0 / dims[0], 256.0 / dims[1], 400.0 / dims[2])
            hu, lab = _head(dims, spacing, seed)
            entries, ghosts = scene.head_neck_entries(seed), (scene.SKELETON,)
        else:
            spacing = (1.0, 1.0, 1.0)
            hu, lab = _torso(dims, seed)
            entries, ghosts = scene.SMALL_ENTRIES, ()
        soft = _soft(lab, spacing, 3 if max(dims) > 300 else 2)
        few = (slice(None, None, 3),) * 3  # label statistics from every third voxel
        labels = scene.label_params(lab[few].cpu().numpy(), hu[few].cpu().numpy(), entries, mode=abi.LABEL_HYBRID,
                                    ghost_groups=ghosts)
        self.hu, self.lab, self.soft = hu.cpu().numpy(), lab.cpu().numpy(), soft
        del hu, lab
        self.cfg = dict(min_spacing=min(spacing), label_params=labels)
        self.contexts, self.renderers, self.engine = [R.Context(0)], [], None
        self.r = R.Renderer(self.contexts[0], abi.volume_struct(self.hu, spacing), abi.tf_struct(abi.PRESETS["bone"]),
                            precision)
        self.renderers.append(self.r)
        self.r.set_labels(self.lab, abi.soft_struct(self.soft))

    def params(self, seed, denoiser=abi.DENOISE_ATROUS):
        """A camera near the default view, a sagittal cut near the middle."""
        rng = np.random.default_rng(seed)
        p = scene.frame_params_for(self.cfg, self.r.center, self.r.diagonal, clip_sagittal=True, denoiser=denoiser)
        p.camera.yaw = abi.f32(p.camera.yaw + rng.uniform(-0.3, 0.3))
        p.camera.pitch = abi.f32(p.camera.pitch + rng.uniform(-0.15, 0.15))
        p.clipping.planes[0].position = abi.f32(self.r.center[0] + self.r.diagonal * rng.uniform(-0.03, 0.03))
        return p

    def __del__(self):
        if getattr(self, "engine", None) is not None:
            self.engine.synchronize()
            self.engine.destroy()
        for r in reversed(getattr(self, "renderers", [])):
            r.destroy()
        for c in getattr(self, "contexts", []):
            c.destroy()


def _pinned(h, w, dtype):
    return torch.empty((h, w, 4), dtype=dtype, pin_memory=True)


def _show(r, out):
    """The tone-mapped image into a pinned buffer of the viewer's."""
    R.check(R.load().vv_read_output(r.handle, C.c_void_p(out.data_ptr()), out.numel()))
    return out


def _hdr(r, out):
    """The RGBA16F image into a pinned buffer."""
    R.check(R.load().vv_read_hdr(r.handle, C.c_void_p(out.data_ptr()), out.numel()))
    return out


def _smooth(gen, n, h, w, c, cell):
    low = torch.randn((n, c, -(-h // cell) + 1, -(-w // cell) + 1), generator=gen, device="cuda")
    return torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear").permute(0, 2, 3, 1)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("unet", "train"):
        n, h, w = case["n"], case["h"], case["w"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        net = learned_denoiser.UNet(seed=seed)
        # Log radiance (noisy, as from 4 paths), albedo and normals of shaded surfaces.
        clean = _smooth(gen, n, h, w, 3, 24).abs() * 0.3
        noisy = clean * (0.5 + torch.rand((n, h, w, 3), generator=gen, device="cuda"))
        albedo = (0.5 + 0.2 * _smooth(gen, n, h, w, 3, 48)).clamp(0, 1)
        normal = torch.nn.functional.normalize(_smooth(gen, n, h, w, 3, 32), dim=-1)
        x = torch.cat([noisy, albedo, normal, torch.zeros((n, h, w, 7), device="cuda")], -1).half().contiguous()
        return dict(kind=kind, net=net, x=x, target=clean.contiguous())
    w, h = case["w"], case["h"]
    precision = abi.precision(density_format=case.get("density", 0), sums=case.get("kahan", 0))
    s = Scene(case, seed, precision)
    st = dict(kind=kind, scene=s, w=w, h=h)
    if kind == "serve":
        rng = np.random.default_rng(seed)
        other = Scene(dict(case, nx=(case["nx"] * 3) // 4, body="torso"), seed + 1)
        st.update(other=other, items=[], outs=[])
        s.contexts.append(R.Context(0))
        s.engine = R.BatchEngine(s.contexts[-1], 2, 16)
        for k in range(case["requests"]):
            base = (s, other)[k % 2]
            base.contexts.append(R.Context(0))
            view = R.Renderer.view(base.contexts[-1], base.r)
            base.renderers.append(view)
            scale = 1 + 0.5 * (k % 3)
            vw, vh = int(w * scale) - k, int(h * scale)
            view.resize(vw, vh)
            p = base.params(seed + 10 + k)
            for v in rng.choice(np.arange(2, 10), 2, replace=False):  # the request's label visibility
                p.labels.colors[int(v)][3] = 0.0
            st["items"].append((view, p, 1, case["frames"], True))
            st["outs"].append(_pinned(vh, vw, torch.float16))
        return st
    s.r.resize(w, h)
    st["params"] = s.params(seed)
    st["out"] = _pinned(h, w, torch.uint8)
    if kind == "batch":
        st.update(out=_pinned(h, w, torch.float16), frames=case["frames"])
        if case["light_map"]:
            st["map"] = scene.synthetic_light_map(case["light_map"], case["light_map"] // 2, seed)
            s.r.set_environment_map(abi.env_struct(st["map"]))
            st["params"].lighting.environment = abi.ENV_MAP
    elif kind == "offscreen":
        st["frames"] = case["frames"]
    elif kind == "relabel":
        st["hidden"], st["out2"] = s.params(seed), _pinned(h, w, torch.uint8)
        hide = range(62, 119) if case["body"] == "head" else range(5, 11)
        for v in hide:  # the muscles switched off
            st["hidden"].labels.colors[v][3] = 0.0
    elif kind in ("march", "cut"):
        st["params"].path_tracing.enabled = 0
        if kind == "cut":
            st["moved"], st["out2"] = s.params(seed), _pinned(h, w, torch.uint8)
            st["moved"].path_tracing.enabled = 0
            st["moved"].clipping.planes[0].position += abi.f32(0.02 * s.r.diagonal)
        else:
            s.r.record(0, st["params"])  # the lighting volumes of the view that is orbited
    return st


def run(st):
    kind = st["kind"]
    if kind == "unet":
        return st["net"].forward(st["x"])
    if kind == "train":
        net = st["net"]
        pred = net.forward(st["x"])
        loss, dpred = net.loss(pred, st["target"])
        net.backward(dpred)
        return {"pred": pred, "loss": loss, "gw": [p["gw"] for p in net.params.values()],
                "gb": [p["gb"] for p in net.params.values()]}
    s = st["scene"]
    if kind == "serve":
        for view, *_ in st["items"]:
            view.reset_view()
        s.engine.record(st["items"])
        return [_hdr(item[0], out) for item, out in zip(st["items"], st["outs"])]
    r = s.r
    r.reset_view()
    if kind == "frame":
        r.record(1, st["params"])
        return _show(r, st["out"])
    if kind == "offscreen":
        out = st["out"]
        R.check(R.load().vv_render_to_rgba(r.handle, C.byref(st["params"]), st["w"], st["h"], st["frames"],
                                           C.c_void_p(out.data_ptr()), out.numel()))
        return out
    if kind == "batch":
        r.record_frames(1, st["frames"], st["params"])
        return _hdr(r, st["out"])
    if kind == "march":
        r.record(1, st["params"])
        return _show(r, st["out"])
    first = st["hidden"] if kind == "relabel" else st["moved"]  # relabel, cut
    r.record(1, first)
    a = _show(r, st["out2"])
    r.record(2, st["params"])
    return [a, _show(r, st["out"])]


# ------------------------------------------------------------------------ work
def work(case):
    kind = case["kind"]
    if kind in ("unet", "train"):
        px = case["n"] * case["w"] * case["h"]
        ch, shapes = learned_denoiser.channels()
        flops = sum(18 * ci * co * px / 4 ** _level(n) for n, (ci, co) in shapes.items())
        weights = sum(9 * ci * co for ci, co in shapes.values())
        if kind == "unet":
            return {"bytes": px * 64 + weights * 2, "flops": flops}
        # Weight and input gradients; the activations are written once and read again.
        acts = sum(ch[n] * px / 4 ** _level(n) for n in shapes)
        return {"bytes": px * 76 + 4 * acts + weights * 6, "flops": 3 * flops}
    px, vox = case["w"] * case["h"], case["nx"] * case["ny"] * case["nz"]
    shown = px * 60  # sums in, HDR and RGBA8 out
    if kind in ("frame", "offscreen", "batch"):
        paths = px * case.get("frames", 1)
        return {"bytes": paths * PATH_BYTES + shown, "flops": paths * PATH_FLOPS}
    if kind == "serve":
        paths = sum((1 + 0.5 * (k % 3)) ** 2 for k in range(case["requests"])) * px * case["frames"]
        return {"bytes": paths * PATH_BYTES + vox * 7 * case["requests"], "flops": paths * PATH_FLOPS}
    if kind == "relabel":
        return {"bytes": 2 * (vox * 7 + px * PATH_BYTES + shown), "flops": 2 * (vox * 50 + px * PATH_FLOPS)}
    march = px * 1500  # about 60 lit samples of a ray, or the skipped bricks before them
    if kind == "march":
        return {"bytes": march + shown, "flops": px * 30000}
    # cut: occlusion (128 samples per 4^3 voxels) and shadow volume (one per 2^3), twice
    return {"bytes": 2 * (march + shown + vox * 8), "flops": 2 * (px * 30000 + vox * 200)}


def _level(name):
    return 0 if name == "head" else int(name[1])


# ----------------------------------------------------------------------- exact
def _forward64(params, x):
    """The U-Net in 64 bits (torch), weights as the kernels read them."""
    F = torch.nn.functional

    def conv(name, v, relu=True):
        w, b = params[name]
        y = F.conv2d(v, w.permute(0, 3, 1, 2), b, padding=1)
        return F.relu(y) if relu else y

    v, skips, levels = x, [], len(learned_denoiser.LEVELS)
    for lv in range(levels):
        if lv:
            v = F.avg_pool2d(v, 2)
        v = conv(f"e{lv}b", conv(f"e{lv}a", v))
        skips.append(v)
    for lv in range(levels - 2, -1, -1):
        v = torch.cat([F.interpolate(v, scale_factor=2, mode="nearest"), skips[lv]], 1)
        v = conv(f"d{lv}b", conv(f"d{lv}a", v))
    return conv("head", v, False)


def exact(case, seed):
    if case["kind"] not in ("unet", "train"):
        return None  # random walks: no 64-bit value that a rounding would not divert
    st = prepare(case, seed)
    train = case["kind"] == "train"
    params = {n: tuple(t.double().clone().requires_grad_(train) for t in (p["w16"], p["b"]))
              for n, p in st["net"].params.items()}
    pred = _forward64(params, st["x"].double().permute(0, 3, 1, 2)).permute(0, 2, 3, 1)
    if not train:
        return pred
    loss = (pred[..., :3] - st["target"].double()).abs().mean()
    loss.backward()
    scale = learned_denoiser.GRAD_SCALE
    return {"pred": pred.detach(), "loss": loss.detach().reshape(1), "gw": [w.grad * scale for w, _ in params.values()],
            "gb": [b.grad * scale for _, b in params.values()]}
