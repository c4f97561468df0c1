"""The work a user has the renderer do, as cases that can be timed and compared.

Each case is one call (or the few calls of one frame) through the public entry
points: `Renderer.draw_frame` in its four render modes, camera and gsanim state
batches, the display pass, a training step of the denoiser, and the device
sort.  The scenes are the seeded synthetic ones of `gamesplat_b200.scene`
(the uniform cube and the clustered room, same distributions), drawn on the
GPU: a scene is set-up, not the measured work.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) scene, camera, targets and handles a program keeps
    run(state)          one pass
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the pass in 64-bit arithmetic, where it has such a value
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gamesplat_b200 import _lib as L
from gamesplat_b200 import renderer as R
from gamesplat_b200 import scene
from gamesplat_b200.denoiser import LAYERS, Denoiser

ORBIT = 120          # cameras of the orbit
VISIBLE = 0.67       # share of the room's Gaussians an orbit camera sees
ENTRIES = 3.2        # (16x16 tile, splat) pairs per visible Gaussian at 1080p
SH_C1 = 0.4886025119029199
SH_C2 = (1.0925484305920792, -1.0925484305920792, 0.31539156525252005, -1.0925484305920792, 0.5462742152960396)
SH_C3 = (-0.5900435899266435, 2.890611442640554, -0.4570457994644658, 0.3731763325901154, -0.4570457994644658,
         1.445305721320277, -0.5900435899266435)


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def frame(n, w, h, world="room", half=False, degree=3, **more):
    return dict(kind="frame", n=n, w=w, h=h, world=world, half=half, degree=degree, **more)


def listed():
    return [
        # a small captured object in a viewer window: launches and latency count
        dict(frame(100_000, 1280, 720, world="cube"), name="frame_100k_720p"),
        # the ordinary frame: a captured room at full HD, a free-flying camera
        dict(frame(3_000_000, 1920, 1080), name="frame_3m_1080p"),
        # a large capture on a 4K display, rows with half-precision SH to halve the upload
        dict(frame(6_000_000, 3840, 2160, half=True), name="frame_6m_2160p_half"),
        # the order-independent mode with its temporal filter (4 jittered samples a frame), camera moving
        dict(kind="stochastic", n=3_000_000, w=1920, h=1080, samples=4, name="stochastic_3m_1080p"),
        # point splatting in a window, 2x2 supersampled, with a work budget that holds the frame
        dict(kind="gps", n=1_000_000, w=1280, h=720, ss=2, budget=32 << 20, name="gps_1m_720p"),
        # two stochastic samples, temporal history and the denoiser, over-budget tiles sorted
        dict(kind="denoised", n=3_000_000, w=1920, h=1080, name="denoised_3m_1080p"),
        # a server rendering many viewers of one scene, viewports of every size
        dict(kind="batch", n=3_000_000, cams=16, name="batch_3m_16cams"),
        # appearance playback rendered ahead: blended states of one camera
        dict(kind="states", n=1_000_000, w=1920, h=1080, states=4, frames=16, name="states_1m_16frames"),
        # a layered (gsanim 0.3) asset played back: new layer weights, then the frame
        dict(kind="layers", n=1_000_000, w=1920, h=1080, layers=4, name="layers_1m_1080p"),
        # that asset's display pass: exposure and its 33^3 table over a linear frame
        dict(kind="display", w=1920, h=1080, lut=33, name="display_1080p"),
        # a step of the denoiser's training, as train_denoiser.py makes them
        dict(kind="train", batch=8, crop=256, name="train_8x256"),
        # the sort of a host engine's own (key, index) pairs: float depth keys
        dict(kind="sort", n=2_000_003, bits=32, name="sort_2m"),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "stochastic", "gps", "denoised", "batch", "states", "layers",
                       "display", "train", "sort"])
    # any viewport from a thumbnail to 4K, odd sizes included; heavy scenes up to 1440p
    h = log_int(rng, 180, 1440)
    w = max(64, int(h * rng.uniform(0.8, 2.2)))
    if kind == "frame":
        world = rng.choice(["room", "room", "cube"])
        n = log_int(rng, 5_000, 4_000_000 if world == "room" else 200_000)
        return frame(n, w, h, world=world, half=rng.random() < 0.25, degree=rng.choice([3, 3, 3, 2, 1, 0]))
    if kind == "stochastic":
        return dict(kind=kind, n=log_int(rng, 20_000, 3_000_000), w=w, h=h, samples=rng.choice([1, 2, 4, 4]))
    if kind == "gps":
        h = min(h, 1080)
        w = min(w, 1920)
        n = log_int(rng, 20_000, 1_500_000)
        need = n * 16.0 * (h / 720.0) ** 2 * 1.8   # work items of a frame, with room to spare
        budget = 16 << 20
        while budget < need:
            budget *= 2
        return dict(kind=kind, n=n, w=w, h=h, ss=rng.choice([1, 2, 2, 3]), budget=budget)
    if kind == "denoised":
        return dict(kind=kind, n=log_int(rng, 50_000, 3_000_000), w=2 * (w // 2), h=2 * (h // 2))
    if kind == "batch":
        return dict(kind=kind, n=log_int(rng, 50_000, 3_000_000), cams=rng.randint(2, 12))
    if kind == "states":
        return dict(kind=kind, n=log_int(rng, 20_000, 1_000_000), w=w, h=h, states=rng.randint(1, 4),
                    frames=rng.randint(2, 12))
    if kind == "layers":
        return dict(kind=kind, n=log_int(rng, 20_000, 1_000_000), w=w, h=h, layers=rng.randint(1, 6))
    if kind == "display":
        return dict(kind=kind, w=w, h=h, lut=rng.choice([17, 33, 65]))
    if kind == "train":
        return dict(kind=kind, batch=rng.randint(1, 10), crop=2 * rng.randint(32, 128))
    return dict(kind="sort", n=log_int(rng, 1_000, 8_000_000), bits=rng.choice([32, 32, 24, 13]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + salt)


def scene_rows(world, n, seed):
    """n GpuGaussian rows (n x 64 float32) on the GPU with the distributions of
    scene.small_scene ("cube") or scene.room_scene ("room")."""
    g = generator(seed, 1)

    def normal(*shape, mu=0.0, sd=1.0):
        return torch.randn(*shape, device="cuda", generator=g) * sd + mu

    def uniform(*shape, lo=0.0, hi=1.0):
        return torch.rand(*shape, device="cuda", generator=g) * (hi - lo) + lo

    rows = torch.zeros(n, 64, device="cuda")
    if world == "cube":
        rows[:, 0:3] = uniform(n, 3, lo=-1.0, hi=1.0)
        log_scale, logit = normal(n, 3, mu=-4.0, sd=0.5), normal(n, sd=1.5)
    else:
        nc = int(round(0.7 * n))
        centres, stds = uniform(256, 3, lo=-5.0, hi=5.0), uniform(256, lo=0.05, hi=0.5)
        which = torch.randint(0, 256, (nc,), device="cuda", generator=g)
        rows[:nc, 0:3] = centres[which] + normal(nc, 3) * stds[which, None]
        face = torch.randint(0, 6, (n - nc,), device="cuda", generator=g)
        wall = uniform(n - nc, 3, lo=-7.0, hi=7.0)
        side = torch.where(face % 2 == 0, -7.0, 7.0) + normal(n - nc, sd=0.01)
        wall.scatter_(1, (face // 2)[:, None], side[:, None])
        rows[nc:, 0:3] = wall
        log_scale, logit = normal(n, 3, mu=-4.5, sd=0.7), normal(n, mu=0.5, sd=2.0)
    rows[:, 3] = torch.sigmoid(logit)
    rows[:, 4:7] = torch.exp(log_scale)
    quat = normal(n, 4)
    rows[:, 8:12] = quat / quat.norm(dim=1, keepdim=True)
    rows[:, 12:15] = normal(n, 3, sd=0.5)
    rows[:, 16:61] = normal(n, 45, sd=0.05)
    return rows


def orbit(seed, w, h, step=0):
    """A camera of the room's orbit; the seed says where the orbit starts."""
    pos, yaw, pitch = scene.orbit_pose((37 * int(seed) + step) % ORBIT, ORBIT)
    return R.camera_uniforms(pos, yaw, pitch, w, h)


def frame_camera(case, seed):
    if case.get("world") == "cube":
        return R.camera_uniforms(*scene.small_camera_pose(), case["w"], case["h"])
    return orbit(seed, case["w"], case["h"])


def batch_cams(case, seed):
    return [(R.camera_uniforms(p, y, pt, w, h), w, h)
            for p, y, pt, w, h in scene.batch_cameras(int(seed) % 100_000, case["cams"])]


def state_frames(case, seed):
    """(state a, state b, weight) of each frame: a playback over the states."""
    rng = np.random.default_rng(int(seed))
    a = rng.integers(0, case["states"] + 1, case["frames"])
    b = rng.integers(0, case["states"] + 1, case["frames"])
    return a, b, rng.uniform(0.0, 1.0, case["frames"]).astype(np.float32)


def state_deltas(case, seed):
    g = generator(seed, 2)
    d = [torch.randn(case["n"], 48, device="cuda", generator=g).mul_(20.0).round_().clamp_(-127, 127).to(torch.int8)
         for _ in range(case["states"])]
    return torch.stack(d), np.full(48, 1.0 / 256.0, np.float32)


def layer_halves(case, seed):
    g = generator(seed, 3)
    return torch.stack([torch.randn(case["n"], 48, device="cuda", generator=g).mul_(0.4).half()
                        for _ in range(case["layers"])])


def layer_weights(case, seed):
    return np.random.default_rng(int(seed)).uniform(0.1, 1.5, (case["layers"], 3)).astype(np.float32)


def display_input(case, seed):
    """A linear frame (radiance over about ten stops) and a smooth display table."""
    g = generator(seed, 4)
    rgb = torch.exp2(torch.randn(case["h"], case["w"], 4, device="cuda", generator=g) * 2.0 - 2.0)
    img = rgb.clamp_(max=1000.0).half()
    img[..., 3] = 1.0
    n = case["lut"]
    z, y, x = np.meshgrid(*[np.linspace(0.0, 1.0, n)] * 3, indexing="ij")
    lut = np.stack([0.9 * x + 0.1 * y, 0.9 * y + 0.1 * z, 0.9 * z + 0.1 * x], -1)
    lut = np.rint(65535.0 * np.clip(lut * lut * (3.0 - 2.0 * lut), 0.0, 1.0)).astype(np.uint16)
    return img, lut, -10.0, 6.0, 0.35


def train_input(case, seed):
    """Crops of a smooth picture (target), its two-sample noise and history
    (features), and He-initialised parameters."""
    g = generator(seed, 5)
    b, c = case["batch"], case["crop"]
    yy, xx = torch.meshgrid(torch.linspace(0.0, 6.0, c, device="cuda"), torch.linspace(0.0, 6.0, c, device="cuda"),
                            indexing="ij")
    phase = torch.rand(b, 4, 2, device="cuda", generator=g) * 6.28
    target = 0.5 + 0.4 * torch.sin(yy[None, None] + phase[:, :, 0, None, None]) * torch.cos(
        2.0 * xx[None, None] + phase[:, :, 1, None, None])
    target = target.permute(0, 2, 3, 1).contiguous()
    noise = torch.randn(b, c, c, 7, device="cuda", generator=g)
    x = torch.zeros(b, c, c, 16, device="cuda")
    x[..., 0:4] = target + 0.25 * noise[..., 0:4]
    x[..., 4] = 0.9 + 0.02 * target[..., 0]
    x[..., 5:8] = target[..., 0:3] + 0.05 * noise[..., 4:7]
    rng = np.random.default_rng(int(seed))
    flat = []
    for k, (cin, cout) in enumerate(LAYERS):
        sd = math.sqrt(2.0 / (9 * cin)) * (0.1 if k == len(LAYERS) - 1 else 1.0)
        flat += [rng.normal(0.0, sd, 9 * cin * cout), rng.normal(0.0, 0.01, cout)]
    return x.bfloat16(), target, np.concatenate(flat).astype(np.float32)


class Shown:
    """A renderer with its scene and the images it draws into."""

    def __init__(self, case, seed, mode="alpha", half=False, **knobs):
        self.r = R.Renderer(0, torch.cuda.current_stream().cuda_stream)
        self.r.set(splat_render_mode=mode, black_background=1, **knobs)
        rows = scene_rows(case.get("world", "room"), case["n"], seed)
        self.r.set_row_format(half)
        self.r.upload_gaussians_device(rows.data_ptr(), case["n"])
        torch.cuda.synchronize()

    def image(self, w, h):
        return torch.zeros(h, w, 4, dtype=torch.float16, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": int(seed), "passes": 0}
    if kind == "frame":
        s["show"] = Shown(case, seed, half=case["half"], sh_degree=case["degree"])
        s["cam"], s["out"] = frame_camera(case, seed), s["show"].image(case["w"], case["h"])
    elif kind in ("stochastic", "gps", "denoised"):
        knobs = {"stochastic": dict(stochastic_taa_current_samples=case.get("samples", 4)),
                 "gps": dict(gps_supersample_factor=case.get("ss", 2)), "denoised": {}}[kind]
        s["show"] = Shown(case, seed, mode=kind, **knobs)
        if kind == "gps":
            s["show"].r.set_gps_work_budget(case["budget"])
        if kind == "denoised":
            s["net"] = Denoiser(0, torch.cuda.current_stream().cuda_stream)
            s["net"].set_params(np.fromfile(L.LIB_PATH.parent / "denoiser_room3m.f32", "<f4"))
            s["show"].r.set_denoiser(s["net"])
        s["cams"] = [R.camera_from_array(orbit(seed, case["w"], case["h"], k)) for k in range(ORBIT)]
        s["out"] = s["show"].image(case["w"], case["h"])
    elif kind == "batch":
        s["show"] = Shown(case, seed)
        cams = batch_cams(case, seed)
        s["cams"], s["out"] = [R.camera_from_array(c) for c, _, _ in cams], [s["show"].image(w, h) for _, w, h in cams]
    elif kind == "states":
        s["show"] = Shown(case, seed)
        deltas, scales = state_deltas(case, seed)
        s["show"].r.upload_animation(deltas.cpu().numpy(), scales)
        s["cam"], s["frames"] = orbit(seed, case["w"], case["h"]), state_frames(case, seed)
        s["out"] = [s["show"].image(case["w"], case["h"]) for _ in range(case["frames"])]
    elif kind == "layers":
        s["show"] = Shown(case, seed, linear_color=1)
        s["show"].r.upload_layers(layer_halves(case, seed).view(torch.int16).cpu().numpy().view(np.uint16))
        s["cam"], s["weights"] = orbit(seed, case["w"], case["h"]), layer_weights(case, seed)
        s["out"] = s["show"].image(case["w"], case["h"])
    elif kind == "display":
        s["r"] = R.Renderer(0, torch.cuda.current_stream().cuda_stream)
        s["in"], lut, lo, hi, s["ev"] = display_input(case, seed)
        s["r"].set_display_lut(lut, lo, hi)
        s["out"] = torch.zeros(case["h"], case["w"], 4, device="cuda")
    elif kind == "train":
        s["x"], s["target"], params = train_input(case, seed)
        s["net"] = Denoiser(0, torch.cuda.current_stream().cuda_stream)
        s["net"].set_params(params)
    else:
        g = generator(seed, 6)
        n, bits = case["n"], case["bits"]
        if bits == 32:   # the depth keys of a frame: inverted bits of positive floats
            z = torch.rand(n, device="cuda", generator=g) * 15.0 + 0.2
            keys = torch.bitwise_not(z.view(torch.int32))
        else:
            keys = torch.randint(0, 1 << bits, (n,), device="cuda", generator=g, dtype=torch.int32)
        s["keys"], s["vals"] = keys, torch.arange(n, device="cuda", dtype=torch.int32)
        s["out"] = torch.empty_like(keys), torch.empty_like(keys)
        s["bytes"] = R.sort_pairs_scratch_bytes(n)
        s["scratch"] = torch.empty(s["bytes"], dtype=torch.uint8, device="cuda")
        s["stream"] = torch.cuda.current_stream().cuda_stream
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "frame":
        s["show"].r.draw_frame(s["cam"], out_ptr=s["out"].data_ptr())
        return s["out"]
    if kind in ("stochastic", "gps", "denoised"):
        cam = s["cams"][s["passes"] % ORBIT]   # the camera moves on along the orbit
        s["passes"] += 1
        s["show"].r.draw_frame(cam, out_ptr=s["out"].data_ptr())
        return s["out"]
    if kind == "batch":
        s["show"].r.render_batch(s["cams"], [o.data_ptr() for o in s["out"]])
        return s["out"]
    if kind == "states":
        a, b, w = s["frames"]
        s["show"].r.render_anim_batch(s["cam"], a, [o.data_ptr() for o in s["out"]], states_b=b, weights=w)
        return s["out"]
    if kind == "layers":
        s["show"].r.set_layer_weights(s["weights"])
        s["show"].r.draw_frame(s["cam"], out_ptr=s["out"].data_ptr())
        return s["out"]
    if kind == "display":
        s["r"].display(s["in"].data_ptr(), s["out"].data_ptr(), case["w"], case["h"], s["ev"])
        return s["out"]
    if kind == "train":
        b, c = case["batch"], case["crop"]
        s["net"].train_step(s["x"].data_ptr(), s["target"].data_ptr(), b, c, c, 1e-4, want_loss=False)
        return s["net"].grads()
    k, v = s["out"]
    R.sort_pairs(s["keys"].data_ptr(), s["vals"].data_ptr(), k.data_ptr(), v.data_ptr(), case["n"],
                 s["scratch"].data_ptr(), s["bytes"], 0, case["bits"], s["stream"])
    return {"keys": k, "vals": v}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def frame_work(n, w, h, row_bytes=256, world="room", blends=1.0):
    """The heads of all rows and the rest of the visible ones once, the image
    once; projection and SH of the visible rows, blending of their fragments."""
    vis = n * (1.0 if world == "cube" else VISIBLE)
    entries = vis * (ENTRIES if world != "cube" else 8.0) * (h / 1080.0) ** 2 + vis
    return {"bytes": 16.0 * n + (row_bytes - 16.0) * vis + 8.0 * w * h, "flops": 700.0 * vis + blends * 20.0 * 64.0 * entries}


def work(case):
    kind = case["kind"]
    if kind == "frame":
        row = 144 if case["half"] else 64 + 64 * case["degree"] if case["degree"] < 3 else 256
        return frame_work(case["n"], case["w"], case["h"], row, case["world"])
    if kind in ("stochastic", "gps", "denoised"):
        f = frame_work(case["n"], case["w"], case["h"])
        px = case["w"] * case["h"]
        if kind == "gps":   # 2 pi sqrt(det) Li2(opacity) pixels a splat, ss^2 points each, about 80 operations
            f["flops"] = 700.0 * case["n"] * VISIBLE + 16.0 * case["n"] * (case["h"] / 720.0) ** 2 * case["ss"] ** 2 * 80.0
        else:               # the temporal history (colour and position) read and written
            f["bytes"] += 64.0 * px
        if kind == "stochastic":
            f["flops"] += 30.0 * 64.0 * case["n"] * VISIBLE * case["samples"]
        if kind == "denoised":
            f["flops"] += 2.0 * 9.0 * px * (16 * 32 + 2 * 32 * 32 / 4 + 32 * 32 + 32 * 16)
        return f
    if kind == "batch":
        each = [frame_work(case["n"], w, h) for _, _, _, w, h in scene.batch_cameras(0, case["cams"])]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    if kind == "states":
        f = frame_work(case["n"], case["w"], case["h"])
        vis, k = VISIBLE * case["n"], case["frames"]
        return {"bytes": f["bytes"] + 48.0 * case["states"] * vis + 8.0 * (k - 1) * case["w"] * case["h"],
                "flops": k * f["flops"]}
    if kind == "layers":
        f = frame_work(case["n"], case["w"], case["h"], 64)
        f["bytes"] += 96.0 * case["layers"] * VISIBLE * case["n"]
        return f
    if kind == "display":
        px = case["w"] * case["h"]
        return {"bytes": 24.0 * px + 6.0 * case["lut"] ** 3, "flops": 120.0 * px}
    if kind == "train":
        px = case["batch"] * case["crop"] ** 2
        macs = 9.0 * px * (16 * 32 + 2 * 32 * 32 / 4 + 32 * 32 + 32 * 16)
        return {"bytes": 48.0 * px, "flops": 6.0 * macs}
    return {"bytes": 16.0 * case["n"], "flops": 0.0}


# ---------------------------------------------------------------------------
# The same in 64 bits: plain torch, without the library
# ---------------------------------------------------------------------------
def sh_colour(dirs, dc, sh, degree):
    """SH colour before the bias; dirs n x 3, dc n x 3, sh n x 15 x 3."""
    x, y, z = (dirs[:, k, None] for k in range(3))
    res = 0.28209479177387814 * dc
    if degree >= 1:
        res = res - SH_C1 * y * sh[:, 0] + SH_C1 * z * sh[:, 1] - SH_C1 * x * sh[:, 2]
    if degree >= 2:
        xx, yy, zz, xy, yz, xz = x * x, y * y, z * z, x * y, y * z, x * z
        for k, f in enumerate([xy, yz, 2 * zz - xx - yy, xz, xx - yy]):
            res = res + SH_C2[k] * f * sh[:, 3 + k]
    if degree >= 3:
        for k, f in enumerate([y * (3 * xx - yy), xy * z, y * (4 * zz - xx - yy), z * (2 * zz - 3 * xx - 3 * yy),
                               x * (4 * zz - xx - yy), z * (xx - yy), x * (xx - 3 * yy)]):
            res = res + SH_C3[k] * f * sh[:, 8 + k]
    return res


class Exact:
    """The sorted-alpha frame of one camera in 64 bits: geometry once, any colours."""

    def __init__(self, rows, cam, w, h):
        c = torch.tensor(np.asarray(cam, np.float64), device="cuda")
        V, P = c[0:16].view(4, 4), c[16:32]          # V[column][row]
        fxp = c[35]
        pos = rows[:, 0:3].double()
        v = pos @ V[0:3, 0:3] + V[3, 0:3]
        ndc = torch.stack([P[0] * v[:, 0], P[5] * v[:, 1]], 1) / -v[:, 2:3]
        vis = (v[:, 2] <= -0.2) & (ndc.abs() <= 1.3).all(1)
        self.ids = vis.nonzero()[:, 0]
        r, v = rows[self.ids].double(), v[self.ids]
        vx, vy, vz = v.unbind(1)
        qw, qx, qy, qz = r[:, 8:12].unbind(1)
        rot = torch.stack([1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy + qw * qz), 2 * (qx * qz - qw * qy),
                           2 * (qx * qy - qw * qz), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz + qw * qx),
                           2 * (qx * qz + qw * qy), 2 * (qy * qz - qw * qx), 1 - 2 * (qx * qx + qy * qy)], 1)
        m = rot.view(-1, 3, 3) * r[:, 4:7, None]     # row k: axis k scaled
        m = m @ V[0:3, 0:3]                          # in view space
        j = torch.zeros(len(r), 3, 2, dtype=torch.float64, device="cuda")
        j[:, 0, 0] = j[:, 1, 1] = fxp / vz
        j[:, 2, 0], j[:, 2, 1] = -fxp * vx / vz ** 2, -fxp * vy / vz ** 2
        p = m @ j
        cov = p.transpose(1, 2) @ p
        a, b, d = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
        det = (a * d - b * b).clamp_min(1e-6)
        cx, cy = fxp * vx / vz + w / 2, fxp * vy / vz + h / 2
        rx, ry = torch.ceil(3 * a.sqrt()), torch.ceil(3 * d.sqrt())
        z = (P[10] * vz + P[14]) / -vz
        camw = -(V[0:3, 0:3] @ V[3, 0:3])
        dirs = r[:, 0:3] - camw
        self.dirs = dirs / dirs.norm(dim=1, keepdim=True)
        self.row = r
        op = r[:, 3]
        cut = torch.log((1.0 / 255.0) / op.clamp_min(1e-8))
        # covered pixels: centres k + 0.5 of the quad snapped to 1/256, left and top edges inside,
        # and those the ellipse alpha >= 1/255 can reach
        i0, i1 = (torch.ceil((torch.round((cx + s * rx) * 256) - 128) / 256) for s in (-1, 1))
        j0, j1 = (torch.floor((torch.round((cy + s * ry) * 256) - 128) / 256) + 1 for s in (-1, 1))
        ok = (z.abs() <= 1) & (cut <= 0)
        k = (-2 * cut).clamp_min(0)
        ex, ey = (k * a).sqrt() + 1, (k * d).sqrt() + 1
        i0, i1 = torch.maximum(i0, torch.floor(cx - ex)).clamp(0, w), torch.minimum(i1, torch.ceil(cx + ex)).clamp(0, w)
        j0, j1 = torch.maximum(j0, torch.floor(cy - ey)).clamp(0, h), torch.minimum(j1, torch.ceil(cy + ey)).clamp(0, h)
        ok &= (i1 > i0) & (j1 > j0)
        back = torch.arange(len(r) - 1, -1, -1, device="cuda")
        order = back[torch.argsort(-vz[back], stable=True)]   # near to far; ties: the later index in front
        order = order[ok[order]]
        self.w, self.h, self.order = w, h, order
        self.geo = torch.stack([cx, cy, d / det, -b / det, a / det, op, cut], 1)[order]
        rect = torch.stack([i0, i1, j0, j1], 1)[order].long()
        self.rect = rect
        t0, t1 = rect[:, 0::2] // 16, (rect[:, 1::2] - 1) // 16
        size = t1 - t0 + 1
        count = size[:, 0] * size[:, 1]
        splat = torch.repeat_interleave(torch.arange(len(order), device="cuda"), count)
        at = torch.arange(len(splat), device="cuda") - torch.repeat_interleave(count.cumsum(0) - count, count)
        self.tx = (w + 15) // 16
        tile = (t0[splat, 1] + at // size[splat, 0]) * self.tx + t0[splat, 0] + at % size[splat, 0]
        tile, by = torch.sort(tile, stable=True)
        self.splat = splat[by]
        self.tiles, self.length = torch.unique_consecutive(tile, return_counts=True)
        self.first = self.length.cumsum(0) - self.length
        heavy = torch.argsort(-self.length)
        self.tiles, self.length, self.first = self.tiles[heavy], self.length[heavy], self.first[heavy]

    def colours(self, degree=3, dc=None, sh=None, bias=0.5):
        dc = self.row[:, 12:15] if dc is None else dc
        sh = self.row[:, 16:61].reshape(-1, 15, 3) if sh is None else sh
        return (sh_colour(self.dirs, dc, sh, degree) + bias).clamp_min(0)

    def image(self, rgb):
        """h x w x 4, top row first, on black."""
        w, h = self.w, self.h
        rgb = rgb[self.order]
        out = torch.zeros(((h + 15) // 16) * self.tx, 256, 4, dtype=torch.float64, device="cuda")
        px = torch.arange(256, device="cuda")
        lx, ly = px % 16, px // 16
        T = torch.ones(len(self.tiles), 256, dtype=torch.float64, device="cuda")
        C = torch.zeros(len(self.tiles), 256, 3, dtype=torch.float64, device="cuda")
        X = (self.tiles % self.tx)[:, None] * 16 + lx
        Y = (self.tiles // self.tx)[:, None] * 16 + ly
        lengths = self.length.cpu().numpy()
        live = torch.arange(len(self.tiles), device="cuda")
        for k in range(int(lengths[0]) if len(lengths) else 0):
            if k % 64 == 0:   # tiles with entries left whose light is not all taken
                live = live[(self.length[live] > k) & (T[live].amax(1) > 1e-7)]
                if not len(live):
                    break
            m = live[self.length[live] > k] if k % 64 else live
            s = self.splat[self.first[m] + k]
            cx, cy, ca, cb, cc, op, cut = self.geo[s].unsqueeze(1).unbind(2)
            x, y, rect = X[m], Y[m], self.rect[s][:, None, :]
            dx, dy = x + 0.5 - cx, y + 0.5 - cy
            power = -0.5 * (ca * dx * dx + 2 * cb * dx * dy + cc * dy * dy)
            keep = (power <= 0) & (power >= cut) & (x >= rect[..., 0]) & (x < rect[..., 1]) & (y >= rect[..., 2]) & \
                (y < rect[..., 3])
            wgt = torch.where(keep, (op * power.exp()).clamp_max(0.99), 0.0) * T[m]
            C[m] += wgt[..., None] * rgb[s][:, None, :]
            T[m] -= wgt
        out[..., 3] = 0.0
        out[self.tiles] = torch.cat([C, 1 - T[..., None]], 2)
        full = out.view(-1, self.tx, 16, 16, 4).permute(0, 2, 1, 3, 4).reshape(-1, self.tx * 16, 4)
        return full[:h, :w].flip(0)


def exact_train(case, seed):
    """Gradients of the training loss, 64-bit autograd."""
    x, target, flat = train_input(case, seed)
    x, t = x.double().permute(0, 3, 1, 2), target.double().permute(0, 3, 1, 2)
    flat = torch.tensor(flat, dtype=torch.float64, device="cuda", requires_grad=True)
    F = torch.nn.functional
    weights, o = [], 0
    for cin, cout in LAYERS:
        wt = flat[o:o + 9 * cin * cout].view(3, 3, cin, cout).permute(3, 2, 0, 1)
        o += 9 * cin * cout
        weights.append((wt, flat[o:o + cout]))
        o += cout

    def conv(v, k):   # as a sum over taps: 64-bit matrix products
        wt, b = weights[k]
        p = F.pad(v, (1, 1, 1, 1))
        h, w = v.shape[2:]
        return sum(torch.einsum("bchw,oc->bohw", p[:, :, i:i + h, j:j + w], wt[:, :, i, j])
                   for i in range(3) for j in range(3)) + b[None, :, None, None]

    e1 = F.relu(conv(x, 0))
    e3 = F.relu(conv(F.relu(conv(F.avg_pool2d(e1, 2), 1)), 2))
    d4 = F.relu(conv(F.interpolate(e3, scale_factor=2, mode="nearest") + e1, 3))
    pred = torch.cat([x[:, 5:8], x[:, 3:4]], 1) + conv(d4, 4)[:, 0:4]
    o4 = conv(d4.detach(), 4)[:, 4]      # the error head trains the last layer alone
    k = torch.exp(-torch.arange(-5, 6, dtype=torch.float64, device="cuda") ** 2 / (2 * 1.5 ** 2))
    k = k / k.sum()

    def blur(v):      # interior pixels
        v = sum(k[i] * v[:, :, i:v.shape[2] - 10 + i] for i in range(11))
        return sum(k[i] * v[:, :, :, i:v.shape[3] - 10 + i] for i in range(11))

    p, q = pred[:, 0:3], t[:, 0:3]
    mx, my = blur(p), blur(q)
    sxx, syy, sxy = blur(p * p) - mx * mx, blur(q * q) - my * my, blur(p * q) - mx * my
    ssim = ((2 * mx * my + 1e-4) * (2 * sxy + 9e-4)) / ((mx * mx + my * my + 1e-4) * (sxx + syy + 9e-4))
    err = 1000.0 * ((pred - t) ** 2).mean(1).detach()
    loss = (pred - t).abs().mean() + 0.2 * (1 - ssim.mean()) + 0.01 * ((o4 - err) ** 2).mean()
    return torch.autograd.grad(loss, flat)[0]


def exact_display(case, seed):
    img, lut, lo, hi, ev = display_input(case, seed)
    n = case["lut"]
    table = torch.tensor(lut.astype(np.float64) / 65535.0, device="cuda").reshape(-1, 3)
    rad = (img[..., 0:3].double() * 2.0 ** ev).clamp_min(2.0 ** lo)
    p = ((torch.log2(rad) - lo) / (hi - lo)).clamp(0, 1) * (n - 1)
    i0 = p.floor().long()
    i1, f = (i0 + 1).clamp_max(n - 1), p - i0
    rgb = 0.0
    for k in range(8):
        bits = [(k >> c) & 1 for c in range(3)]
        at = [(i1 if b else i0)[..., c] for c, b in enumerate(bits)]
        wt = math.prod((f if b else 1 - f)[..., c] for c, b in enumerate(bits))
        rgb = rgb + wt[..., None] * table[(at[2] * n + at[1]) * n + at[0]]
    return torch.cat([rgb, torch.ones_like(rgb[..., :1])], -1)


def exact(case, seed):
    """None where a pass has no 64-bit value: the hashed samples of the
    stochastic, point and denoised modes, and the sort's whole numbers."""
    kind = case["kind"]
    if kind == "train":
        return exact_train(case, seed)
    if kind == "display":
        return exact_display(case, seed)
    if kind not in ("frame", "batch", "states", "layers"):
        return None
    rows = scene_rows(case.get("world", "room"), case["n"], seed)
    if kind == "frame":
        if case["half"]:   # the row format the caller chose
            rows[:, 12:15] = rows[:, 12:15].half().float()
            rows[:, 16:61] = rows[:, 16:61].half().float()
        e = Exact(rows, frame_camera(case, seed), case["w"], case["h"])
        return e.image(e.colours(case["degree"]))
    if kind == "batch":    # the first three frames: more would take too long
        out = []
        for cam, w, h in batch_cams(case, seed)[:3]:
            e = Exact(rows, cam, w, h)
            out.append(e.image(e.colours()))
        return out + [None] * (case["cams"] - len(out))
    e = Exact(rows, orbit(seed, case["w"], case["h"]), case["w"], case["h"])
    if kind == "states":   # the first three states
        deltas, scales = state_deltas(case, seed)
        scale = torch.tensor(scales, device="cuda").double()
        base = torch.cat([e.row[:, 12:15], e.row[:, 16:61].reshape(-1, 15, 3).transpose(1, 2).reshape(-1, 45)], 1)

        def coeff(state):
            return base if state == 0 else base + deltas[state - 1][e.ids].double() * scale

        out = []
        for a, b, wt in list(zip(*state_frames(case, seed)))[:3]:
            c = (1.0 - float(wt)) * coeff(int(a)) + float(wt) * coeff(int(b))
            out.append(e.image(e.colours(3, c[:, 0:3], c[:, 3:].reshape(-1, 3, 15).transpose(1, 2))))
        return out + [None] * (case["frames"] - len(out))
    rgb = 0.0
    for half, wt in zip(layer_halves(case, seed), layer_weights(case, seed)):
        c = half[e.ids].double()
        sh = c[:, 3:].reshape(-1, 3, 15).transpose(1, 2)
        rgb = rgb + e.colours(3, c[:, 0:3], sh, bias=0.0) * torch.tensor(wt, device="cuda").double()
    return e.image(rgb)
