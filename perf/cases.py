"""The work that programs have this library do, as timed cases.

Every case goes through the package's public entry points: frames of the
reference renderer's qualities into device or host memory, batches of frames,
ray and ball batches, and trees built from voxel sets or raw volumes.  The
volumes are seeded value noise (a CT-like scan) or Gaussian blobs, the sizes
those of the benchmark and the tests.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import voxvision_gb300 as vg
from voxvision_gb300.cameras import HostCamera

BEST, FAST, ADAPTIVE, MERGE = 0, 1, 2, 6   # the quality values of vox_context_set_quality

RESOLUTIONS = [(320, 240), (640, 480), (1280, 720), (1920, 1080), (3840, 2160)]
MIXED_TREES = [(64, 0.05), (128, 0.10), (256, 0.15), (512, 0.20)]   # side, solid share of the resident volumes


def listed():
    return [
        # a preview or thumbnail, the smallest frame: launch latency counts
        {"name": "frame 256x256 blobs 64", "kind": "frame", "volume": "blobs", "side": 64, "solid": 0.20,
         "w": 256, "h": 256, "quality": BEST, "camera": "simple", "distance": 1.5},
        # a viewer's full-HD frame of a scan, every pixel traced
        {"name": "frame 1080p best 256", "kind": "frame", "volume": "noise", "side": 256, "solid": 0.08,
         "w": 1920, "h": 1080, "quality": BEST, "camera": "simple", "distance": 1.5},
        # the same viewer in the renderer's default quality
        {"name": "frame 1080p adaptive 256", "kind": "frame", "volume": "noise", "side": 256, "solid": 0.08,
         "w": 1920, "h": 1080, "quality": ADAPTIVE, "camera": "simple", "distance": 1.5},
        # a walk close to a large volume on a 4K screen: the tree fills the frame
        {"name": "frame 4k fast 512 near", "kind": "frame", "volume": "noise", "side": 512, "solid": 0.10,
         "w": 3840, "h": 2160, "quality": FAST, "camera": "doom", "distance": 0.7},
        # an orbit rendered to device frames in one batch (video, thumbnails of a turntable)
        {"name": "orbit batch 32x1080p 256", "kind": "orbit", "volume": "noise", "side": 256, "solid": 0.08,
         "w": 1920, "h": 1080, "frames": 32, "distance": 1.5},
        # many viewers' frames of uneven sizes over four resident volumes
        {"name": "mixed batch 24 of 4 trees", "kind": "mixed", "frames": 24},
        # the orbit delivered into the caller's page-locked host frames
        {"name": "host frames 24x1080p 256", "kind": "host_frames", "volume": "noise", "side": 256, "solid": 0.08,
         "w": 1920, "h": 1080, "frames": 24, "distance": 1.5},
        # one frame lit by a light manager, into ordinary host memory
        {"name": "host lit 720p merge 128", "kind": "host_lit", "volume": "noise", "side": 128, "solid": 0.10,
         "w": 1280, "h": 720, "quality": MERGE, "camera": "simple", "distance": 0.9, "lights": 64},
        # visibility or sensor queries: rays from anywhere in any direction
        {"name": "rays 4M 256", "kind": "rays", "volume": "noise", "side": 256, "solid": 0.08, "n": 1 << 22},
        # a picking or collision loop on the host: a few rays a call
        {"name": "rays host 100 256", "kind": "rays_host", "volume": "noise", "side": 256, "solid": 0.08, "n": 100},
        # collision queries of many bodies at once
        {"name": "balls 1M 256", "kind": "balls", "volume": "noise", "side": 256, "solid": 0.08, "n": 1000000,
         "rmin": 0.5, "rmax": 8.0},
        # loading a raw 8-bit scan and looking at it
        {"name": "raw volume 256 u8", "kind": "raw", "side": 256, "solid": 0.08, "bytes": 1},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame", "frame", "frame", "orbit", "mixed", "host_frames", "host_lit", "rays", "rays_host",
                       "balls", "balls", "raw", "voxels"])
    blobs = rng.random() < 0.2
    c = {"kind": kind, "volume": "blobs" if blobs else "noise", "side": rng.randint(40, 96) if blobs else log(64, 400),
         "solid": 0.20 if blobs else round(rng.uniform(0.04, 0.20), 3)}
    if kind in ("frame", "host_lit"):
        c.update(w=16 * log(12, 240), h=4 * log(40, 540),
                 quality=rng.choice([BEST, FAST, ADAPTIVE, MERGE]), camera=rng.choice(["simple", "doom"]),
                 distance=round(rng.uniform(0.3, 1.6), 2))
        if kind == "host_lit":
            c["lights"] = log(1, 200)
    elif kind in ("orbit", "host_frames"):
        w, h = 16 * log(20, 120), 4 * log(60, 270)
        most = 24 if kind == "host_frames" else 32
        c.update(w=w, h=h, frames=log(2, max(2, min(most, most * 1920 * 1080 // (w * h)))),
                 distance=round(rng.uniform(1.0, 1.6), 2))
    elif kind == "mixed":
        c = {"kind": kind, "frames": rng.randint(4, 24)}
    elif kind == "rays":
        c["n"] = log(1000, 1 << 22)
    elif kind == "rays_host":
        c["n"] = log(1, 20000)
    elif kind == "balls":
        c.update(n=log(1000, 1000000), rmin=0.5, rmax=round(rng.uniform(1.0, 8.0), 2))
    else:
        if kind == "raw":
            c = {"kind": kind, "solid": c["solid"], "bytes": rng.choice([1, 2])}
        c["side"] = rng.randint(40, 96) if c.get("volume") == "blobs" else log(40, 224)
        c["solid"] = min(c["solid"], 0.20 if c.get("volume") == "blobs" else 0.10)
    return c


# ------------------------------------------------------------------ inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(0x5EED0000 + seed)
    return g


def _noise_u8(side, g, spacing=16):
    """Trilinear-upsampled value noise, (side, side, side) uint8: the shape of a CT scan."""
    m = (side - 1) // spacing + 2
    lat = torch.randint(0, 256, (m, m, m), generator=g, device="cuda").to(torch.float32)
    at = torch.arange(side, device="cuda")
    i, t = at // spacing, (at % spacing).to(torch.float32) / spacing
    s = lat[i] * (1 - t)[:, None, None] + lat[i + 1] * t[:, None, None]
    s = s[:, i] * (1 - t)[None, :, None] + s[:, i + 1] * t[None, :, None]
    s = s[:, :, i] * (1 - t) + s[:, :, i + 1] * t
    return s.clamp_(0, 255).to(torch.uint8)


def _band(vol, solid):
    """The smallest band [lo, hi] around 128 that holds the solid share of the samples."""
    hist = torch.bincount(vol.reshape(-1), minlength=256).tolist()
    for w in range(1, 256):
        lo = max(0, min(256 - w, 128 - w // 2))
        if sum(hist[lo:lo + w]) >= solid * vol.numel():
            break
    return lo, lo + w - 1


def _mask(case, seed):
    """Which samples of the case's volume are solid."""
    g, side = _generator(seed), case["side"]
    if case["volume"] == "noise":
        vol = _noise_u8(side, g)
        lo, hi = _band(vol, case["solid"])
        return (vol >= lo) & (vol <= hi)
    vol = 16 * torch.rand((side, side, side), generator=g, device="cuda")
    at = torch.arange(side, device="cuda", dtype=torch.float32)
    for _ in range(20):   # Gaussian blobs of sigma 3..10
        u = torch.rand(4, generator=g, device="cuda")
        e = [torch.exp(-((at - u[a] * side) ** 2) / (2 * (3 + 7 * u[3]) ** 2)) for a in range(3)]
        vol += 255 * e[0][:, None, None] * e[1][None, :, None] * e[2][None, None, :]
    k = int((1 - case["solid"]) * vol.numel())
    return vol > vol.reshape(-1).kthvalue(max(1, k)).values


def _voxels(mask):
    """The solid samples' corners in the order of a raw volume, (n, 3) float32."""
    return mask.nonzero().to(torch.float32).contiguous()


def _tree(case, seed):
    return vg.DeviceTree.build_device(_voxels(_mask(case, seed)))


def _texture(seed):
    return torch.randint(0, 256, (32 * 32 * 32,), generator=_generator(seed + 77), device="cuda").to(torch.uint8)


def _camera(kind, w, h, side, distance, azimuth, elevation):
    """A camera `distance` volume diagonals from the centre of the volume, looking at it."""
    cam = HostCamera(1 if kind == "doom" else 0)
    cam.set_fov(1.0)
    cam.set_window_size(w, h)
    c, r = side / 2.0, distance * side * math.sqrt(3.0)
    if kind == "doom":   # yaw only: the camera stands level with the volume
        elevation = 0.0
    p = np.array([c + r * math.cos(elevation) * math.cos(azimuth), c + r * math.cos(elevation) * math.sin(azimuth),
                  c + r * math.sin(elevation)], np.float32)
    cam.set_position(p)
    cam.look_at(np.full(3, c, np.float32))
    return cam.gpu_struct()


def _rays(case, seed, g):
    """Origins in a box twice the volume's, directions on the sphere."""
    n, side = case["n"], case["side"]
    o = (torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64) * 2 - 0.5) * side
    d = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    d = d / d.norm(dim=1, keepdim=True)
    return o.to(torch.float32).contiguous(), d.to(torch.float32).contiguous()


def _lights(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    m, side = vg.LightManager(), case["side"]
    m.ambient((0.2, 0.2, 0.25))
    for _ in range(case["lights"]):
        m.insert(r.uniform(0, side, 3), r.uniform(0.05, 0.4) * side, r.uniform(0.1, 1.0, 3))
    return m


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    r = np.random.RandomState((seed + 12345) % (1 << 31))
    if kind in ("frame", "orbit", "host_frames", "host_lit"):
        w, h, side = case["w"], case["h"], case["side"]
        s["tree"] = _tree(case, seed)
        turn = r.uniform(0, 2 * math.pi)
        if kind in ("frame", "host_lit"):
            s["cams"] = [_camera(case["camera"], w, h, side, case["distance"], turn, math.radians(r.uniform(5, 45)))]
        else:
            s["cams"] = [_camera("simple", w, h, side, case["distance"], turn + 2 * math.pi * i / 120,
                                 math.radians(20)) for i in range(case["frames"])]
        tex = _texture(seed)
        if kind in ("frame", "orbit"):
            s["tex"] = tex
            s["out"] = torch.empty((len(s["cams"]), h, w), dtype=torch.int32, device="cuda")
        else:
            s["tex"] = tex.cpu().numpy()
        if kind == "orbit":
            s["batch"] = vg.FrameBatch([(s["tree"], c, w, h, tex, s["out"][i]) for i, c in enumerate(s["cams"])],
                                       vg.BatchConfig(8, 4, 2, 8, 0))
        elif kind == "host_frames":
            s["out"] = torch.empty((case["frames"], h, w), dtype=torch.int32, pin_memory=True)
            s["frames"] = [s["out"][i] for i in range(case["frames"])]
        elif kind == "host_lit":
            s["lights"] = _lights(case, seed).upload()
    elif kind == "mixed":
        s["tex"] = _texture(seed)
        s["trees"] = [_tree({"volume": "noise", "side": n, "solid": solid}, seed + i)
                      for i, (n, solid) in enumerate(MIXED_TREES)]
        jobs, s["out"] = [], []
        for i in range(case["frames"]):   # every size over every tree
            t, (w, h) = i % 4, RESOLUTIONS[i % 5]
            s["out"].append(torch.empty((h, w), dtype=torch.int32, device="cuda"))
            cam = _camera("simple", w, h, MIXED_TREES[t][0], 1.5, r.uniform(0, 2 * math.pi),
                          math.radians(r.uniform(5, 45)))
            jobs.append((s["trees"][t], cam, w, h, s["tex"], s["out"][-1]))
        s["batch"] = vg.FrameBatch(jobs, vg.BatchConfig(8, 4, 1, 8, 0))
    elif kind in ("rays", "rays_host"):
        s["tree"] = _tree(case, seed)
        o, d = _rays(case, seed, _generator(seed + 991))
        if kind == "rays":
            s.update(o=o, d=d, leaf=torch.zeros(case["n"], dtype=torch.int32, device="cuda"),
                     slot=torch.zeros(case["n"], dtype=torch.uint8, device="cuda"), points=torch.zeros_like(o))
        else:
            s.update(o=o.cpu().numpy(), d=d.cpu().numpy())
    elif kind == "balls":
        s["tree"] = _tree(case, seed)
        g, n = _generator(seed + 992), case["n"]
        s["c"] = (torch.rand((n, 3), generator=g, device="cuda") * case["side"]).contiguous()
        s["r"] = case["rmin"] + (case["rmax"] - case["rmin"]) * torch.rand(n, generator=g, device="cuda")
        s["hit"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
    else:   # a tree made in the pass, and a small frame of it
        w, h, side = 640, 480, case["side"]
        if kind == "raw":
            vol = _noise_u8(side, _generator(seed))
            s["band"] = _band(vol, case["solid"])
            if case["bytes"] == 2:   # the same scan in 16-bit samples
                s["samples"] = (vol.to(torch.int32) * 257).cpu().numpy().astype("<u2")
                s["band"] = (s["band"][0] * 257, s["band"][1] * 257)
            else:
                s["samples"] = vol.cpu().numpy()
        else:
            s["voxels"] = _voxels(_mask(case, seed))
        s["cam"] = _camera("simple", w, h, side, 1.2, r.uniform(0, 2 * math.pi), math.radians(20))
        s["tex"] = _texture(seed)
        s["out"] = torch.empty((h, w), dtype=torch.int32, device="cuda")
        s["wh"] = (w, h)
    return s


def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "frame":
        if c["quality"] == BEST:
            s["tree"].render_device(s["cams"][0], c["w"], c["h"], s["tex"], s["out"])
        else:
            s["tree"].render_quality_device(s["cams"][0], c["w"], c["h"], c["quality"], s["tex"], s["out"])
        return s["out"]
    if kind in ("orbit", "mixed"):
        s["batch"].launch()
        return s["out"]
    if kind == "host_frames":
        s["tree"].render_frames(s["cams"], c["w"], c["h"], s["tex"], s["frames"])
        return s["out"]
    if kind == "host_lit":
        return s["tree"].render_lit(s["cams"][0], c["w"], c["h"], c["quality"], s["tex"], s["lights"]).view(np.int32)
    if kind == "rays":
        s["tree"].rays_device(s["o"], s["d"], s["leaf"], s["slot"], s["points"])
        return {"leaf": s["leaf"], "slot": s["slot"], "points": s["points"]}
    if kind == "rays_host":
        leaf, slot, points = s["tree"].rays(s["o"], s["d"])
        return {"leaf": leaf.view(np.int32), "slot": slot, "points": points}
    if kind == "balls":
        s["tree"].balls_device(s["c"], s["r"], s["hit"])
        return s["hit"]
    if kind == "raw":
        tree = vg.DeviceTree.from_raw(s["samples"], (c["side"],) * 3, c["bytes"], s["band"][0], s["band"][1])
    else:
        tree = vg.DeviceTree.build_device(s["voxels"])
    s["tree"] = tree   # the program keeps the volume it looks at; the one before it goes
    tree.render_device(s["cam"], s["wh"][0], s["wh"][1], s["tex"], s["out"])
    return {"frame": s["out"], "tree": tree.info()}


def work(case):
    """The bytes a pass reads and writes by its nature: queries, samples or
    voxels in, frames, answers or the tree out.  (The nodes a search visits
    depend on the data and are not counted.)"""
    kind, tex = case["kind"], 32768
    if kind in ("frame", "host_lit"):
        b = 4 * case["w"] * case["h"] + tex
    elif kind in ("orbit", "host_frames"):
        b = 4 * case["w"] * case["h"] * case["frames"] + tex
    elif kind == "mixed":
        b = sum(4 * RESOLUTIONS[i % 5][0] * RESOLUTIONS[i % 5][1] for i in range(case["frames"])) + tex
    elif kind in ("rays", "rays_host"):
        b = case["n"] * (24 + 4 + 1 + 12)
    elif kind == "balls":
        b = case["n"] * (16 + 1)
    else:
        samples, voxels = case["side"] ** 3, case["solid"] * case["side"] ** 3
        # about 0.4 nodes of 48 bytes and an id of 4, and 0.5 stored voxels of 16, to a solid sample
        b = (samples * case["bytes"] if kind == "raw" else 12 * voxels) + voxels * (0.4 * 52 + 0.5 * 16) + 4 * 640 * 480
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    """Rays' intersection points in 64 bits: the first solid voxel along each
    ray by a walk of the grid's cells.  The other cases' outputs are whole."""
    if case["kind"] not in ("rays", "rays_host"):
        return None
    mask, side, n = _mask(case, seed), case["side"], case["n"]
    o, d = (x.to(torch.float64) for x in _rays(case, seed, _generator(seed + 991)))
    box = mask.nonzero()
    lo, hi = box.min(0).values.to(torch.float64), box.max(0).values.to(torch.float64) + 1
    ta, tb = (lo - o) / d, (hi - o) / d
    t0 = torch.minimum(ta, tb).amax(1).clamp_min(0.0)
    t1 = torch.maximum(ta, tb).amin(1)
    points = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    live = (t0 <= t1).nonzero().squeeze(1)
    o, d, t, step = o[live], d[live], t0[live], (d[live] > 0).to(torch.int64) * 2 - 1
    at = torch.minimum(torch.maximum((o + t[:, None] * d).floor(), lo), hi - 1).to(torch.int64)
    for _ in range(3 * side + 3):
        if live.numel() == 0:
            break
        solid = mask[at[:, 0], at[:, 1], at[:, 2]]
        points[live[solid]] = (o + t[:, None] * d)[solid]
        nxt = (at + (step > 0).to(torch.int64)).to(torch.float64)
        tn = (nxt - o) / d
        t, axis = tn.min(1)
        at = at + step * torch.nn.functional.one_hot(axis, 3)
        keep = ~solid & ((at >= lo) & (at < hi)).all(1)
        live, o, d, t, step, at = live[keep], o[keep], d[keep], t[keep], step[keep], at[keep]
    return {"leaf": None, "slot": None, "points": points.cpu().numpy()}
