"""The work that users of this framework have it do, as timed cases through the public Python entry points.

Every case is a dict of plain values; ``kind`` says which call it stands for:

* ``run``        one photometric run on host states (``PatchMatchSession.run``), the trait call of a host driver;
* ``schedule``   the whole single-level schedule on resident states (``schedule_resident``) and the download of the
                 filtered maps: the way a batch of views is densified;
* ``multiscale`` the coarse-to-fine driver with the fast profile (``densify.compute_depth_maps_resident``);
* ``host``       a whole job through the host-buffer interface: session begin (image upload), ``schedule_host``, end;
* ``calls``      the session's single calls on host states: evaluate, upsample, median filter, filter;
* ``learned``    proposals from the network, then the short schedule that starts from them;
* ``train``      loss and parameter gradients of the proposal network for one batch;
* ``fuse``       readout, speckle removal, consistency fusion and the download of the cloud.

Images are 8-bit gray (f32 where the case says so) of a seeded rolling terrain with a noise texture, rendered on the
GPU and seen by the camera formations of ``cumulus3d_b200.scenes``.  ``tuning`` is the half-step variant a program asks
for: 0 is the default, 10 and 42 are what the autotuner returns for large and for small batches.
"""
import math

import numpy as np
import torch

from cumulus3d_b200 import _lib, densify, fusion, proposal, scenes
from cumulus3d_b200.patchstereo import DepthSnapshot, PatchMatchBackend, RunParams, ViewState


def listed():
    return [
        # one call of a host driver on a thumbnail-sized pair with odd sides: launches and latency
        {"name": "run_thumbnail", "kind": "run", "w": 161, "h": 119, "views": 3, "sources": 2, "radius": 3, "step": 1,
         "iters": 2, "tuning": 0, "f32": False},
        # 3 cameras at 640x480, 11x11 window, 5 iterations
        {"name": "vga_triplet", "kind": "schedule", "sizes": "640x480", "views": 3, "sources": 2, "radius": 5, "step": 1,
         "iters": 5, "rounds": 0, "geo": 0, "tuning": 42, "f32": False},
        # drone imagery at 1920x1080, 13x13 window, 4 sources, photometric and geometric iterations
        {"name": "drone_1080p", "kind": "schedule", "sizes": "1920x1080", "views": 5, "sources": 4, "radius": 6,
         "step": 1, "iters": 2, "rounds": 1, "geo": 1, "tuning": 10, "f32": False},
        # an uneven batch: image sizes and source counts differ, some sides are odd
        {"name": "mixed_batch", "kind": "schedule", "sizes": "960x540,1280x720,801x603,640x361", "views": 8,
         "sources": 5, "radius": 6, "step": 1, "iters": 3, "rounds": 1, "geo": 2, "tuning": 10, "f32": False},
        # one 3840x2160 view against 5 sources, the largest image
        {"name": "uhd_view", "kind": "schedule", "sizes": "3840x2160", "views": 1, "sources": 5, "radius": 6, "step": 1,
         "iters": 2, "rounds": 0, "geo": 0, "tuning": 10, "f32": False},
        # f32 images and a window that has no kernel of its own
        {"name": "f32_window9", "kind": "schedule", "sizes": "401x299", "views": 4, "sources": 3, "radius": 4, "step": 1,
         "iters": 3, "rounds": 1, "geo": 1, "tuning": 0, "f32": True},
        # the coarse-to-fine fast profile: 9 views of 384x288, 3 scales, 11x11 window with step 2
        {"name": "fast_profile", "kind": "multiscale", "w": 384, "h": 288, "views": 9, "sources": 8, "radius": 5,
         "step": 2, "iters": 6, "rounds": 2, "geo": 2, "tuning": 0, "f32": False},
        # a job through the host-buffer interface, upload and every host state included
        {"name": "host_job_540p", "kind": "host", "w": 960, "h": 540, "views": 6, "sources": 4, "radius": 6, "step": 1,
         "iters": 2, "rounds": 1, "geo": 1, "tuning": 10, "f32": False},
        # the session's single calls on host states
        {"name": "single_calls_vga", "kind": "calls", "w": 640, "h": 480, "views": 4, "sources": 3, "radius": 5,
         "step": 1, "tuning": 10, "f32": False},
        # learned start: sweep, network, decode, 2 + 1 iterations
        {"name": "learned_720p", "kind": "learned", "w": 1280, "h": 720, "views": 3, "sources": 2, "radius": 6, "step": 1,
         "iters": 2, "rounds": 1, "geo": 1, "tuning": 10, "f32": False},
        # one training batch of 256x256 crops
        {"name": "train_batch8", "kind": "train", "w": 256, "h": 256, "batch": 8},
        # maps of 12 views to a point cloud
        {"name": "fuse_540p", "kind": "fuse", "w": 960, "h": 540, "views": 12, "sources": 4, "radius": 5, "step": 1,
         "tuning": 10, "f32": False},
    ]


#: Multiplications and additions that the largest listed case's windows take; a drawn case stays below it.
_MOST = 2.0e12


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "schedule", "schedule", "schedule", "schedule", "multiscale", "host", "calls", "learned",
                       "train", "fuse"])
    radius, step = rng.choice([(3, 1), (5, 1), (5, 2), (6, 1), (6, 1), (4, 1), (7, 2)])
    f32 = rng.random() < 0.15
    views = rng.randint(3, 8)
    sources = rng.randint(2, min(5, views - 1))
    tuning = rng.choice([0, 10, 10, 42])
    if kind == "train":
        return {"kind": kind, "w": 8 * rng.randint(8, 32), "h": 8 * rng.randint(8, 32), "batch": rng.randint(1, 8)}
    while True:
        w = _log(rng, 120, 1920)
        h = max(90, int(w * rng.uniform(0.5, 0.8)))
        iters, rounds, geo = rng.randint(1, 4), rng.randint(0, 1), rng.randint(1, 2)
        c = {"kind": kind, "w": w, "h": h, "views": views, "sources": sources, "radius": radius, "step": step,
             "iters": iters, "rounds": rounds, "geo": geo, "tuning": tuning, "f32": f32}
        if kind == "schedule":
            del c["w"], c["h"]
            c["sizes"] = ",".join("%dx%d" % (max(120, int(w * s)), max(90, int(h * s)))
                                  for s in [1.0] + [rng.uniform(0.5, 1.0) for _ in range(rng.randint(0, 2))])
        elif kind == "run":
            del c["rounds"], c["geo"]
        elif kind == "multiscale":
            w = c["w"] = min(w, 800)
            c["h"] = min(h, 600)
            c["f32"] = False
            if min(c["w"], c["h"]) < 128:
                continue
        elif kind == "calls":
            if min(w, h) < 128 or w > 1280:
                continue
            for k in ("iters", "rounds", "geo"):
                del c[k]
            c["f32"] = False
        elif kind == "learned":
            c["radius"], c["step"], c["f32"] = 6, 1, False
        elif kind == "fuse":
            c["views"] = rng.randint(4, 12)
            for k in ("iters", "rounds", "geo"):
                del c[k]
        if work(c)["flops"] <= _MOST:
            return c


def _sizes(case):
    if "sizes" in case:
        s = [tuple(int(x) for x in t.split("x")) for t in case["sizes"].split(",")]
        n = _num_cams(case)
        return [s[i % len(s)] for i in range(n)]
    return [(case["w"], case["h"])] * _num_cams(case)


def _num_cams(case):
    """Cameras of the session: every view that runs, and at least as many as its sources need."""
    return max(case["views"], case["sources"] + 1)


def work(case):
    """Bytes: images and states read once, results written once.  Operations: the NCC windows that a pass cannot do
    without (9 propagated hypotheses per source and iteration at most half of the refinement's; 33 operations a tap),
    or the network's multiplications and additions."""
    kind = case["kind"]
    if kind == "train":
        px = case["batch"] * case["w"] * case["h"]
        return {"bytes": px * (48 * 2 + 6 * 4) + proposal.NUM_PARAMS * 8, "flops": 3 * _net_flops() * px}
    sizes = _sizes(case)
    px = sum(w * h for w, h in sizes[: case["views"]])
    image = sum(w * h for w, h in sizes) * (4 if case["f32"] else 1)
    tap = 33 * ((2 * case["radius"]) // case["step"] + 1) ** 2
    win = px * case["sources"] * tap
    if kind == "fuse":
        return {"bytes": image + px * 20 + px * 8, "flops": px * 12 * 60}
    if kind == "calls":
        return {"bytes": image + px * (20 * 5 + 5), "flops": 2 * win}
    its = case["iters"] + case.get("rounds", 0) * case.get("geo", 0)
    if kind == "multiscale":
        # finest scale (3 photometric iterations there) and the coarser ones, 1/4 and 1/16 of its pixels
        its = (3 + case["rounds"] * case["geo"]) * 1.25 + 6 / 16.0
    flops = win * (1 + its * 12)
    bytes_ = image + px * 20
    if kind == "learned":
        flops += px * (_net_flops() + 32 * 2 * 33 * 49)
    if kind in ("host", "run"):
        bytes_ += px * 20
    return {"bytes": bytes_, "flops": flops}


def _net_flops():
    """Multiplications and additions per input pixel of the proposal network (12 convolutions on 4 scales)."""
    scale = (1, 1, 4, 4, 16, 16, 64, 64, 16, 4, 1, 1)
    return sum(18 * ci * co / s for (ci, co), s in zip(proposal.LAYERS, scale))


# ---------------------------------------------------------------------------------------------------- inputs
class _Terrain:
    """z = h(x, y), a few seeded waves, with a texture of four octaves of value noise."""

    def __init__(self, seed, cell):
        g = torch.Generator().manual_seed(seed)
        self.freq = (torch.rand(6, 2, generator=g, dtype=torch.float64) - 0.5) * 0.5
        self.phase = torch.rand(6, generator=g, dtype=torch.float64) * 6.2832
        self.amp = 0.3 + torch.rand(6, generator=g, dtype=torch.float64) * 0.9
        self.grid = torch.rand(4, 256, 256, generator=g).cuda()
        self.cell = cell
        self.gen = torch.Generator(device="cuda").manual_seed(seed + 1)

    def height(self, x, y):
        z, gx, gy = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)
        for (fx, fy), p, a in zip(self.freq.tolist(), self.phase.tolist(), self.amp.tolist()):
            arg = x * fx + y * fy + p
            z += a * torch.sin(arg)
            c = a * torch.cos(arg)
            gx += c * fx
            gy += c * fy
        return z, gx, gy

    def albedo(self, x, y):
        v = torch.zeros_like(x)
        for o, wgt in enumerate((0.35, 0.25, 0.25, 0.15)):
            s = self.cell * (1.0, 3.0, 9.0, 40.0)[o]
            a, b = x / s, y / s
            i, j = torch.floor(a), torch.floor(b)
            u, w = a - i, b - j
            u, w = u * u * (3 - 2 * u), w * w * (3 - 2 * w)
            i, j = i.long(), j.long()
            t = self.grid[o]
            at = lambda p, q: t[q & 255, p & 255]  # noqa: E731
            top = at(i, j) + u * (at(i + 1, j) - at(i, j))
            bot = at(i, j + 1) + u * (at(i + 1, j + 1) - at(i, j + 1))
            v += wgt * (top + w * (bot - top))
        return v

    def view(self, cam):
        """(image f32, depth, camera-frame normal) of one camera, on the GPU."""
        fx, fy, cx, cy = cam.k
        u = torch.arange(cam.width, device="cuda", dtype=torch.float32)
        v = torch.arange(cam.height, device="cuda", dtype=torch.float32)
        rx, ry = ((u - cx) / fx)[None, :], ((v - cy) / fy)[:, None]
        r = cam.r
        ctr = cam.center
        d = [float(r[0, k]) * rx + float(r[1, k]) * ry + float(r[2, k]) for k in range(3)]
        down = (-d[2]).clamp_min(1e-3)
        t = ctr[2] / down
        for _ in range(8):
            z, _, _ = self.height(ctr[0] + t * d[0], ctr[1] + t * d[1])
            t = (ctr[2] - z) / down
        x, y = ctr[0] + t * d[0], ctr[1] + t * d[1]
        _, gx, gy = self.height(x, y)
        n = [-gx, -gy, torch.ones_like(gx)]
        length = torch.sqrt(gx * gx + gy * gy + 1)
        nc = torch.stack([sum(float(r[a, k]) * n[k] for k in range(3)) / length for a in range(3)], -1)
        img = (0.15 + 0.7 * self.albedo(x, y)
               + 0.01 * torch.randn(x.shape, device="cuda", generator=self.gen)).clamp(0, 1)
        return img, t.expand_as(x).contiguous(), nc.contiguous()


def _cameras(case, seed):
    sizes = _sizes(case)
    base = scenes.formation(1920, 1080, (len(sizes) + 2) // 3, prefix="perf%d" % (seed & 0xFFFF))[: len(sizes)]
    cams = []
    for c, (w, h) in zip(base, sizes):
        f = (w / 2.0) / math.tan(math.radians(30.0))
        cams.append(scenes.Camera(c.name, (f, f, (w - 1) / 2.0, (h - 1) / 2.0), c.r, c.t, w, h))
    return cams


_RANGE = (20.0, 80.0)


def _scene(case, seed):
    cams = _cameras(case, seed)
    land = _Terrain(seed, 0.12 * 1920.0 / max(c.width for c in cams))
    images, depths, normals = [], [], []
    for c in cams:
        img, dep, nrm = land.view(c)
        images.append(img.cpu().numpy() if case["f32"] else (img * 255.0).round().to(torch.uint8).cpu().numpy())
        depths.append(dep)
        normals.append(nrm)
    src = scenes.nearest_sources(cams, case["sources"])
    return cams, images, depths, normals, src


def _perturbed(land_depth, normal, seed):
    """A map as a run leaves it: most pixels near the surface, some far off, some without depth."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    d = land_depth * (1 + 0.002 * torch.randn(land_depth.shape, device="cuda", generator=g))
    r = torch.rand(d.shape, device="cuda", generator=g)
    d = torch.where(r < 0.05, d * (0.6 + torch.rand(d.shape, device="cuda", generator=g)), d)
    d = torch.where(r > 0.98, torch.zeros_like(d), d)
    n = normal + 0.05 * torch.randn(normal.shape, device="cuda", generator=g)
    n = n / n.norm(dim=-1, keepdim=True)
    c = (0.1 + 0.3 * torch.rand(d.shape, device="cuda", generator=g)) + (r < 0.05) * 0.8
    s = ViewState.new(d.shape[1], d.shape[0])
    s.depth[...], s.normal[...], s.cost[...] = d.cpu().numpy(), n.cpu().numpy(), c.cpu().numpy()
    return s


class _State:
    """A backend with its open session, as a program keeps them."""

    def __init__(self, case):
        self.case = case
        self.be = PatchMatchBackend(0, tuning=case.get("tuning", 0)) if case["kind"] != "train" else None
        self.sess = self.net = None

    def close(self):
        for name in ("sess", "net", "be"):
            o = getattr(self, name, None)
            setattr(self, name, None)
            if o is not None:
                o.close()

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def _train_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    b, h, w = case["batch"], case["h"], case["w"]
    smooth = torch.rand(b, 3, max(2, h // 16), max(2, w // 16), device="cuda", generator=g)
    smooth = torch.nn.functional.interpolate(smooth, size=(h, w), mode="bilinear")
    t = 0.1 + 0.8 * smooth[:, 0]  # normalised inverse depth of the label
    x = torch.zeros(b, h, w, 48, device="cuda")
    x[..., 0] = smooth[:, 1]
    k = (torch.arange(32, device="cuda") + 0.5) / 32
    x[..., 1:33] = (1 - torch.exp(-200 * (t[..., None] - k) ** 2)
                    + 0.2 * torch.randn(b, h, w, 32, device="cuda", generator=g)).clamp(0, 2)
    lab = torch.zeros(b, h, w, 6, device="cuda")
    lab[..., 0] = t
    n = torch.stack([smooth[:, 1] - 0.5, smooth[:, 2] - 0.5, -torch.ones_like(t)], -1)
    lab[..., 1:4] = n / n.norm(dim=-1, keepdim=True)
    lab[..., 4] = (torch.rand(b, h, w, device="cuda", generator=g) < 0.9).float()
    lab[..., 5] = 1.0 / (1 / 60.0 + t * (1 / 25.0 - 1 / 60.0))
    lab *= lab[..., 4:5]
    return x.to(torch.bfloat16), lab.contiguous()


def _params():
    return np.load(proposal.DEFAULT_WEIGHTS)["params"].astype(np.float32)


def prepare(case, seed):
    s = _State(case)
    kind = case["kind"]
    if kind == "train":
        s.x, s.labels = _train_inputs(case, seed)
        s.net = proposal.ProposalNet(0, weights=proposal.DEFAULT_WEIGHTS)
        torch.cuda.synchronize()
        return s
    cams, images, depths, normals, src = _scene(case, seed)
    s.views = list(range(case["views"]))
    if kind in ("multiscale", "calls"):
        pm = _lib.default_pm()
        pm.window_radius, pm.window_step = case["radius"], case["step"]
        s.inp = densify.kernel_input(cams, images, src, [_RANGE] * len(cams), pm=pm, seed=seed & 0xFFFFFFFF,
                                     max_levels=3 if kind == "multiscale" else 2)
    else:
        s.inp = scenes.kernel_input(cams, images, src, _RANGE, window_radius=case["radius"], window_step=case["step"],
                                    seed=seed & 0xFFFFFFFF, gray8=not case["f32"])
    if kind == "host":
        return s
    s.sess = s.be.begin(s.inp)
    if kind == "run":
        s.states = [ViewState.new(cams[v].width, cams[v].height) for v in s.views]
    elif kind == "calls":
        s.states = [_perturbed(depths[v], normals[v], seed + v) for v in s.views]
        s.low = []
        for v in s.views:
            li = s.inp.views[v].levels[0]
            d = depths[v][::2, ::2][: li.height, : li.width]
            n = normals[v][::2, ::2][: li.height, : li.width]
            s.low.append(_perturbed(d.contiguous(), n.contiguous(), seed + 50 + v))
        s.passes = 0
    elif kind == "learned":
        s.net = proposal.ProposalNet(0, weights=proposal.DEFAULT_WEIGHTS)
    elif kind == "fuse":
        s.cams = fusion.FusionCams(cams, src)
        s.sess.upload(0, s.views, [_perturbed(depths[v], normals[v], seed + v) for v in s.views])
        s.sess.snapshot_capture(0, s.views, 1)
        s.sess.filter_resident(s.views, download=False)
        s.sess.synchronize()
        cap = sum(cams[v].width * cams[v].height for v in s.views) // 2  # a point takes at least two pixels
        s.cloud = {"positions": np.zeros((cap, 3), np.float32), "normals": np.zeros((cap, 3), np.float32),
                   "colors": np.zeros((cap, 3), np.uint8), "vis_counts": np.zeros(cap, np.uint8)}
        s.kept = 0
    return s


# ---------------------------------------------------------------------------------------------------- one pass
def _maps(states):
    return [{"depth": x.depth, "normal": x.normal, "cost": x.cost} for x in states]


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "run":
        s.sess.run(s.views, s.states, RunParams(0, False, True, case["iters"], 1))
        return _maps(s.states)
    if kind == "schedule":
        s.sess.schedule_resident(s.views, case["iters"], case["rounds"], case["geo"])
        return _maps(s.sess.readout_download(0, s.views))
    if kind == "multiscale":
        sch = densify.Schedule(photometric_iters=case["iters"], geometric_rounds=case["rounds"],
                               geometric_iters=case["geo"])
        return _maps(densify.compute_depth_maps_resident(s.sess, s.inp, s.views, sch))
    if kind == "host":
        with s.be.begin(s.inp) as sess:
            raw, kept, counts = densify.schedule_host(sess, s.inp, s.views, case["iters"], case["rounds"], case["geo"])
        return {"raw": _maps(raw), "kept": [x.depth for x in kept], "counts": counts}
    if kind == "learned":
        n = s.sess.propose(s.net, 0, s.views)
        s.sess.schedule_resident(s.views, case["iters"], case["rounds"], case["geo"], proposal=True)
        return {"proposed": n, "maps": _maps(s.sess.readout_download(0, s.views))}
    if kind == "train":
        loss, grads = s.net.train_step(s.x, s.labels, (25.0, 60.0), 0.0, grads=True)
        return {"loss": np.float32(loss), "grads": grads}
    if kind == "fuse":
        s.sess.readout_resident(s.views, download=False)
        removed = s.sess.postprocess_resident(0, s.views)
        n = s.sess.fuse_resident(0, s.views, s.cams)
        c = s.sess.fused_points()
        for k, part in s.cloud.items():  # into the program's own arrays; what the last pass left behind the end goes
            part[:n] = getattr(c, k)[: len(part)]
            part[n:s.kept] = 0
        s.kept = n
        return {"removed": removed, "points": n, **s.cloud}
    top = s.inp.num_levels - 1  # calls
    cost = s.sess.evaluate(top, s.views, s.states)
    up = s.sess.upsample(s.inp, top, s.views, s.low, 1.0, 0.04) if top else []
    med = s.sess.median_filter(s.inp, top, s.views, s.states)
    s.passes += 1  # every call brings its own snapshot
    maps = [None] * len(s.inp.views)
    for v, x in zip(s.views, s.states):
        maps[v] = x.depth
    counts = s.sess.filter(s.views, s.states, DepthSnapshot(s.passes, top, maps))
    return {"cost": cost, "counts": counts, "up": [{"depth": x.depth, "normal": x.normal} for x in up],
            "median": [{"depth": x.depth, "normal": x.normal} for x in med]}


# ---------------------------------------------------------------------------------------------------- 64 bits
def _exact_costs(inp, views, states, level):
    """Mean of the smallest top_k costs 1 - rho over the sources, for the given planes."""
    dev, dt = "cuda", torch.float64
    pm = inp.pm
    sig = pm.sigma_spatial if pm.sigma_spatial > 0 else float(pm.window_radius)
    offs = list(range(-pm.window_radius, pm.window_radius + 1, pm.window_step))
    images = [torch.from_numpy(np.asarray(v.levels[level].pixels)).to(dev).to(dt) / 255.0 for v in inp.views]

    def at(img, x, y):
        ok = (x >= 0) & (y >= 0) & (x < img.shape[1]) & (y < img.shape[0])
        return torch.where(ok, img[y.clamp(0, img.shape[0] - 1), x.clamp(0, img.shape[1] - 1)], 0.0)

    out = []
    for v, st in zip(views, states):
        kv, ref = inp.views[v], images[v]
        h, w = ref.shape
        fx, fy, cx, cy = (float(np.float32(k)) for k in kv.levels[level].k)
        yy, xx = torch.meshgrid(torch.arange(h, device=dev), torch.arange(w, device=dev), indexing="ij")
        d = torch.from_numpy(st.depth).to(dev).to(dt)
        n = torch.from_numpy(st.normal).to(dev).to(dt)
        ray = torch.stack([(xx - cx) / fx, (yy - cy) / fy, torch.ones_like(d)], -1)
        delta = d * (n * ray).sum(-1)
        taps = []
        wsum, msum, ssum = (torch.zeros_like(d) for _ in range(3))
        for dy in offs:
            for dx in offs:
                ik = at(ref, xx + dx, yy + dy)
                wt = torch.exp(-(dx * dx + dy * dy) / (2 * sig * sig) - (ref - ik) ** 2 / (2 * pm.sigma_color ** 2))
                taps.append((dx, dy, ik, wt))
                wsum, msum, ssum = wsum + wt, msum + wt * ik, ssum + wt * ik * ik
        mu = msum / wsum
        var = ssum / wsum - mu * mu
        costs = []
        for j, p in zip(kv.sources, np.asarray(kv.pairs_f64)):
            img = images[j]
            sfx, sfy, scx, scy = (float(np.float32(k)) for k in inp.views[j].levels[level].k)
            r, t = p[:9].reshape(3, 3), p[9:12]

            def project(x, y):
                q = torch.stack([(x - cx) / fx, (y - cy) / fy, torch.ones_like(d)], -1)
                s = (n * q).sum(-1) / delta  # X = q / s on the plane n X = delta
                z = [r[k, 0] * q[..., 0] + r[k, 1] * q[..., 1] + r[k, 2] * q[..., 2] + t[k] * s for k in range(3)]
                return (sfx * z[0] + scx * z[2]) / z[2], (sfy * z[1] + scy * z[2]) / z[2], z[2]

            u, vv, z = project(xx.to(dt), yy.to(dt))
            ok = (delta < -1e-12) & (z > 1e-8) & (u >= 0) & (vv >= 0) & (u <= img.shape[1] - 1) & \
                (vv <= img.shape[0] - 1) & (var >= 1e-5)
            ss, s2, sr = (torch.zeros_like(d) for _ in range(3))
            for dx, dy, ik, wt in taps:
                u, vv, z = project(xx + float(dx), yy + float(dy))
                u, vv = torch.nan_to_num(u).clamp(-4, 1e6), torch.nan_to_num(vv).clamp(-4, 1e6)
                x0, y0 = torch.floor(u), torch.floor(vv)
                a, b = u - x0, vv - y0
                x0, y0 = x0.long(), y0.long()
                sv = (at(img, x0, y0) * (1 - a) + at(img, x0 + 1, y0) * a) * (1 - b) + \
                    (at(img, x0, y0 + 1) * (1 - a) + at(img, x0 + 1, y0 + 1) * a) * b
                sv = torch.where(z > 1e-8, sv, 0.0)
                ss, s2, sr = ss + wt * sv, s2 + wt * sv * sv, sr + wt * sv * ik
            mus = ss / wsum
            vs = s2 / wsum - mus * mus
            rho = (sr / wsum - mu * mus) / torch.sqrt((var * vs).clamp_min(1e-30))
            costs.append(torch.where(ok & (vs >= 1e-5), (1 - rho).clamp(0, 2), 2.0))
        k = min(pm.top_k, len(costs))
        c = torch.stack(costs).sort(0).values[:k].mean(0)
        out.append(torch.where(d > 0, c, 2.0))
    return out


def _exact_train(x, lab):
    """Loss and parameter gradients of the proposal network in binary64."""
    flat = torch.from_numpy(_params()).to("cuda").double().requires_grad_(True)
    o, layers = 0, []
    for ci, co in proposal.LAYERS:
        wt = flat[o:o + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        o += co * 9 * ci
        layers.append((wt, flat[o:o + co]))
        o += co
    F = torch.nn.functional
    a = x.double().permute(0, 3, 1, 2)

    def conv(i, v, relu=True):
        wt, b = layers[i]
        vp = F.pad(v, (1, 1, 1, 1))
        h, w = v.shape[2:]
        y = b[None, :, None, None] + sum(torch.einsum("oc,bchw->bohw", wt[:, :, k // 3, k % 3],
                                                      vp[:, :, k // 3:k // 3 + h, k % 3:k % 3 + w]) for k in range(9))
        return torch.relu(y) if relu else y

    def up(v):
        return v.repeat_interleave(2, 2).repeat_interleave(2, 3)

    s0 = conv(1, conv(0, a))
    s1 = conv(3, conv(2, F.avg_pool2d(s0, 2)))
    s2 = conv(5, conv(4, F.avg_pool2d(s1, 2)))
    b3 = conv(7, conv(6, F.avg_pool2d(s2, 2)))
    d2 = conv(8, torch.cat([up(b3), s2], 1))
    d1 = conv(9, torch.cat([up(d2), s1], 1))
    d0 = conv(10, torch.cat([up(d1), s0], 1))
    out = conv(11, d0, False).permute(0, 2, 3, 1)
    lab = lab.double()
    valid = lab[..., 4] > 0.5
    t = torch.sigmoid(out[..., 0])
    nv = out[..., 1:4]
    cosine = (nv * lab[..., 1:4]).sum(-1) / (nv.norm(dim=-1) + 1e-6)
    depth = 1.0 / (1 / 60.0 + t * (1 / 25.0 - 1 / 60.0))
    target = ((depth - lab[..., 5]).abs() < 0.01 * lab[..., 5]).double().detach()
    cf = torch.sigmoid(out[..., 4])
    bce = -(target * torch.log(cf.clamp_min(1e-7)) + (1 - target) * torch.log((1 - cf).clamp_min(1e-7)))
    loss = ((t - lab[..., 0]).abs() + 1 - cosine + 0.5 * bce)[valid].sum() / valid.sum()
    loss.backward()
    return loss.detach(), flat.grad


def exact(case, seed):
    """Costs of the evaluate call, and the training batch's loss and gradients.  The other results are the outcome of
    comparisons between random draws (or whole numbers): they have no value that 64 bits would give."""
    if case["kind"] == "train":
        x, lab = _train_inputs(case, seed)
        loss, grads = _exact_train(x, lab)
        return {"loss": loss.cpu().numpy(), "grads": grads.cpu().numpy()}
    if case["kind"] == "calls":
        s = prepare(case, seed)
        costs = _exact_costs(s.inp, s.views, s.states, s.inp.num_levels - 1)
        s.close()
        return {"cost": [c.cpu().numpy() for c in costs]}
    return None
