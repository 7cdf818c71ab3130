"""The calls that a user of the depth-map engine makes, as performance cases.

Each case names a path (a public entry point) and its sizes; ``prepare`` makes a seeded survey
view or flight of that size on the GPU, ``run`` makes one call, ``exact`` gives the plane sweeps'
results in float64. The surveys are nadir flights 80 m above hilly terrain with flat-roofed
buildings, 80 % / 70 % overlap (75 % both ways for whole flights), uint8 images with 4-octave
texture - the geometry and value distributions of the repository's benchmark configurations.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

from py_ortho_b200 import _lib as L
from py_ortho_b200 import batch, dense, densify, fast, height, views

ALTITUDE = 80.0
NEAR, FAR = 60.0, 90.0
PRECISION = {"fp32": L.PREC_FP32, "fp16": L.PREC_FP16, "fp64sums": L.PREC_FP64_SUMS}


def listed():
    return [
        # a thumbnail or preview view with masked borders: latency and launches count
        dict(name="depth_map 320x240", path="depth_map", width=320, height=240, sources=4, window=5, distorted=True,
             masked=True, sums="fp32"),
        # the default settings of a flight: 1600 px, 4 neighbours, 11 x 11 window, calibrated lens
        dict(name="depth_map 1600x1200", path="depth_map", width=1600, height=1200, sources=4, window=5,
             distorted=True, masked=False, sums="fp32"),
        # full resolution, 8 neighbours, 7 x 7 (the benchmark's depth-map mode)
        dict(name="depth_map 4000x3000", path="depth_map", width=4000, height=3000, sources=8, window=3,
             distorted=False, masked=False, sums="fp32"),
        # the small plane sweep configuration
        dict(name="sweep 640x480 4src 128", path="sweep", width=640, height=480, sources=4, planes=128, window=2,
             top_k=2, sums="fp32"),
        # odd size, the reference's default window, window sums in the reference's float64
        dict(name="sweep 1003x749 5src 96 f64", path="sweep", width=1003, height=749, sources=5, planes=96, window=5,
             top_k=2, sums="fp64sums"),
        # the benchmark's sweep
        dict(name="sweep 4000x3000 8src 256", path="sweep", width=4000, height=3000, sources=8, planes=256, window=3,
             top_k=2, sums="fp32"),
        # uneven views (crops of a flight, 4-12 sources, 5 x 5 / 7 x 7) in one batched plan, FP16 images
        dict(name="batch 8 uneven views", path="batch", jobs=8, long_min=1200, long_max=2400, planes_max=192, mix=1,
             sums="fp16"),
        # pass 2 of one view with the default options: consistency, then the float64 repair of the
        # pixels it selects, calibrated lens
        dict(name="repair 1600x1200", path="repair", width=1600, height=1200, sources=4, window=4, step=2, iters=2,
             distorted=True),
        # the benchmark's float32 PatchMatch: every pixel, 7 x 7, 4 iterations
        dict(name="patchmatch 4000x3000 f32", path="patchmatch", width=4000, height=3000, sources=8, window=3, step=1,
             iters=4, precision="fp32"),
        # passes 1 and 2 of a small flight, the whole call
        dict(name="densify 5 views 800x600", path="densify", width=800, height=600, views=5, window=5),
        # point fusion of a flight
        dict(name="fuse 16 views 2000x1500", path="fuse", width=2000, height=1500, views=16, neighbours=4, stride=2),
        # the ground-grid height sweep of a flight
        dict(name="height 9 views 1000x750", path="height", width=1000, height=750, views=9, cell=2.0),
    ]


def _log_size(rng, lo, hi):
    """A 4:3 image with a long side log-uniform in [lo, hi], odd sizes as likely as even ones."""
    w = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return w, max(1, 3 * w // 4 + rng.randrange(-3, 4))


def draw(rng):
    path = rng.choice(["depth_map", "depth_map", "sweep", "sweep", "batch", "repair", "patchmatch", "densify", "fuse",
                       "height"])
    if path == "depth_map":
        w, h = _log_size(rng, 320, 4000)
        return dict(path=path, width=w, height=h, sources=rng.choice([2, 3, 4, 4, 4, 6, 8]), window=rng.choice([3, 5, 5, 7]),
                    distorted=rng.random() < 0.6, masked=rng.random() < 0.3,
                    sums=rng.choice(["fp32", "fp32", "fp64sums"]))
    if path == "sweep":
        w, h = _log_size(rng, 320, 3000)
        return dict(path=path, width=w, height=h, sources=rng.choice([2, 4, 5, 8, 12]),
                    planes=rng.choice([33, 64, 96, 128, 200, 256]), window=rng.choice([1, 2, 3, 3, 4, 5]),
                    top_k=rng.choice([1, 2, 2, 3]), sums=rng.choice(["fp32", "fp32", "fp16", "fp64sums"]))
    if path == "batch":
        return dict(path=path, jobs=rng.randrange(2, 9), long_min=400, long_max=rng.randrange(800, 2401),
                    planes_max=rng.randrange(96, 193), mix=rng.randrange(1000), sums=rng.choice(["fp32", "fp16"]))
    if path == "repair":
        w, h = _log_size(rng, 320, 1600)
        return dict(path=path, width=w, height=h, sources=rng.choice([2, 4, 4, 5, 8]), window=rng.choice([3, 4, 4, 5]),
                    step=rng.choice([1, 2, 2]), iters=rng.choice([1, 2, 2, 3]), distorted=rng.random() < 0.6)
    if path == "patchmatch":
        w, h = _log_size(rng, 320, 3000)
        return dict(path=path, width=w, height=h, sources=rng.choice([3, 4, 5, 8]), window=rng.choice([2, 3, 3, 4]),
                    step=rng.choice([1, 1, 2]), iters=rng.choice([1, 2, 4]), precision="fp32")
    if path == "densify":
        w, h = _log_size(rng, 240, 800)
        return dict(path=path, width=w, height=h, views=rng.randrange(3, 6), window=rng.choice([3, 5]))
    if path == "fuse":
        w, h = _log_size(rng, 320, 2000)
        return dict(path=path, width=w, height=h, views=rng.choice([4, 9, 16]), neighbours=rng.choice([2, 4, 6]),
                    stride=rng.choice([1, 2, 2, 3]))
    w, h = _log_size(rng, 300, 1000)
    return dict(path=path, width=w, height=h, views=rng.choice([4, 9]), cell=rng.choice([2.0, 2.5, 3.0]))


# ------------------------------------------------------------------ seeded surveys
def _attitude(rng, sigma_deg):
    w = rng.normal(0.0, math.radians(sigma_deg), 3)
    th = float(np.linalg.norm(w))
    k = w / th
    K = np.array([[0, -k[2], k[1]], [k[2], 0, -k[0]], [-k[1], k[0], 0]])
    return (np.eye(3) + math.sin(th) * K + (1 - math.cos(th)) * K @ K) @ np.diag([1.0, -1.0, -1.0])


class _Survey:
    """Terrain height and ground texture as rasters around the origin, and cameras over them.
    ``land`` seeds the terrain, the attitudes and the tie points where they are not ``seed``'s."""

    def __init__(self, seed, half, gsd, land=None):
        self.dev = L.require_cuda()
        self.rng = np.random.default_rng(seed if land is None else land)
        self.gen = torch.Generator(device=self.dev)
        self.gen.manual_seed(seed)
        self.half, self.gsd = half, gsd
        rng, n = self.rng, 20
        cell = max(0.125, gsd)
        m = int(2 * half / cell) + 1
        ax = torch.linspace(-half, half, m, device=self.dev)
        z = torch.zeros((m, m), device=self.dev)
        for x0, y0, s, a in zip(rng.uniform(-half, half, n), rng.uniform(-half, half, n), rng.uniform(5, 20, n),
                                rng.uniform(0, 6, n)):
            z += a * torch.exp(-(ax[:, None] - y0) ** 2 / (2 * s * s)) * torch.exp(-(ax[None] - x0) ** 2 / (2 * s * s))
        for x0, y0, sx, sy, top in zip(rng.uniform(-half, half, n), rng.uniform(-half, half, n), rng.uniform(3, 10, n),
                                       rng.uniform(3, 10, n), rng.uniform(3, 12, n)):
            inside = ((ax[:, None] - y0).abs() <= sy / 2) & ((ax[None] - x0).abs() <= sx / 2)
            z = torch.where(inside, torch.clamp(z, min=top), z)
        self.z = z
        t = int(2 * half / gsd) + 1
        tex = torch.zeros((1, 1, t, t), device=self.dev)
        amp = 1.0
        for period in (24, 12, 6, 3):
            g = torch.rand((1, 1, t // period + 2, t // period + 2), generator=self.gen, device=self.dev) - 0.5
            tex += amp * torch.nn.functional.interpolate(g, size=(t, t), mode="bilinear", align_corners=True)
            amp *= 0.6
        self.tex = tex[0, 0] / 2.176

    def _at(self, raster, x, y):
        g = torch.stack([x / self.half, y / self.half], -1)[None]
        return torch.nn.functional.grid_sample(raster[None, None], g, mode="bilinear", padding_mode="border",
                                               align_corners=True)[0, 0]

    def camera(self, x, y, f, w, h, k=(0.0, 0.0, 0.0)):
        return densify._Cam(_attitude(self.rng, 0.3), np.array([x, y, ALTITUDE]), f, k[0], k[1], (w - 1) / 2.0,
                            (h - 1) / 2.0, w, h, k[2])

    def render(self, cam):
        """(uint8 image, float32 camera-axis depth) on the device."""
        f64 = torch.float64
        nx = ((torch.arange(cam.w, device=self.dev, dtype=f64) - cam.cx) / cam.f)[None].expand(cam.h, -1)
        ny = ((torch.arange(cam.h, device=self.dev, dtype=f64) - cam.cy) / cam.f)[:, None].expand(-1, cam.w)
        x, y = nx, ny
        if cam.k1 or cam.k2 or cam.k3:
            for _ in range(8):
                r2 = x * x + y * y
                d = 1 + r2 * (cam.k1 + r2 * (cam.k2 + r2 * cam.k3))
                x, y = nx / d, ny / d
        R = torch.as_tensor(cam.R, device=self.dev)
        ray = [(R[0, i] * x + R[1, i] * y + R[2, i]).float() for i in range(3)]
        cx, cy, cz = (float(v) for v in cam.C)
        t = (cz - 3.0) / -ray[2]
        for _ in range(8):
            z = self._at(self.z, cx + t * ray[0], cy + t * ray[1])
            t = 0.5 * t + 0.5 * (cz - z) / -ray[2]
        gx, gy = cx + t * ray[0], cy + t * ray[1]
        g = self._at(self.tex, gx + 0.37 * z, gy - 0.61 * z)
        return torch.clamp(torch.round(128.0 + 300.0 * g), 0, 255).to(torch.uint8), t

    def tie_points(self, cams, n, hx, hy):
        """rec-like record of n terrain points with their in-image observations."""
        xs, ys = self.rng.uniform(-hx, hx, n), self.rng.uniform(-hy, hy, n)
        xt, yt = (torch.as_tensor(v, device=self.dev, dtype=torch.float32)[None] for v in (xs, ys))
        X = np.column_stack([xs, ys, self._at(self.z, xt, yt)[0].double().cpu().numpy()])
        obs_cam, obs_pt = [], []
        for k, c in enumerate(cams):
            xc = (X - c.C) @ c.R.T
            u, v = c.project_cam(xc[:, 0], xc[:, 1], xc[:, 2])
            ok = np.flatnonzero((xc[:, 2] > 0) & (u >= 0) & (v >= 0) & (u < c.w) & (v < c.h))
            obs_cam.append(np.full(len(ok), k, np.int32))
            obs_pt.append(ok.astype(np.int32))
        c = cams[0]
        intr = [SimpleNamespace(f=c.f, cx=c.cx, cy=c.cy, width=c.w, height=c.h, k1=c.k1, k2=c.k2, k3=c.k3)]
        return SimpleNamespace(used=list(range(len(cams))), intr=intr, cam_group=np.zeros(len(cams), np.int32), X=X,
                               C=np.array([c.C for c in cams]), R=np.array([c.R for c in cams]),
                               obs_cam=np.concatenate(obs_cam), obs_pt=np.concatenate(obs_pt), rms_px=0.5)


def _grey(u8):
    return (u8.float() - 128.0) / 64.0


def _star(case, seed, w, h, n_src):
    """A reference view at the origin and its n_src nearest flight neighbours (80 % / 70 %)."""
    f = 0.9 * w
    gx, gy = w * ALTITUDE / f, h * ALTITUDE / f
    pos = sorted(((i * 0.2 * gx, j * 0.3 * gy) for i in range(-3, 4) for j in range(-2, 3)),
                 key=lambda p: (round(math.hypot(*p), 6), p))[:n_src + 1]
    half = 0.5 * max(gx, gy) + max(max(abs(a), abs(b)) for a, b in pos) + 12.0
    s = _Survey(seed, half, ALTITUDE / f)
    k = (-0.03, 0.01, -0.002) if case.get("distorted") else (0.0, 0.0, 0.0)
    cams = [s.camera(x, y, f, w, h, k) for x, y in pos]
    return s, cams, gx, gy


def _flight(seed, w, h, n_views, land=None):
    """A grid flight with 75 % overlap both ways, as near square as n_views allows."""
    f = 0.9 * w
    gx, gy = w * ALTITUDE / f, h * ALTITUDE / f
    cols = int(math.ceil(math.sqrt(n_views)))
    pos = [((k % cols - 0.5 * (cols - 1)) * 0.25 * gx, (k // cols - 0.5 * (cols - 1)) * 0.25 * gy)
           for k in range(n_views)]
    s = _Survey(seed, 0.5 * max(gx, gy) * (1 + 0.25 * (cols - 1)) + 12.0, ALTITUDE / f, land)
    return s, [s.camera(x, y, f, w, h) for x, y in pos], gx * (1 + 0.25 * (cols - 1)), gy * (1 + 0.25 * (cols - 1))


def _planes(n):
    lo, hi = 1.0 / FAR, 1.0 / NEAR
    return np.array([lo + i * (hi - lo) / (n - 1) for i in range(n)], np.float32)


def _mask(grey, s):
    """NaN strips along two borders and a NaN block (a lens vignette, a masked object)."""
    h, w = grey.shape
    grey = grey.clone()
    grey[:max(2, h // 40)] = float("nan")
    grey[:, w - max(2, w // 50):] = float("nan")
    y, x = int(s.rng.integers(0, h - h // 8)), int(s.rng.integers(0, w - w // 8))
    grey[y:y + h // 8, x:x + w // 10] = float("nan")
    return grey


def _pass1_maps(s, depth, frac):
    """A pass-1 depth map and score: the true depth with noise, wrong patches and holes."""
    h, w = depth.shape
    g = torch.rand((1, 1, max(2, h // 24), max(2, w // 24)), generator=s.gen, device=s.dev)
    blob = torch.nn.functional.interpolate(g, size=(h, w), mode="bilinear", align_corners=True)[0, 0] < frac
    noise = torch.randn((h, w), generator=s.gen, device=s.dev)
    d = depth * (1 + torch.where(blob, 0.03, 0.0008) * noise)
    d[torch.rand((h, w), generator=s.gen, device=s.dev) < 0.02] = float("nan")
    score = torch.where(blob, 0.2 + 0.2 * noise, 0.8 + 0.05 * noise).clamp(-1, 1).half().float()
    return d.contiguous(), score.contiguous()


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["path"]](case, seed)


def _prepare_depth_map(case, seed):
    w, h, n = case["width"], case["height"], case["sources"]
    s, cams, gx, gy = _star(case, seed, w, h, n)
    greys = [_grey(s.render(c)[0]) for c in cams]
    if case["masked"]:
        greys = [_mask(g, s) for g in greys]
    rec = s.tie_points(cams, max(400, w * h // 600), 0.5 * gx, 0.5 * gy)
    greys = [g.cpu().numpy() for g in greys]
    opt = densify.DepthOptions(window=case["window"], precision=PRECISION[case["sums"]])
    return dict(path="depth_map", rec=rec, greys=greys, cams=cams, nbrs=list(range(1, n + 1)), opt=opt,
                views=lambda k: (greys[k], None, cams[k]))


def _prepare_sweep(case, seed):
    s, cams, _, _ = _star(case, seed, case["width"], case["height"], case["sources"])
    greys = [_grey(s.render(c)[0]).contiguous() for c in cams]
    opt = densify.DepthOptions(window=case["window"], top_k=case["top_k"], precision=PRECISION[case["sums"]])
    return dict(path="sweep", greys=greys, cams=cams, opt=opt, hyp=dense.Hypotheses.planes_inv(_planes(case["planes"])))


def _batch_mix(case):
    """The batch's shapes: they belong to the case, not to the seed."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["jobs"]):
        lw = int(round(math.exp(rng.uniform(math.log(case["long_min"]), math.log(case["long_max"])))))
        out.append((lw, 3 * lw // 4, int(rng.integers(4, 13)), int(rng.integers(96, case["planes_max"] + 1)),
                    int(rng.choice([2, 3])), float(rng.random()), float(rng.random())))
    return out


def _prepare_batch(case, seed):
    w, h = case["long_max"], 3 * case["long_max"] // 4
    s, cams, _, _ = _star(case, seed, w, h, 12)
    greys = [_grey(s.render(c)[0]).contiguous() for c in cams]
    f16 = case["sums"] == "fp16"
    imgs = [fast.to_fp16(g) for g in greys] if f16 else greys
    jobs = []
    for lw, lh, n, planes, r, ax, ay in _batch_mix(case):
        x0, y0 = int(ax * (w - lw)), int(ay * (h - lh))
        c = cams[0]
        crop = densify._Cam(c.R, c.C, c.f, 0.0, 0.0, c.cx - x0, c.cy - y0, lw, lh)
        jobs.append(batch.ViewJob(greys[0][y0:y0 + lh, x0:x0 + lw].contiguous(), imgs[1:n + 1], crop, cams[1:n + 1],
                                  _planes(planes), r=r, top_k=2))
    return dict(path="batch", jobs=jobs, plan=batch.Batch(jobs, precision=PRECISION[case["sums"]]))


def _prepare_repair(case, seed):
    w, h, n = case["width"], case["height"], case["sources"]
    s, cams, gx, gy = _star(case, seed, w, h, n)
    got = [s.render(c) for c in cams]
    maps = [_pass1_maps(s, d, 0.25) for _, d in got]
    rec = s.tie_points(cams, max(400, w * h // 600), 0.5 * gx, 0.5 * gy)
    greys = [_grey(g).cpu().numpy() for g, _ in got]
    opt = densify.DepthOptions(patchmatch=True, pm_window=case["window"], pm_step=case["step"], pm_iters=case["iters"])
    nbrs = [list(range(1, n + 1))] + [[0] for _ in range(n)]
    settings = views.PassSettings(rec, dict(enumerate(cams)), nbrs, opt)
    low = torch.rand((h, w), generator=s.gen, device=s.dev) < 0.01
    return dict(path="repair", rec=rec, raw={k: m[0] for k, m in enumerate(maps)}, score=maps[0][1], low=low,
                views=lambda k: (greys[k], None, cams[k]), nbrs=nbrs[0], settings=settings, opt=opt)


def _prepare_patchmatch(case, seed):
    w, h = case["width"], case["height"]
    s, cams, _, _ = _star(case, seed, w, h, case["sources"])
    got = [s.render(c) for c in cams]
    depth = (got[0][1] * (1 + 0.002 * torch.randn((h, w), generator=s.gen, device=s.dev))).contiguous()
    th = math.radians(30.0) * torch.sqrt(torch.rand((h, w), generator=s.gen, device=s.dev))
    ph = 2 * math.pi * torch.rand((h, w), generator=s.gen, device=s.dev)
    normal = torch.stack([torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th)]).contiguous()
    return dict(path="patchmatch", greys=[_grey(g).contiguous() for g, _ in got], cams=cams, depth=depth, normal=normal,
                score=torch.zeros((h, w), device=s.dev), active=torch.ones((h, w), dtype=torch.uint8, device=s.dev),
                ray=fast.rays_world((h, w), cams[0]), par=np.array([fast.cam_row(c) for c in cams[1:]]), case=case,
                seed=int(seed))


def _prepare_densify(case, seed):
    w, h, n = case["width"], case["height"], case["views"]
    s, cams, gx, gy = _star(case, seed, w, h, n - 1)
    greys = [_grey(s.render(c)[0]).cpu().numpy() for c in cams]
    rec = s.tie_points(cams, max(600, w * h // 300), 0.6 * gx, 0.6 * gy)
    opt = densify.DepthOptions(window=case["window"], patchmatch=True, neighbors=4)
    return dict(path="densify", rec=rec, views=lambda k: (greys[k], None, cams[k]), opt=opt)


def _prepare_fuse(case, seed):
    w, h, n = case["width"], case["height"], case["views"]
    s, cams, _, _ = _flight(seed, w, h, n)
    maps, rgbs = {}, {}
    for k, c in enumerate(cams):
        g, d = s.render(c)
        d = d * (1 + 0.002 * torch.randn((h, w), generator=s.gen, device=s.dev))
        d[torch.rand((h, w), generator=s.gen, device=s.dev) < 0.02] = float("nan")
        maps[k], rgbs[k] = d.contiguous(), g[..., None].repeat(1, 1, 3).contiguous()
    C = np.array([c.C for c in cams])
    nbrs = {k: [int(j) for j in np.argsort(np.linalg.norm(C - C[k], axis=1), kind="stable")[1:case["neighbours"] + 1]]
            for k in range(n)}
    return dict(path="fuse", maps=maps, rgbs=rgbs, cams=cams, nbrs=nbrs, tols={k: {j: 0.01 for j in nbrs[k]} for k in nbrs},
                stride=case["stride"])


def _prepare_height(case, seed):
    w, h, n = case["width"], case["height"], case["views"]
    s, cams, gx, gy = _flight(seed, w, h, n, land=1)      # the DSM's grid is the case's, not the seed's
    rgb = [s.render(c)[0].cpu().numpy()[..., None].repeat(3, axis=2) for c in cams]
    rec = s.tie_points(cams, 400 * n, 0.5 * gx, 0.5 * gy)
    frames = [SimpleNamespace(width=w, height=h, path=k) for k in range(n)]
    native = ALTITUDE / cams[0].f

    def load(frame, scale):
        q = int(round(1 / scale))
        return rgb[frame.path][::q, ::q] if q > 1 else rgb[frame.path]
    return dict(path="height", ar=SimpleNamespace(frames=frames, workers=1), rec=rec, native=native, load=load,
                opt=height.DenseOptions(gsd=case["cell"] * native))


# ------------------------------------------------------------------ run
def run(state):
    return globals()["_run_" + state["path"]](state)


def _run_depth_map(s):
    return densify.depth_map(0, s["nbrs"], s["rec"], s["views"], s["opt"])


def _run_sweep(s):
    return densify._sweep(s["greys"][0], s["cams"][0], s["greys"][1:], s["cams"][1:], s["hyp"], s["opt"])


def _run_batch(s):
    s["plan"].run()
    return [(j.depth, j.state[0], j.state[4]) for j in s["jobs"]]


def _run_repair(s):
    score = s["score"].clone()
    depth, changed, n_active = views.repair(0, s["raw"], score, s["low"], s["views"], s["nbrs"], s["rec"],
                                            s["settings"], s["opt"])
    return depth, score, changed, n_active


def _run_patchmatch(s):
    c = s["case"]
    depth, normal, score = s["depth"].clone(), s["normal"].clone(), s["score"].clone()
    changed = dense.pm_refine(s["greys"][0], s["ray"], s["cams"][0].C, s["greys"][1:], [None] * c["sources"], s["par"],
                              depth, normal, score, s["active"], c["window"], c["step"], 2, 0.0, 1.0, c["iters"], NEAR,
                              FAR, s["seed"], precision=c["precision"])
    return depth, normal, score, changed


def _run_densify(s):
    return views.densify_views(s["rec"], s["views"], s["opt"])


def _run_fuse(s):
    xyz, colours, count, owner, used = views.fuse(sorted(s["maps"]), s["maps"], s["cams"], s["nbrs"], s["tols"], 1.5, 2,
                                                  s["stride"], s["rgbs"])
    # the number of points varies with the inputs: filled up to the number of candidates, so that
    # results of different inputs have one shape
    st = s["stride"]
    rows = sum(-(-d.shape[0] // st) * -(-d.shape[1] // st) for d in s["maps"].values()) - xyz.shape[0]
    pad = torch.nn.functional.pad
    return pad(xyz, (0, 0, 0, rows)), pad(colours, (0, 0, 0, rows)), pad(count, (0, rows)), pad(owner, (0, rows)), used


def _run_height(s):
    r = height.dense_reconstruct(s["ar"], s["rec"], {}, s["native"], s["opt"], load_rgb=s["load"])
    return r.Z, r.score, r.rgb, r.covered


# ------------------------------------------------------------------ work
# Operations of one evaluation (pixel x hypothesis x source) of the sweep: the map and one bilinear
# sample, four separable running sums, the NCC; of one window sample of PatchMatch: the map, the
# bilinear sample and three sums.
SWEEP_OPS, SAMPLE_OPS = 50, 40


def work(case):
    p = case["path"]
    if p == "batch":
        mix = _batch_mix(case)
        px = case["long_max"] ** 2 * 3 // 4
        size = 2 if case["sums"] == "fp16" else 4
        return {"bytes": 12 * px * size + sum(w * h * (4 + 4 * 6) for w, h, *_ in mix),
                "flops": SWEEP_OPS * sum(w * h * n * m for w, h, n, m, *_ in mix)}
    px = case["width"] * case["height"]
    n = case.get("sources", 4)
    if p == "sweep":
        return {"bytes": px * 4 * (n + 1 + 3), "flops": SWEEP_OPS * px * n * case["planes"]}
    if p == "depth_map":      # at least 64 hypotheses at 1/4 resolution, 7 at 1/2 and at full resolution
        return {"bytes": px * (4 * (n + 1) + 9), "flops": SWEEP_OPS * px * n * (64 / 16 + 7 / 4 + 7)}
    if p in ("repair", "patchmatch"):
        side = 2 * case["window"] // case["step"] + 1
        share = 0.4 if p == "repair" else 1.0
        return {"bytes": px * 4 * (n + (n if p == "repair" else 0) + 1 + 10),
                "flops": SAMPLE_OPS * share * px * n * case["iters"] * 11 * side * side}
    if p == "densify":
        m = case["views"]
        nb = min(4, m - 1)
        return {"bytes": m * px * 4 * 2, "flops": m * px * nb * (SWEEP_OPS * (64 / 16 + 7 / 4 + 7) +
                                                                 0.3 * SAMPLE_OPS * 2 * 11 * 25)}
    if p == "fuse":
        m = case["views"]
        return {"bytes": m * px * (4 + 3 + 1), "flops": 150 * m * px / case["stride"] ** 2 * case["neighbours"]}
    m = case["views"]
    cells = 2.2 * px / case["cell"] ** 2      # the flight's footprint at the DSM's cell size
    return {"bytes": m * px * 3 + cells * 9, "flops": 60 * cells * 6 * (4 * 9 + 60 / 16)}


# ------------------------------------------------------------------ the sweeps in float64
def exact(case, seed):
    p = case["path"]
    if p == "sweep":
        s = _prepare_sweep(case, seed)
        img = [g.double() for g in s["greys"]]
        if case["sums"] == "fp16":
            img[1:] = [g.half().double() for g in s["greys"][1:]]
        planes = torch.as_tensor(s["hyp"].planes, device=img[0].device, dtype=torch.float64)
        depth, best, sd = _sweep64(img[0], s["cams"][0], img[1:], s["cams"][1:], len(planes), lambda i: planes[i],
                                   case["window"], case["top_k"], _rays64(img[0].shape, s["cams"][0], img[0].device))
        return depth, best, sd
    if p == "depth_map":
        s = _prepare_depth_map(case, seed)
        depth, score = _depth_map64(s, case)
        return depth, score, None
    return None


def _rays64(shape, cam, dev):
    h, w = shape
    nx = ((torch.arange(w, device=dev, dtype=torch.float64) - cam.cx) / cam.f)[None].expand(h, -1)
    ny = ((torch.arange(h, device=dev, dtype=torch.float64) - cam.cy) / cam.f)[:, None].expand(-1, w)
    x, y = nx, ny
    for _ in range(8):
        r2 = x * x + y * y
        d = 1 + r2 * (cam.k1 + r2 * (cam.k2 + r2 * cam.k3))
        x, y = nx / d, ny / d
    R = torch.as_tensor(cam.R, device=dev)
    return torch.stack([R[0, i] * x + R[1, i] * y + R[2, i] for i in range(3)])


def _mean(a, r):
    """(2r + 1)^2 window mean of stacked images, zeros outside."""
    k = 2 * r + 1
    a = torch.nn.functional.avg_pool2d(a[None], (1, k), 1, (0, r))
    return torch.nn.functional.avg_pool2d(a, (k, 1), 1, (r, 0))[0]


def _sweep64(ref, cam, srcs, cams, n, inv_at, r, top_k, ray):
    """densify._sweep with every quantity in float64: (depth, best, sd)."""
    h, w = ref.shape
    dev = ref.device
    mu, m2 = _mean(torch.stack([ref, ref * ref]), r)
    sd = torch.sqrt(torch.clamp(m2 - mu * mu, min=1e-6))
    geo = []
    for c in cams:
        R = torch.as_tensor(np.asarray(c.R, np.float64), device=dev)
        geo.append((torch.einsum("ij,jhw->ihw", R, ray), R @ torch.as_tensor(cam.C - c.C, device=dev)))
    full = lambda v: torch.full((h, w), v, dtype=torch.float64, device=dev)  # noqa: E731
    best, prev, before, after = full(-2.0), full(-2.0), full(-2.0), full(-2.0)
    idx = torch.full((h, w), -1, dtype=torch.int64, device=dev)
    for i in range(n):
        d = 1.0 / inv_at(i)
        scores = []
        for img, c, (mr, b) in zip(srcs, cams, geo):
            sh, sw = img.shape
            z = b[2] + d * mr[2]
            x, y = (b[0] + d * mr[0]) / z, (b[1] + d * mr[1]) / z
            r2 = x * x + y * y
            g = c.f * (1 + r2 * (c.k1 + r2 * (c.k2 + r2 * c.k3)))
            u, v = g * x + c.cx, g * y + c.cy
            ok = (z > 1e-6) & (u >= 0) & (v >= 0) & (u <= sw - 1.001) & (v <= sh - 1.001)
            u, v = torch.where(ok, u, 0.0), torch.where(ok, v, 0.0)
            x0, y0 = u.floor(), v.floor()
            fx, fy = u - x0, v - y0
            o = (y0 * sw + x0).long()
            flat = img.reshape(-1)
            val = (flat[o] * (1 - fx) + flat[o + 1] * fx) * (1 - fy) + (flat[o + sw] * (1 - fx) + flat[o + sw + 1] * fx) * fy
            ok = ok & torch.isfinite(val)
            val = torch.where(ok, val, 0.0)
            cov, mj, mjj, mji = _mean(torch.stack([ok.double(), val, val * val, val * ref]), r)
            good = cov > 0.9
            q = torch.where(good, cov, 1.0)
            mj, mjj, mji = mj / q, mjj / q, mji / q
            var = mjj - mj * mj
            sdj = torch.where(var > 1e-6, torch.sqrt(torch.clamp(var, min=1e-6)), 1e-3)
            scores.append(torch.where(good, torch.clamp((mji - mu * mj) / (sd * sdj), -1.0, 1.0), -1.0))
        k = min(top_k, len(scores))
        sc = torch.topk(torch.stack(scores), k, dim=0).values.mean(0)
        after = torch.where(idx == i - 1, sc, after) if i > 0 else after
        win = sc > best
        before = torch.where(win, prev, before)
        after = torch.where(win, -2.0, after)
        idx = torch.where(win, i, idx)
        best = torch.where(win, sc, best)
        prev = sc
    den = before - 2 * best + after
    mid = (idx > 0) & (idx < n - 1) & (den < -1e-6)
    off = torch.where(mid, torch.clamp(0.5 * (before - after) / torch.where(mid, den, -1.0), -0.5, 0.5), 0.0)
    inv0 = inv_at(0)
    step = (inv_at(1) - inv0) if n > 1 else 0.0
    return 1.0 / torch.clamp(inv0 + (idx + off) * step, min=1e-9), best, sd


def _half64(a):
    h, w = a.shape[-2] // 2 * 2, a.shape[-1] // 2 * 2
    a = a[..., :h, :w]
    return 0.25 * (a[..., ::2, ::2] + a[..., 1::2, ::2] + a[..., ::2, 1::2] + a[..., 1::2, 1::2])


def _depth_range64(rec, c):
    xc = (rec.X - c.C) @ c.R.T
    u, v = c.f * xc[:, 0] / xc[:, 2] + c.cx, c.f * xc[:, 1] / xc[:, 2] + c.cy
    z = xc[(xc[:, 2] > 0) & (u >= 0) & (v >= 0) & (u < c.w) & (v < c.h), 2]
    near, far = np.percentile(z, [1, 99])
    far = max(far, (c.C[2] - np.percentile(rec.X[:, 2], 0.5)) / max(-c.R[2, 2], 0.2))
    span = far - near
    return max(0.3 * near, near - 0.2 * span - 1.0), far + 0.2 * span + 2.0


def _band64(rec, c, shape, rng, block):
    """Per-pixel inverse-depth interval (far, near) of the view's own tie points."""
    h, w = shape
    lo, hi = rng
    pts = rec.X[rec.obs_pt[rec.obs_cam == 0]]
    gh, gw = -(-h // block), -(-w // block)
    zlo, zhi, cnt = np.full((gh + 2, gw + 2), np.inf), np.full((gh + 2, gw + 2), -np.inf), np.zeros((gh, gw), int)
    if len(pts) >= 50:
        xc = (pts - c.C) @ c.R.T
        u, v = c.project_cam(xc[:, 0], xc[:, 1], xc[:, 2])
        ok = (xc[:, 2] > 0) & (u >= 0) & (v >= 0) & (u < w) & (v < h)
        bx = (np.minimum(u[ok], w - 1) // block).astype(int)
        by = (np.minimum(v[ok], h - 1) // block).astype(int)
        np.minimum.at(zlo, (by + 1, bx + 1), xc[ok, 2])
        np.maximum.at(zhi, (by + 1, bx + 1), xc[ok, 2])
        np.add.at(cnt, (by, bx), 1)
    few = np.pad(cnt, 1) < 5
    zlo[few], zhi[few] = np.inf, -np.inf
    nine = [(slice(a, a + gh), slice(b, b + gw)) for a in range(3) for b in range(3)]
    lo3, hi3 = np.min([zlo[q] for q in nine], 0), np.max([zhi[q] for q in nine], 0)
    has = (cnt >= 5) & np.isfinite(lo3)
    pad = 1.0 + 0.05 * np.where(has, hi3 - lo3, 0.0)
    near = np.where(has, np.clip(np.where(has, lo3, 0.0) - pad, lo, hi), lo)
    far = np.where(has, np.clip(np.where(has, hi3, 0.0) + pad, lo, hi), hi)
    grow = lambda a: np.repeat(np.repeat(a, block, 0), block, 1)[:h, :w]  # noqa: E731
    return grow(1.0 / far), grow(1.0 / np.maximum(near, 1e-6))


def _up64(a, h, w):
    a = a.repeat_interleave(2, 0).repeat_interleave(2, 1)[:h, :w]
    return torch.nn.functional.pad(a[None, None], (0, w - a.shape[1], 0, h - a.shape[0]), mode="replicate")[0, 0]


def _depth_map64(s, case):
    dev = L.require_cuda()
    rec, cams, r = s["rec"], s["cams"], case["window"]
    img = [torch.as_tensor(g, device=dev).double() for g in s["greys"]]
    bad = ~torch.isfinite(img[0])
    img[0] = torch.where(bad, 0.0, img[0])
    pyr, pyr_c, ray = [img], [cams], [_rays64(img[0].shape, cams[0], dev)]
    for _ in range(2):
        small = [_half64(a) for a in pyr[-1]]
        pyr_c.append([c.scaled(0.5, a.shape[1], a.shape[0]) for c, a in zip(pyr_c[-1], small)])
        ray.append(_half64(ray[-1]))
        pyr.append(small)
    rng = _depth_range64(rec, cams[0])
    base = float(np.median([np.linalg.norm(rec.C[0] - rec.C[j]) for j in s["nbrs"]]))
    nd = int(min(max(math.ceil(pyr_c[2][0].f * base * (1 / rng[0] - 1 / rng[1])), 64), 192))
    h, w = pyr[2][0].shape
    far, near = (torch.as_tensor(a, device=dev) for a in _band64(rec, pyr_c[2][0], (h, w), rng, max(8, w // 16)))
    step = (near - far) / (nd - 1)
    depth, _, _ = _sweep64(pyr[2][0], pyr_c[2][0], pyr[2][1:], pyr_c[2][1:], nd, lambda i: far + i * step, r, 2, ray[2])
    step = step / 2
    for lv in (1, 0):
        h, w = pyr[lv][0].shape
        inv, step = 1.0 / _up64(depth, h, w), _up64(step, h, w)
        depth, score, _ = _sweep64(pyr[lv][0], pyr_c[lv][0], pyr[lv][1:], pyr_c[lv][1:], 7,
                                   lambda i: torch.clamp(inv + (i - 3) * step, min=1e-6), r, 2, ray[lv])
        step = step / 2
    return torch.where(bad | (depth < rng[0]) | (depth > rng[1]), float("nan"), depth), score
