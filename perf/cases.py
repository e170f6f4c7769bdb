"""The calls this library is measured by.

Each case is one call, or one short run of calls, that a host program makes
through the C-ABI or its Python mirror: training steps (the smallest, the
reference's one-view loop, batched, uneven resolutions, 4K), the
forward/backward op pair, renders, viewer frames, multi-view scores, the k-NN
initialisation and the device sort.  Large results go to pinned host buffers
that the program keeps, as a trainer or a viewer keeps its own.

A training step returns its losses and the first Adam moment of all 59 planes
(the running gradient); the parameters it leaves behind are the input of the
next pass on the same state.
"""
from __future__ import annotations

import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "skyfall-viewer_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

PLANES = 59
SH_C0 = 0.28209479177387814
BETA1 = 0.9  # SkyConfig.beta1's default

# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
# loss "l2l1": w_l2 = 1, w_l1 = 0.2; "default": the configuration's own
# 0.8 L1 + 0.2 SSIM.  scene "uniform": a box seen from outside; "clusters":
# 64 clusters on a scene seen from an orbit; "dense": 64 tight clusters, hundreds of
# splats per tile.  res "mixed": 640x480 / 1280x720 / 1920x1080 in turn.


def listed():
    train = dict(kind="train", sh=3, scene="clusters", loss="l2l1", cull=True, graph=True, tile=16, sh_every=1)
    return [
        # the smallest training step, one view, launched directly: latency
        dict(train, name="step_16k_256", n=16384, sh=0, scene="uniform", views=1, res="256x256", steps=1,
             cull=False, graph=False),
        # the reference's own loop at its default loss and schedule: one view
        # per step, every tile of each rectangle listed, SH updated every 16 steps
        dict(train, name="loop_1m_1080p_default", n=1_000_000, views=1, res="1920x1080", steps=16,
             loss="default", cull=False, graph=False, sh_every=16),
        # the batched, graph-captured trainer: the benchmark's workload
        dict(train, name="train_1m_16x1080p", n=1_000_000, views=16, res="1920x1080", steps=2),
        # batched training at uneven resolutions with the default loss
        dict(train, name="train_1m_16xmixed_default", n=1_000_000, views=16, res="mixed", steps=2, loss="default"),
        # memory stress: 4M Gaussians, one 4K view per step
        dict(train, name="train_4m_4k", n=4_000_000, scene="dense", views=1, res="3840x2160", steps=8),
        # the op pair of a host that owns its optimizer: gradients come back
        dict(kind="grads", name="grads_300k_4x720p", n=300_000, sh=3, scene="clusters", views=4, res="1280x720",
             loss="l2l1", cull=True, tile=16),
        # forward only, odd sizes on one small preview and eight full views
        dict(kind="render", name="render_20k_611x397", n=20_011, sh=1, scene="uniform", views=1, res="611x397",
             tile=16),
        dict(kind="render", name="render_1m_8x1080p", n=1_000_000, sh=3, scene="clusters", views=8,
             res="1920x1080", tile=16),
        # one interactive viewer frame of a trained scene
        dict(kind="frame", name="frame_1m_1080p", n=1_000_000, sh=3, scene="clusters", res="1920x1080", u8=False,
             scaling=1.0),
        # the multi-view scores behind every densify and prune (10 cameras)
        dict(kind="scores", name="scores_500k_10x720p", n=500_000, sh=3, scene="clusters", views=10,
             res="1280x720", loss="l2l1", tile=16),
        # scale initialisation of a point cloud
        dict(kind="knn", name="knn_500k", n=500_000, sh=0, scene="clusters"),
        # the device-pointer sort, as a caller with its own buffers uses it
        dict(kind="sort", name="sort_16m_32bit", n=16_777_216, bits=32),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "grads", "render", "frame", "scores", "knn", "sort"])
    if kind == "sort":
        return dict(kind="sort", n=_log_uniform(rng, 2000, 40_000_000), bits=rng.choice([8, 13, 16, 24, 32]))
    scene = rng.choice(["uniform", "clusters", "clusters", "dense"])
    if kind == "knn":
        return dict(kind="knn", n=_log_uniform(rng, 2000, 1_000_000), sh=0, scene=rng.choice(["uniform", "clusters"]))
    sh = rng.choice([0, 1, 2, 3, 3, 3])
    w = _log_uniform(rng, 120, 1920)
    h = max(90, min(1080, int(w * rng.uniform(0.5, 0.8))))
    res = f"{w}x{h}"
    if kind == "frame":
        return dict(kind="frame", n=_log_uniform(rng, 4000, 1_500_000), sh=sh, scene=scene, res=res,
                    u8=rng.random() < 0.4, scaling=rng.choice([0.5, 1.0, 1.0]))
    if kind == "render":
        return dict(kind="render", n=_log_uniform(rng, 4000, 1_000_000), sh=sh, scene=scene,
                    views=rng.randint(1, 8), res=res, tile=16)
    if kind == "scores":
        return dict(kind="scores", n=_log_uniform(rng, 10_000, 600_000), sh=sh, scene="clusters",
                    views=rng.randint(2, 10), res=res, loss="l2l1", tile=16)
    loss = rng.choice(["l2l1", "default"])
    if kind == "grads":
        return dict(kind="grads", n=_log_uniform(rng, 4000, 500_000), sh=sh, scene=scene, views=rng.randint(1, 6),
                    res=res, loss=loss, cull=rng.random() < 0.7, tile=rng.choice([16, 16, 16, 8]))
    views = rng.choice([1, 1, 2, 4, 7, 16])
    return dict(kind="train", n=_log_uniform(rng, 4000, 1_000_000), sh=sh, scene=scene, views=views,
                res="mixed" if views >= 4 and rng.random() < 0.3 else res, steps=rng.randint(1, 3), loss=loss,
                cull=rng.random() < 0.7, graph=rng.random() < 0.6, tile=rng.choice([16, 16, 16, 8]),
                sh_every=rng.choice([1, 1, 16]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed, stream):
    return torch.Generator("cuda").manual_seed((int(seed) * 1_000_003 + stream * 7919) & 0x7FFFFFFF)


def _scene(kind, n, sh, seed):
    """59 planes of n Gaussians, f32 on the GPU."""
    g = _gen(seed, 1)
    rand = lambda *s: torch.rand(*s, device="cuda", generator=g)  # noqa: E731
    randn = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    P = torch.zeros(PLANES, n, device="cuda")
    if kind == "uniform":
        P[0:3] = rand(3, n) * 2 - 1
        P[3:6] = -4.0 + 0.3 * randn(3, n)
        P[10] = randn(n)
    else:
        sigma, mean = (0.3, -4.5) if kind == "clusters" else (0.05, -5.0)
        centers = (rand(3, 64) * 2 - 1) * 2.0
        P[0:3] = centers[:, torch.randint(64, (n,), device="cuda", generator=g)] + sigma * randn(3, n)
        P[3:6] = mean + 0.5 * randn(3, n)
        P[10] = 1.5 * randn(n)
    q = randn(4, n)
    P[6:10] = q / q.norm(dim=0)
    P[11:14] = (rand(3, n) - 0.5) / SH_C0
    k = (sh + 1) ** 2
    if k > 1:
        P[14:11 + 3 * k] = 0.05 * randn(3 * k - 3, n)
    return P


def _sizes(case):
    if case["res"] == "mixed":
        return [((640, 480), (1280, 720), (1920, 1080))[v % 3] for v in range(case["views"])]
    w, h = (int(v) for v in case["res"].split("x"))
    return [(w, h)] * case.get("views", 1)


def _cameras(case, seed):
    """Pinhole cameras (60 degrees) around the scene looking at its middle:
    column-major f32 view and projection, focal, size."""
    phase = (seed * 0.6180339887498949) % 1.0
    sizes, out = _sizes(case), []
    for v, (w, h) in enumerate(sizes):
        a = 2 * math.pi * (v + phase) / len(sizes)
        r = 3.0 if case["scene"] == "uniform" else 5.0
        eye = np.array([r * math.cos(a), 0.16 * r, r * math.sin(a)])
        f = -eye / np.linalg.norm(eye)
        right = np.cross([0.0, 1.0, 0.0], f)
        right /= np.linalg.norm(right)
        R = np.stack([right, np.cross(f, right), f])
        V = np.eye(4)
        V[:3, :3], V[:3, 3] = R, -R @ eye
        focal = (h / 2.0) / math.tan(math.radians(30.0))
        M = np.zeros((4, 4))
        M[0, 0], M[1, 1], M[2, 2], M[3, 2] = 2 * focal / w, -2 * focal / h, 1.0, 1.0
        out.append(dict(view=V.T.reshape(-1).astype(np.float32), proj=M.T.reshape(-1).astype(np.float32),
                        focal=np.array([focal, focal], np.float32), width=w, height=h))
    return out


def _ground_truth(case, seed):
    """The scene the targets show: another one of the same kind, 3 in 10 as many Gaussians."""
    return _scene(case["scene"], max(1000, case["n"] * 3 // 10), case["sh"], seed + 500_009)


def _weights(case):
    return dict(w_l2=1.0, w_l1=0.2, w_ssim=0.0) if case["loss"] == "l2l1" else dict(w_l2=0.0, w_l1=0.8, w_ssim=0.2)


def _pinned(*shape, dtype=torch.float32):
    return torch.empty(*shape, dtype=dtype, pin_memory=True)


def prepare(case, seed):
    import skyfall
    kind = case["kind"]
    if kind == "sort":
        n, g = case["n"], _gen(seed, 3)
        keys = torch.randint(0, 1 << case["bits"], (n,), device="cuda", generator=g).to(torch.int32)
        vals = torch.randperm(n, device="cuda", generator=g).to(torch.int32)
        return dict(case=case, keys=keys, vals=vals, keys_out=torch.empty_like(keys), vals_out=torch.empty_like(vals))
    cfg = dict(sh_degree=case["sh"], sh_degree_interval=0, tile_size=case.get("tile", 16),
               tile_cull=int(case.get("cull", False)), use_graph=int(case.get("graph", False)),
               sh_update_interval=case.get("sh_every", 1), seed=seed)
    if "loss" in case:
        cfg.update(_weights(case))
    r = skyfall.GaussianRenderer(**cfg)
    r.load_points(_scene(case["scene"], case["n"], case["sh"], seed).cpu().numpy())
    s = dict(case=case, r=r)
    n = case["n"]
    if kind == "knn":
        s.update(density=_pinned(n), params=_pinned(PLANES, n))
        return s
    cams = _cameras(case, seed)
    px = sum(c["width"] * c["height"] for c in cams)
    if kind == "frame":
        s["cam"] = skyfall.renderer.to_sky_camera(cams[0])
        s["settings"] = skyfall._lib.SkyViewSettings(case["scaling"], case["sh"], 1, 0)
        s["image"] = _pinned(cams[0]["height"], cams[0]["width"], 4, dtype=torch.uint8 if case["u8"] else torch.float32)
        return s
    r.setTrainingCameras(cams)
    s["views"] = np.arange(len(cams), dtype=np.uint32)
    if kind == "render":
        s.update(rgba=_pinned(px, 4), alpha=_pinned(px))
        return s
    with skyfall.GaussianRenderer(sh_degree=case["sh"], sh_degree_interval=0) as gt:
        gt.load_points(_ground_truth(case, seed).cpu().numpy())
        gt.setTrainingCameras(cams)
        for v, c in enumerate(cams):
            r.setTrainingImage(v, gt.render([v], with_alpha=False)[0].reshape(c["height"], c["width"], 4))
    if kind in ("train", "grads"):
        s["grads"] = _pinned(PLANES, n)
    return s


# ---------------------------------------------------------------------------
# The measured call
# ---------------------------------------------------------------------------
def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(state):
    import skyfall
    L, check = skyfall.lib(), skyfall._lib.check
    case, kind = state["case"], state["case"]["kind"]
    if kind == "sort":
        check(L.sky_sort_pairs(_ptr(state["keys"]), _ptr(state["vals"]), _ptr(state["keys_out"]),
                               _ptr(state["vals_out"]), case["n"], case["bits"],
                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return dict(keys=state["keys_out"], vals=state["vals_out"])
    r, n = state["r"], case["n"]
    if kind == "knn":
        check(L.sky_knn_init(r._h, 0.0, _ptr(state["density"])))
        check(L.sky_get_params(r._h, _ptr(state["params"]), n))
        return dict(density=state["density"], params=state["params"])
    if kind == "frame":
        img = _ptr(state["image"])
        check(L.sky_view_render(r._h, ctypes.byref(state["cam"]), ctypes.byref(state["settings"]),
                                None if case["u8"] else img, img if case["u8"] else None))
        return state["image"]
    views = state["views"]
    if kind == "render":
        check(L.sky_render(r._h, skyfall._lib.ptr(views), len(views), _ptr(state["rgba"]), _ptr(state["alpha"])))
        return dict(rgba=state["rgba"], alpha=state["alpha"])
    if kind == "scores":
        hits, score = r.scoreViews(views)
        return dict(hits=hits, score=score)
    if kind == "grads":
        loss = r.forward(views)
        check(L.sky_backward(r._h, _ptr(state["grads"]), n))
        return dict(loss=loss, grads=state["grads"])
    losses = [r.trainStep(views).loss for _ in range(case["steps"])]
    check(L.sky_get_moments(r._h, _ptr(state["grads"]), None, n))
    return dict(loss=losses, moment=state["grads"])


# ---------------------------------------------------------------------------
# Work a pass cannot do without
# ---------------------------------------------------------------------------
def _pairs(case):
    """(pixel, splat) pairs a pass composites, roughly: splats whose alpha >=
    1/255 ellipse covers a pixel, at most what fills it (about 50)."""
    log_sigma = dict(uniform=-4.0, clusters=-4.5, dense=-5.0)[case["scene"]]
    dist = 3.0 if case["scene"] == "uniform" else 5.0
    total = 0.0
    for w, h in _sizes(case):
        sigma_px = (h / 2.0) / math.tan(math.radians(30.0)) * math.exp(log_sigma) / dist
        area = 2 * math.pi * 4.8 * (sigma_px ** 2 + 0.3)
        total += min(case["n"] * area, 50.0 * w * h)
    return total


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "sort":
        return dict(bytes=16 * n, flops=0)
    if kind == "knn":
        return dict(bytes=n * (12 + 4 + 2 * PLANES * 4), flops=n * 60 * 9)
    px = sum(w * h for w, h in _sizes(case))
    geo, coef = 11, 3 * (case["sh"] + 1) ** 2
    views = len(_sizes(case))
    scene = n * (geo + coef) * 4
    pairs = _pairs(case)
    project = n * views * 300
    if kind == "frame":
        return dict(bytes=scene + px * (4 if case["u8"] else 16), flops=project + 40 * pairs)
    if kind == "render":
        return dict(bytes=scene + px * 20, flops=project + 40 * pairs)
    if kind == "scores":
        return dict(bytes=scene + px * 12 + n * 8, flops=project + 50 * pairs)
    ssim = 0 if case["loss"] == "l2l1" else px * 3 * 200
    step = dict(bytes=scene + px * 12, flops=2 * project + 120 * pairs + ssim)
    if kind == "grads":
        return dict(bytes=step["bytes"] + n * PLANES * 4, flops=step["flops"])
    sh_steps = max(case["steps"] // case["sh_every"], 0)
    adam = n * 4 * (geo * 5 * case["steps"] + coef * 5 * sh_steps) + n * 64 * case["steps"]
    return dict(bytes=case["steps"] * step["bytes"] + adam + n * PLANES * 4,
                flops=case["steps"] * step["flops"] + 12 * n * (geo * case["steps"] + coef * sh_steps))


# ---------------------------------------------------------------------------
# The same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _rounded(P):
    """Parameters as the packed f16 storage holds them."""
    return P.half().double()


def _project(P, cam, scaling=None):
    """Differentiable screen-space quantities of every Gaussian in one view.
    scaling: None for the training projection (y grows with ndc y), else the
    viewer's (y down, sigma scaled, no near plane)."""
    V = torch.tensor(cam["view"].astype(np.float64), device=P.device).reshape(4, 4).T
    M = torch.tensor(cam["proj"].astype(np.float64), device=P.device).reshape(4, 4).T
    w, h = cam["width"], cam["height"]
    fx, fy = (float(v) for v in cam["focal"])
    n = P.shape[1]
    pc = V[:3, :3] @ P[0:3] + V[:3, 3:4]
    clip = M @ torch.cat([pc, torch.ones(1, n, dtype=P.dtype, device=P.device)])
    ndc = clip[:2] / clip[3]
    # the depth as f32 products added in order: the sort order is made from it
    v32, p32 = V.float(), P[0:3].detach().float()
    depth = ((v32[2, 0] * p32[0] + v32[2, 1] * p32[1]) + v32[2, 2] * p32[2]) + v32[2, 3]
    ok = (ndc.abs() <= 1.2).all(0)
    ok &= (pc[2] >= 0) if scaling is not None else (pc[2] > 0) & (pc[2] >= 0.2) & (pc[2] <= 1e4)
    sig = torch.exp(P[3:6].clamp(-10, 10)) * (scaling or 1.0)
    q = P[6:10] / P[6:10].norm(dim=0)
    x, y, z, s = q
    one = torch.ones_like(x)
    R = torch.stack([one - 2 * (y * y + z * z), 2 * (x * y - s * z), 2 * (x * z + s * y),
                     2 * (x * y + s * z), one - 2 * (x * x + z * z), 2 * (y * z - s * x),
                     2 * (x * z - s * y), 2 * (y * z + s * x), one - 2 * (x * x + y * y)]).reshape(3, 3, n)
    A = R * sig  # R diag(sigma)
    C3 = torch.einsum("akn,bkn->abn", A, A)
    tz = pc[2]
    J = torch.stack([fx / tz, fy / tz])
    W = V[:2, :3]
    T = J[:, None, :] * W[:, :, None]
    C2 = torch.einsum("ain,ijn,bjn->abn", T, C3, T)
    c00, c11, c01 = C2[0, 0] + 0.3, C2[1, 1] + 0.3, C2[0, 1]
    det = c00 * c11 - c01 * c01
    ok &= det > 0
    mid = 0.5 * (c00 + c11)
    radius = torch.ceil(3 * torch.sqrt(mid + torch.sqrt((mid * mid - det).clamp(min=0)))).detach()
    if scaling is None:
        ok &= (radius <= 512) & (radius >= 1)
    my = 0.5 * (ndc[1] + 1) * h if scaling is None else (ndc[1] * -0.5 + 0.5) * h
    d = -pc / pc.norm(dim=0)
    return dict(mean=torch.stack([0.5 * (ndc[0] + 1) * w, my]),
                conic=torch.stack([c11 / det, -c01 / det, c00 / det]), opacity=torch.sigmoid(P[10]),
                color=_sh_color(P, d).clamp(min=0), radius=radius, depth=depth, ok=ok)


def _sh_color(P, d):
    x, y, z = d
    xx, yy, zz = x * x, y * y, z * z
    basis = [SH_C0 * torch.ones_like(x), -0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x,
             1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * zz - xx - yy),
             -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy),
             -0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z,
             -0.4570457994644658 * y * (4 * zz - xx - yy), 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
             -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
             -0.5900435899266435 * x * (xx - 3 * yy)]
    sh = P[11:59].reshape(16, 3, -1)
    return torch.einsum("kn,kcn->cn", torch.stack(basis), sh) + 0.5


def _lists(p, cam, ts, viewer):
    """Per-tile splat lists in draw order: (tiles' starts, Gaussian per entry)."""
    w, h = cam["width"], cam["height"]
    nx, ny = -(-w // ts), -(-h // ts)
    mx, my, r = p["mean"][0].detach(), p["mean"][1].detach(), p["radius"]
    if viewer:
        x0, y0 = torch.floor((mx - r) / ts), torch.floor((my - r) / ts)
        x1, y1 = torch.floor((mx + r) / ts) + 1, torch.floor((my + r) / ts) + 1
        order = torch.argsort(-p["depth"], stable=True)
    else:
        x0, y0 = torch.floor(mx / ts - r / ts), torch.floor(my / ts - r / ts)
        x1, y1 = torch.ceil(mx / ts + r / ts), torch.ceil(my / ts + r / ts)
        order = torch.argsort(p["depth"].clamp(0, 65535).to(torch.int64) & 0xFFFF, stable=True)
    x0, x1 = x0.clamp(0, nx).long(), x1.clamp(0, nx).long()
    y0, y1 = y0.clamp(0, ny).long(), y1.clamp(0, ny).long()
    count = torch.where(p["ok"], (x1 - x0).clamp(min=0) * (y1 - y0).clamp(min=0), 0)[order]
    g = torch.repeat_interleave(order, count)
    k = torch.arange(g.numel(), device=g.device) - torch.repeat_interleave(count.cumsum(0) - count, count)
    wide = (x1 - x0)[g].clamp(min=1)
    tile = (y0[g] + k // wide) * nx + x0[g] + k % wide
    tile, by = torch.sort(tile, stable=True)
    starts = torch.searchsorted(tile, torch.arange(nx * ny + 1, device=g.device))
    return starts, g[by], nx


def _chunks(starts, ts, room=1 << 25):
    """Groups of tiles of about equal list length, as (tiles, longest list)."""
    length = starts[1:] - starts[:-1]
    order = torch.argsort(length, descending=True)
    sizes, at = length[order].tolist(), 0
    while at < len(sizes) and sizes[at] > 0:
        m = max(1, min(room // (sizes[at] * ts * ts), 4096))
        yield order[at:at + m], sizes[at]
        at += m


def _tile_splats(p, starts, gauss, tiles, k, ts, nx, viewer):
    """Alphas of the tiles' lists at their pixels: (splat ids [B, K], valid, dx, dy, alpha, unclamped)."""
    dev = starts.device
    idx = starts[tiles][:, None] + torch.arange(k, device=dev)
    live = idx < starts[tiles + 1][:, None]
    ids = gauss[idx.clamp(max=max(gauss.numel() - 1, 0))]
    lane = torch.arange(ts * ts, device=dev)
    px = ((tiles % nx) * ts)[:, None] + lane % ts
    py = ((tiles // nx) * ts)[:, None] + lane // ts
    m, c = p["mean"].detach(), p["conic"].detach()
    dx = (px + 0.5)[:, None, :] - m[0][ids][:, :, None]
    dy = (py + 0.5)[:, None, :] - m[1][ids][:, :, None]
    s = 0.5 * (c[0][ids][:, :, None] * dx * dx + c[2][ids][:, :, None] * dy * dy) + c[1][ids][:, :, None] * dx * dy
    raw = p["opacity"].detach()[ids][:, :, None] * torch.exp(-s)
    valid = live[:, :, None] & (s >= 0)
    if viewer:
        r = p["radius"][ids][:, :, None]
        valid &= (dx >= -r) & (dx < r) & (dy >= -r) & (dy < r)
        alpha = raw.clamp(0, 1)
    else:
        alpha = raw.clamp(max=0.999)
        valid &= alpha >= 1 / 255
    return ids, px, py, valid, dx, dy, torch.where(valid, alpha, 0.0), raw


def _composite(P, cam, ts, scaling=None, residual_of=None):
    """The image (rgb, alpha) of one view; with residual_of(rgb), also the
    gradient of sum(residual * rgb) with respect to the 59 planes of P."""
    viewer = scaling is not None
    P = P.detach().requires_grad_(residual_of is not None)
    p = _project(P, cam, scaling)
    starts, gauss, nx = _lists(p, cam, ts, viewer)
    w, h = cam["width"], cam["height"]
    col = p["color"].detach()
    rgb = torch.zeros(h, w, 3, dtype=torch.float64, device=P.device)
    acc = torch.zeros(h, w, dtype=torch.float64, device=P.device)

    def weights(tiles, k):
        ids, px, py, valid, dx, dy, a, raw = _tile_splats(p, starts, gauss, tiles, k, ts, nx, viewer)
        if viewer:  # back to front: what lies in front of a splat follows it in the list
            T = torch.flip(torch.cumprod(torch.flip(1 - a, [1]), 1), [1])
            T = torch.cat([T[:, 1:], torch.ones_like(T[:, :1])], 1)
        else:
            T = torch.cumprod(1 - a, 1)
            T = torch.cat([torch.ones_like(T[:, :1]), T[:, :-1]], 1)
            a = torch.where(T < 1e-4, 0.0, a)  # a pixel stops once it is full
        return ids, px, py, dx, dy, a, raw, T, a * T

    for tiles, k in _chunks(starts, ts):
        ids, px, py, dx, dy, a, raw, T, wt = weights(tiles, k)
        inside = (px < w) & (py < h)
        c = torch.einsum("bkp,cbk->bpc", wt, col[:, ids])
        rgb[py[inside], px[inside]] = c[inside]
        acc[py[inside], px[inside]] = wt.sum(1)[inside]
    if residual_of is None:
        return rgb, acc
    res = residual_of(rgb)
    up = dict(mean=torch.zeros_like(p["mean"]), conic=torch.zeros_like(p["conic"]), color=torch.zeros_like(col),
              opacity=torch.zeros_like(p["opacity"]))
    for tiles, k in _chunks(starts, ts):
        ids, px, py, dx, dy, a, raw, T, wt = weights(tiles, k)
        inside = ((px < w) & (py < h))[:, :, None]
        r = torch.where(inside, res[py.clamp(max=h - 1), px.clamp(max=w - 1)], 0.0)
        rc = torch.einsum("bpc,cbk->bkp", r, col[:, ids])
        behind = torch.flip(torch.cumsum(torch.flip(wt * rc, [1]), 1), [1]) - wt * rc
        da = torch.where(a > 0, rc * T - behind / (1 - a), 0.0)
        da = torch.where(raw > 0.999, 0.0, da)
        ds = -da * raw
        c = p["conic"].detach()[:, ids][..., None]
        flat = ids.reshape(-1)
        add = lambda to, v: to.index_add_(0, flat, v.sum(2).reshape(-1))  # noqa: E731
        for ch in range(3):
            add(up["color"][ch], wt * r[:, None, :, ch])
        add(up["opacity"], da * raw / p["opacity"].detach()[ids][..., None])
        add(up["conic"][0], 0.5 * ds * dx * dx)
        add(up["conic"][1], ds * dx * dy)
        add(up["conic"][2], 0.5 * ds * dy * dy)
        add(up["mean"][0], -ds * (c[0] * dx + c[1] * dy))
        add(up["mean"][1], -ds * (c[1] * dx + c[2] * dy))
    keys = ("mean", "conic", "color", "opacity")
    scalar = sum((torch.where(p["ok"], p[k], 0.0) * torch.where(p["ok"], up[k], 0.0)).sum() for k in keys)
    return rgb, acc, torch.nan_to_num(torch.autograd.grad(scalar, P)[0])


def _ssim_term(img, tgt):
    """The loss's SSIM pseudo-gradient: (1 - ssim) / 2 of the 5x5 windows times the difference."""
    pad = lambda t: torch.nn.functional.pad(t.permute(2, 0, 1)[None], (2, 2, 2, 2), mode="replicate")  # noqa: E731
    box = lambda t: torch.nn.functional.avg_pool2d(t, 5, 1)[0].permute(1, 2, 0)  # noqa: E731
    a, b = pad(img), pad(tgt)
    ma, mb = box(a), box(b)
    va, vb, vab = box(a * a) - ma * ma, box(b * b) - mb * mb, box(a * b) - ma * mb
    ssim = ((2 * ma * mb + 1e-4) * (2 * vab + 9e-4)) / ((ma * ma + mb * mb + 1e-4) * (va + vb + 9e-4))
    return 0.5 * (1 - ssim) * (img - tgt)


def _exact_grads(case, seed):
    P = _rounded(_scene(case["scene"], case["n"], case["sh"], seed))
    G = _rounded(_ground_truth(case, seed))
    w = _weights(case)
    grads, loss = torch.zeros_like(P), 0.0
    for cam in _cameras(case, seed):
        tgt = _composite(G, cam, 16)[0]

        def residual(img, tgt=tgt):
            d = img - tgt
            d = torch.where(d.abs() < 1e-12, 0.0, d)
            out = w["w_l2"] * d + w["w_l1"] * torch.sign(d)
            return out + w["w_ssim"] * _ssim_term(img, tgt) if w["w_ssim"] else out

        img, _, g = _composite(P, cam, case["tile"], residual_of=residual)
        d = img - tgt
        loss += float((0.5 * w["w_l2"] * d * d + w["w_l1"] * d.abs()).sum())
        grads += g
    grads[11 + 3 * (case["sh"] + 1) ** 2:] = 0
    return loss, grads


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sort", "scores"):  # a permutation; counts and the counts' scaled sums
        return None
    if kind == "knn":
        if case["n"] > 120_000:
            return None
        P = _rounded(_scene(case["scene"], case["n"], 0, seed))
        x, density = P[0:3].T.contiguous(), []
        step = max(1, (1 << 27) // case["n"])
        for i in range(0, case["n"], step):
            q = x[i:i + step]
            d2 = sum((q[:, k:k + 1] - x[None, :, k]) ** 2 for k in range(3))
            d2[torch.arange(q.shape[0]), torch.arange(i, i + q.shape[0])] = math.inf
            density.append(torch.topk(d2, 3, dim=1, largest=False).values.sqrt().mean(1))
        density = torch.cat(density)
        raw = _scene(case["scene"], case["n"], 0, seed)[0:3]
        extent = float((raw.amax(1) - raw.amin(1)).max())
        sigma = torch.clamp((density / 3).clamp(min=0.0015 * extent), 0.0007 * extent, 0.007 * extent).clamp(max=0.1)
        P[3:6] = torch.log(sigma).half().double()
        return dict(density=density, params=P)
    if _pairs(case) > 4e8 or case["n"] * len(_sizes(case)) > 2_000_000:
        return None
    if kind == "frame":
        rgb, a = _composite(_rounded(_scene(case["scene"], case["n"], case["sh"], seed)), _cameras(case, seed)[0], 16,
                            scaling=case["scaling"])
        return None if case["u8"] else torch.cat([rgb, a[..., None]], 2)
    if kind == "render":
        P = _rounded(_scene(case["scene"], case["n"], case["sh"], seed))
        got = [_composite(P, c, case["tile"]) for c in _cameras(case, seed)]
        rgb = torch.cat([g[0].reshape(-1, 3) for g in got])
        return dict(rgba=torch.cat([rgb, torch.ones_like(rgb[:, :1])], 1), alpha=torch.cat([g[1].reshape(-1) for g in got]))
    if kind == "train" and (case["steps"] > 1 or case["sh_every"] > 1):
        return None
    loss, grads = _exact_grads(case, seed)
    if kind == "grads":
        return dict(loss=loss, grads=grads)
    return dict(loss=[loss], moment=(1 - BETA1) * grads)
