"""Performance cases of the densifier, through its public entry points.

Each case is one pass of work that a user of the library has it do: a keyframe
densified in one call or as a resident request, the stages after it (filter
and fusion), several requests in one batch, a served stream, fixed-hypothesis
scoring and input preparation.  Scenes are rendered from the seed on the GPU.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from patchmatch_gb300 import native, scene

# kinds of a case:
#   oneshot     Context.densify: host images in, host maps out
#   resident    Request.run + read of the maps into pinned host arrays that the caller keeps, waiting for each keyframe
#   step        Request.run, consistency filter and fusion chained on the device
#   seeded      a request seeded from an earlier keyframe's retained result, few sweeps
#   batch       one Batch over requests of different sizes and source counts
#   served      a keyframe stream through Server
#   hypotheses  Request.score_hypotheses
#   tail_host   filter_consistency + fuse with host arrays
#   tail_device the same with device maps
#   input       gray conversion, resize and FP16 pyramid

_SCENES = {"room": scene.ROOM, "objects": scene.ROOM_OBJECTS, "hall": scene.HALL}
_COMBINE = {"fold": native.COMBINE_FOLD, "max": native.COMBINE_MAX, "top": native.COMBINE_TOPK,
            "fold_separate": native.COMBINE_FOLD_SEPARATE}
_SEAM = {"clamp": native.SEAM_CLAMP, "wrap": native.SEAM_WRAP, "zero": native.SEAM_ZERO}
_CTX = None


def _ctx():
    """The process's context, as a program keeps one."""
    global _CTX
    if _CTX is None:
        _CTX = native.Context(0)
    return _CTX


def _keyframe(kind, name, W, H, S, sweeps=8, scene="room", combine="fold", fmt="u8", sampler="texture", seam="clamp",
              plain=False, patch_half=5, mask=False, sd=0.0):
    c = {"kind": kind, "W": W, "H": H, "S": S, "sweeps": sweeps, "scene": scene, "combine": combine, "fmt": fmt,
         "sampler": sampler, "seam": seam, "plain": plain, "patch_half": patch_half, "mask": mask, "sd": sd}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest keyframes, one call each: host images in, host maps out, the
        # reference's own configuration of two sources (a thumbnail-sized SLAM keyframe)
        _keyframe("oneshot", "oneshot_256x128x2", 256, 128, 2),
        # the small correctness workload of the benchmark, resident and read back by a
        # caller that waits for it: latency, few tiles per SM
        _keyframe("resident", "resident_512x256x4", 512, 256, 4),
        # the headline workload: one keyframe through densification with top-3 views,
        # post-filter, consistency filter and fusion, device-resident
        _keyframe("step", "step_1920x960x6_top3", 1920, 960, 6, scene="objects", combine="top"),
        # the precision form: FP16 images with noise at full resolution, the largest case
        _keyframe("step", "step_3840x1920x8_f16", 3840, 1920, 8, fmt="f16"),
        # steady state of the served form: seeded from an earlier keyframe's result, 2 sweeps
        _keyframe("seeded", "seeded_1920x960x6", 1920, 960, 6, sweeps=2, scene="objects"),
        # the reference's host variant at an odd size: exact bilinear samples that read 0
        # past the border, maximum over the views, propagation without smoothness, mask
        _keyframe("resident", "hostvariant_641x321x5", 641, 321, 5, combine="max", sampler="exact", seam="zero",
                  plain=True, mask=True, sd=2.0),
        # the batched form: requests of different sizes and 3-10 sources in one graph
        {"kind": "batch", "name": "batch_6_requests", "requests": 6, "Wmin": 480, "Wmax": 1920, "Smin": 3, "Smax": 10,
         "sweeps": 4},
        # the served form: a keyframe stream submitted at once, neighbours from the cache,
        # results reused as priors, filter and fusion running on the stream
        {"kind": "served", "name": "served_960x480_16", "W": 960, "H": 480, "keyframes": 16, "sweeps": 8},
        # cost of fixed hypotheses with its per-source parts, as a parity check or an outside
        # optimiser reads it: FP16 images, exact weights
        {"kind": "hypotheses", "name": "hypotheses_500k_x8_f16", "W": 3840, "H": 1920, "S": 8, "n": 500000,
         "fmt": "f16", "combine": "fold"},
        # consistency filter and fusion of finished maps, host arrays in and out: what the
        # reference's cleaner and pruner threads do between keyframes
        {"kind": "tail_host", "name": "tail_host_1920x960x5", "W": 1920, "H": 960, "views": 5},
        # the same chained on device maps at the largest keyframe size
        {"kind": "tail_device", "name": "tail_device_3840x1920x5", "W": 3840, "H": 1920, "views": 5},
        # a colour frame from the camera: gray, half-size thumbnail, FP16 pyramid
        {"kind": "input", "name": "input_3840x1920", "W": 3840, "H": 1920, "channels": 3, "levels": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["oneshot", "resident", "resident", "step", "step", "seeded", "batch", "served", "hypotheses",
                       "tail_host", "tail_device", "input"])
    W = _log_int(rng, 128, 3840)
    H = max(48, W // 2 - rng.choice([0, 0, 0, 1, 5]))
    if kind in ("oneshot", "resident", "step", "seeded"):
        if kind in ("oneshot", "resident"):
            W = _log_int(rng, 128, 1280)
            H = max(48, W // 2 - rng.choice([0, 0, 0, 1, 5]))
        c = _keyframe(kind, None, W, H, rng.randint(1, 10) if kind != "step" else rng.randint(2, 8),
                      sweeps=2 if kind == "seeded" else rng.choice([2, 4, 8]),
                      scene=rng.choice(["room", "objects"]),
                      combine=rng.choice(["fold", "fold", "top", "max", "fold_separate"]),
                      fmt=rng.choice(["u8", "u8", "f16"]))
        if W <= 1280 and rng.random() < 0.4:
            c["sampler"] = "exact"
            c["seam"] = rng.choice(["clamp", "wrap", "zero"])
            c["plain"] = rng.random() < 0.3
        if rng.random() < 0.2:
            c["patch_half"] = 3
        if rng.random() < 0.25:
            c["mask"], c["sd"] = True, 2.0
        return c
    if kind == "batch":
        lo = _log_int(rng, 128, 480)
        return {"kind": kind, "requests": rng.randint(2, 10), "Wmin": lo, "Wmax": lo * 3, "Smin": rng.randint(1, 3),
                "Smax": rng.randint(4, 10), "sweeps": rng.choice([2, 4, 8])}
    if kind == "served":
        W = _log_int(rng, 256, 1280)
        return {"kind": kind, "W": W, "H": W // 2, "keyframes": rng.randint(10, 16), "sweeps": rng.choice([4, 8])}
    if kind == "hypotheses":
        return {"kind": kind, "W": W, "H": H, "S": rng.randint(1, 10), "n": _log_int(rng, 1000, 500000),
                "fmt": rng.choice(["u8", "f16"]), "combine": rng.choice(["fold", "top", "max", "fold_separate"])}
    if kind in ("tail_host", "tail_device"):
        if kind == "tail_host":
            W = min(W, 1920)
            H = W // 2
        return {"kind": kind, "W": W, "H": H, "views": rng.randint(2, 8)}
    return {"kind": "input", "W": W, "H": H, "channels": rng.choice([1, 3, 4]), "levels": rng.randint(1, 5)}


# ---------------------------------------------------------------- inputs

def _render(sc, R, t, W, H, fmt="u8", noise_seed=0, depth=None, bgr=None):
    if fmt == "f16":  # unrounded intensities with sigma-2 noise
        g = torch.empty((H, W), dtype=torch.float32, device="cuda")
        sc.render_device_f32(R, t, W, H, g, noise_sigma=2.0, noise_seed=noise_seed)
        g = g.clamp_(0, 255).half()
        if depth is not None:
            sc.render_device(R, t, W, H, depth=depth)
        return g
    g = torch.empty((H, W), dtype=torch.uint8, device="cuda")
    sc.render_device(R, t, W, H, gray=g, depth=depth, bgr=bgr)
    return g


def _views(c, seed, n):
    """n views of a seeded scene: device images, poses, and the depth map of view 0."""
    objects = c.get("scene", "room") == "objects"
    sc = scene.Scene(_SCENES[c.get("scene", "room")], seed & 0x7FFFFFFF)
    R, t = sc.poses(n, seed & 0x7FFFFFFF, 0.1 if objects else 0.2, 0.8 if objects else 0.5, 15.0)
    depth = torch.empty((c["H"], c["W"]), dtype=torch.float32, device="cuda")
    imgs = [_render(sc, R[k], t[k], c["W"], c["H"], c.get("fmt", "u8"), 100 + k, depth if k == 0 else None)
            for k in range(n)]
    torch.cuda.synchronize()
    return imgs, R, t, depth


def _params(c, seed, **kw):
    p = dict(iterations=c["sweeps"], seed=seed & 0x7FFFFFFF, combine=_COMBINE[c.get("combine", "fold")],
             image_format=native.IMAGE_F16 if c.get("fmt") == "f16" else native.IMAGE_U8,
             sampler=native.SAMPLER_EXACT if c.get("sampler") == "exact" else native.SAMPLER_TEXTURE,
             seam=_SEAM[c.get("seam", "clamp")], patch_half=c.get("patch_half", 5), min_patch_sd=c.get("sd", 0.0),
             propagation=native.PROPAGATION_PLAIN if c.get("plain") else native.PROPAGATION_SMOOTH)
    p.update(kw)
    return native.default_params(**p)


def _mask(c, seed):
    if not c.get("mask"):
        return None
    m = np.ones((c["H"], c["W"]), np.uint8)
    m[-c["H"] // 6:] = 0  # the rig below the camera
    m[:, :: max(7, c["W"] // 40)] = seed & 1
    return m


def _request(c, imgs, R, t, params, mask=None):
    r = _ctx().request(c["W"], c["H"], len(imgs) - 1, params)
    for k, im in enumerate(imgs):
        m = torch.from_numpy(mask).cuda() if k == 0 and mask is not None else None
        r.set_view(k, im.data_ptr(), R[k], t[k], mask=m)
        r.synchronize()
    return r


def _noisy_maps(W, H, n, seed):
    """Depth maps of n views as the densifier leaves them: 0.4 % noise, 10 % holes."""
    sc = scene.Scene(scene.ROOM_OBJECTS, seed & 0x7FFFFFFF)
    R, t = sc.poses(n, seed & 0x7FFFFFFF, 0.1, 0.4, 15.0)
    g = torch.Generator(device="cuda").manual_seed(seed)
    maps = []
    bgr = torch.empty((H, W, 3), dtype=torch.uint8, device="cuda")
    for v in range(n):
        d = torch.empty((H, W), dtype=torch.float32, device="cuda")
        sc.render_device(R[v], t[v], W, H, depth=d, bgr=bgr if v == 0 else None)
        d *= 1 + 0.004 * torch.randn((H, W), generator=g, device="cuda")
        d[torch.rand((H, W), generator=g, device="cuda") < 0.1] = 0
        maps.append(d)
    torch.cuda.synchronize()
    return maps, R, t, bgr


class _Tail:
    """Filter and fusion on device maps: buffers that a program keeps."""

    def __init__(self, maps, R, t, W, H, center, stream):
        self.maps, self.R, self.t, self.W, self.H, self.center, self.stream = maps, R, t, W, H, center, stream
        self.work = [torch.empty((H, W), dtype=torch.float32, device="cuda") for _ in range(len(R) - 1)]
        self.cleaned = torch.zeros((H, W), dtype=torch.float32, device="cuda")
        self.pruned = torch.zeros((H, W), dtype=torch.float32, device="cuda")
        self.xyz = torch.zeros((H * W, 3), dtype=torch.float32, device="cuda")
        self.ij = torch.zeros((H * W, 2), dtype=torch.int32, device="cuda")
        self.count = torch.zeros(1, dtype=torch.int32, device="cuda")
        self.bytes = native.fuse_workspace_bytes(W, H)
        self.ws = torch.empty(self.bytes + 256, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def run(self, center_ptr):
        """Clean view `center` against the others, then fuse it against fresh copies of them."""
        n, st = len(self.R), self.stream
        others = [k for k in range(n) if k != self.center]
        ptrs = [center_ptr if k == self.center else self.maps[k].data_ptr() for k in range(n)]
        _ctx().filter_consistency_device(ptrs, self.W, self.H, self.R, self.t, self.center, 0.01,
                                         self.cleaned.data_ptr(), min_consistent=min(3, n), reproj_px=1.0, stream=st)
        with torch.cuda.stream(torch.cuda.ExternalStream(st)):
            for w, k in zip(self.work, others):  # fusion edits the later maps in place
                w.copy_(self.maps[k], non_blocking=True)
        order = [self.center] + others
        _ctx().fuse_device([self.cleaned.data_ptr()] + [w.data_ptr() for w in self.work], self.W, self.H,
                           self.R[order], self.t[order], 0.08, self.pruned.data_ptr(), self.xyz.data_ptr(),
                           self.count.data_ptr(), (self.ws.data_ptr() + 255) & ~255, self.bytes,
                           ij_ptr=self.ij.data_ptr(), stream=st)
        return {"cleaned": self.cleaned, "pruned": self.pruned, "edited": self.work, "xyz": self.xyz, "ij": self.ij,
                "count": self.count}


# ---------------------------------------------------------------- prepare / run

def prepare(case, seed):
    c, kind, s = dict(case), case["kind"], {}
    if kind == "oneshot":
        imgs, R, t, _ = _views(c, seed, c["S"] + 1)
        s.update(imgs=[i.cpu().numpy() for i in imgs], R=R, t=t, params=_params(c, seed), mask=_mask(c, seed))
        _ctx()
    elif kind == "resident":
        imgs, R, t, _ = _views(c, seed, c["S"] + 1)
        s["req"] = _request(c, imgs, R, t, _params(c, seed), _mask(c, seed))
        H, W = c["H"], c["W"]
        s["out"] = {"depth": torch.zeros((H, W)).pin_memory(), "score": torch.zeros((H, W)).pin_memory(),
                    "plane": torch.zeros((H, W, 3)).pin_memory(), "normal": torch.zeros((H, W, 3)).pin_memory(),
                    "best_view": torch.zeros((H, W), dtype=torch.int32).pin_memory()}
    elif kind == "step":
        imgs, R, t, _ = _views(c, seed, c["S"] + 1)
        s["req"] = _request(c, imgs, R, t, _params(c, seed), _mask(c, seed))
        # resident depth maps of up to four neighbours (the window's other keyframes)
        n = min(5, c["S"] + 1)
        sc = scene.Scene(_SCENES[c["scene"]], seed & 0x7FFFFFFF)
        g = torch.Generator(device="cuda").manual_seed(seed)
        maps = [None]
        for k in range(1, n):
            d = torch.empty((c["H"], c["W"]), dtype=torch.float32, device="cuda")
            sc.render_device(R[k], t[k], c["W"], c["H"], depth=d)
            d *= 1 + 0.004 * torch.randn(d.shape, generator=g, device="cuda")
            d[torch.rand(d.shape, generator=g, device="cuda") < 0.1] = 0
            maps.append(d)
        s["tail"] = _Tail(maps, R[:n], t[:n], c["W"], c["H"], 0, s["req"].stream_handle)
    elif kind == "seeded":
        # the keyframe before this one, densified and retained
        imgs, R, t, _ = _views(c, seed, c["S"] + 1)
        order = [1, 0] + list(range(2, c["S"] + 1))
        prev = _request(c, [imgs[k] for k in order], R[order], t[order], _params(c, seed, iterations=2, keyframe_id=1))
        prev.run()
        s["prior"] = native.Result(_ctx(), c["W"], c["H"])
        s["prior"].snapshot(prev)
        prev.synchronize()
        prev.close()
        s["req"] = _request(c, imgs, R, t, _params(c, seed, keyframe_id=2), _mask(c, seed))
        s["req"].set_prior(s["prior"])
        s["out"] = {"depth": torch.zeros((c["H"], c["W"]), dtype=torch.float32, device="cuda"),
                    "score": torch.zeros((c["H"], c["W"]), dtype=torch.float32, device="cuda"),
                    "normal": torch.zeros((c["H"], c["W"], 3), dtype=torch.float32, device="cuda")}
        torch.cuda.synchronize()
    elif kind == "batch":
        g = np.random.default_rng(seed)
        n = c["requests"]
        s["reqs"] = []
        for k in range(n):
            # sizes and source counts spread evenly over the range, the same for every seed
            f = k / max(1, n - 1)
            W = int(round(c["Wmin"] * (c["Wmax"] / c["Wmin"]) ** f))
            S = c["Smin"] + (k * 5) % (c["Smax"] - c["Smin"] + 1)
            d = {"W": W, "H": W // 2, "S": S, "sweeps": c["sweeps"]}
            sd = int(g.integers(1 << 30))
            imgs, R, t, _ = _views(d, sd, S + 1)
            s["reqs"].append(_request(d, imgs, R, t, _params(d, sd, keyframe_id=k)))
        s["batch"] = native.Batch(_ctx(), s["reqs"])
        s["out"] = [torch.zeros((r.H, r.W), dtype=torch.float32, device="cuda") for r in s["reqs"]]
        torch.cuda.synchronize()
    elif kind == "served":
        sc = scene.Scene(scene.HALL, seed & 0x7FFFFFFF)
        s["stream"] = []
        for k in range(c["keyframes"]):
            R, t = sc.trajectory_pose(seed & 0x7FFFFFFF, 20, 60.0, 1.0 + 0.08 * k)
            s["stream"].append((_render(sc, R, t, c["W"], c["H"]).cpu().numpy(), R, t))
        s["cfg"] = native.server_config(params=native.default_params(iterations=c["sweeps"]), max_inflight=4,
                                        prior_lag=2, dense_output=1)
        _ctx()
    elif kind == "hypotheses":
        imgs, R, t, depth = _views(c, seed, c["S"] + 1)
        s["req"] = _request(c, imgs, R, t, _params(dict(c, sweeps=1, sampler="exact"), seed))
        ij, planes = _hypotheses(c, seed, depth)
        s.update(ij=ij, planes=planes)
    elif kind == "tail_host":
        maps, R, t, bgr = _noisy_maps(c["W"], c["H"], c["views"], seed)
        s.update(maps=[m.cpu().numpy() for m in maps], R=R, t=t, bgr=bgr.cpu().numpy())
        _ctx()
    elif kind == "tail_device":
        maps, R, t, _ = _noisy_maps(c["W"], c["H"], c["views"], seed)
        s["tail"] = _Tail(maps, R, t, c["W"], c["H"], c["views"] // 2, _ctx().stream_handle)
    elif kind == "input":
        s["img"] = _frame(c, seed)
        _ctx()
    s["case"] = c
    return s


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "oneshot":
        return _ctx().densify(state["imgs"], state["R"], state["t"], state["params"], mask=state["mask"])
    if kind == "resident":
        state["req"].run()
        _read(native.lib().pm_request_read, state["req"], state["out"])
        return state["out"]
    if kind == "step":
        state["req"].run()
        out = state["tail"].run(state["req"].depth_device_ptr)
        return out
    if kind == "seeded":
        state["req"].run()
        _read(native.lib().pm_request_read_async, state["req"], state["out"])
        return state["out"]
    if kind == "batch":
        state["batch"].run()
        for r, o in zip(state["reqs"], state["out"]):
            _read(native.lib().pm_request_read_async, r, {"depth": o})
        return state["out"]
    if kind == "served":
        srv = native.Server(_ctx(), state["cfg"])
        tickets = [srv.submit(g, R, t) for g, R, t in state["stream"]]
        maps = [srv.wait(tk, want_score=True)[1:3] for tk in tickets]
        srv.finish()
        dense = [[_whole(a) for a in srv.wait_dense(tk)[1:]] for tk in tickets]
        srv.close()
        return {"maps": maps, "dense": dense}
    if kind == "hypotheses":
        scores, best, per_source = state["req"].score_hypotheses(state["ij"], state["planes"], per_source=True)
        return {"scores": scores, "best": best, "per_source": per_source}
    if kind == "tail_host":
        cl = _ctx().filter_consistency(state["maps"], state["R"], state["t"], 0, 0.01,
                                       min_consistent=min(3, c["views"]), reproj_px=1.0)
        pruned, xyz, bgr, ij, edited = _ctx().fuse([cl] + state["maps"][1:], state["R"], state["t"], state["bgr"], 0.08)
        return {"cleaned": cl, "pruned": pruned, "points": len(xyz), "xyz": _whole(xyz), "bgr": _whole(bgr),
                "ij": _whole(ij), "edited": edited[1:]}
    if kind == "tail_device":
        return state["tail"].run(state["tail"].maps[state["tail"].center].data_ptr())
    ctx = _ctx()
    # the converter's work is enqueued on the context's stream
    with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream_handle)):
        gray = ctx.to_gray(state["img"])
        small = ctx.resize(gray, max(1, c["W"] // 2), max(1, c["H"] // 2))
        thumb = ctx.resize(state["img"], max(1, c["W"] // 2), max(1, c["H"] // 2))
        levels = ctx.pyramid_f16(gray, c["levels"])
    return {"gray": gray, "small": small, "thumb": thumb, "levels": levels}


def _whole(a):
    """The zero-filled array that a call cut its points from: one shape for any number of points."""
    return a if a is None or a.base is None else a.base


def _read(call, req, out):
    """pm_request_read or pm_request_read_async into tensors that the caller keeps (host or device addresses)."""
    m = native.Maps()
    for k, v in out.items():
        setattr(m, k, v.data_ptr())
    _ctx().check(call(req.h, C.byref(m), 0))


def _frame(c, seed):
    sc = scene.Scene(scene.ROOM_OBJECTS, seed & 0x7FFFFFFF)
    R, t = sc.poses(1, seed & 0x7FFFFFFF, 0.1, 0.4, 15.0)
    bgr = torch.empty((c["H"], c["W"], 3), dtype=torch.uint8, device="cuda")
    g = _render(sc, R[0], t[0], c["W"], c["H"], bgr=bgr)
    torch.cuda.synchronize()
    if c["channels"] == 1:
        return g
    return bgr if c["channels"] == 3 else torch.cat([bgr, torch.full_like(bgr[..., :1], 255)], 2).contiguous()


def _hypotheses(c, seed, depth):
    """Planes near and away from the surface at random interior pixels."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, W, H = c["n"], c["W"], c["H"]
    i = torch.randint(6, H - 6, (n,), generator=g, device="cuda")
    j = torch.randint(6, W - 6, (n,), generator=g, device="cuda")
    lat = -math.pi * (i.double() / H - 0.5)
    lon = 2 * math.pi * (j.double() / W - 0.5)
    b = torch.stack([lat.cos() * lon.sin(), -lat.sin(), lat.cos() * lon.cos()], 1)
    nrm = -b + 0.5 * torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    d = depth[i, j].double() * (1 + 0.05 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64)).clamp(0.5, 2)
    dot = (nrm * b).sum(1)
    dot = torch.where(dot.abs() < 0.05, torch.full_like(dot, -0.05), dot)
    planes = (nrm / (dot * d)[:, None]).float()
    return (torch.stack([i, j], 1).int().cpu().numpy(), planes.cpu().numpy())


# ---------------------------------------------------------------- work

TAPS = {1: 4, 3: 16, 5: 36}
FLOP_PER_SAMPLE = 40  # warp, projection, bilinear weight and moments of one sample


def _sweep_work(W, H, S, sweeps, patch_half, es):
    """One densification: every pixel's own plane once, then six refinements per
    visit (the propagated planes a pixel can accept vary and are not counted);
    images in, depth, score and normal out."""
    samples = W * H * S * TAPS[patch_half] * (1 + 6 * sweeps)
    return {"bytes": W * H * (es * (S + 1) + 20), "flops": FLOP_PER_SAMPLE * samples}


def work(case):
    c, kind = case, case["kind"]
    if kind in ("oneshot", "resident", "step", "seeded"):
        w = _sweep_work(c["W"], c["H"], c["S"], c["sweeps"], c["patch_half"], 2 if c["fmt"] == "f16" else 1)
        if kind == "step":
            w["bytes"] += _tail_bytes(c["W"], c["H"], min(5, c["S"] + 1))
        if kind == "seeded":
            w["bytes"] += c["W"] * c["H"] * 20
        return w
    if kind == "batch":
        n, tot = c["requests"], {"bytes": 0, "flops": 0}
        for k in range(n):
            W = int(round(c["Wmin"] * (c["Wmax"] / c["Wmin"]) ** (k / max(1, n - 1))))
            w = _sweep_work(W, W // 2, c["Smin"] + (k * 5) % (c["Smax"] - c["Smin"] + 1), c["sweeps"], 5, 1)
            tot = {q: tot[q] + w[q] for q in tot}
        return tot
    if kind == "served":
        # keyframes with a prior run 2 sweeps from 4 or more neighbours
        w = _sweep_work(c["W"], c["H"], 4, 2, 5, 1)
        return {q: v * max(1, c["keyframes"] - 4) for q, v in w.items()}
    if kind == "hypotheses":
        return {"bytes": c["n"] * (20 + 8 + 4 * c["S"]), "flops": FLOP_PER_SAMPLE * c["n"] * c["S"] * 36}
    if kind in ("tail_host", "tail_device"):
        return {"bytes": _tail_bytes(c["W"], c["H"], c["views"]), "flops": 60 * c["W"] * c["H"] * c["views"]}
    px = c["W"] * c["H"]
    return {"bytes": px * (c["channels"] + 1) + px // 4 * (1 + c["channels"]) + int(px * 2 * 4 / 3),
            "flops": px * 10}


def _tail_bytes(W, H, n):
    """n maps in; the cleaned, pruned and edited maps out; points of about a third of the pixels."""
    return W * H * 4 * (n + 2 + n - 1) + W * H // 3 * 20


# ---------------------------------------------------------------- 64-bit values

def exact(case, seed):
    c, kind = dict(case), case["kind"]
    if kind == "hypotheses":
        return _exact_hypotheses(c, seed)
    if kind == "tail_host":
        maps, R, t, _ = _noisy_maps(c["W"], c["H"], c["views"], seed)
        maps = [m.double() for m in maps]
        cl = _exact_clean(maps, R, t, 0, 0.01, min(3, c["views"]), 1.0)
        return {"cleaned": cl.float().cpu().numpy().astype(np.float64)}
    if kind == "tail_device":
        maps, R, t, _ = _noisy_maps(c["W"], c["H"], c["views"], seed)
        return {"cleaned": _exact_clean([m.double() for m in maps], R, t, c["views"] // 2, 0.01, min(3, c["views"]),
                                        1.0)}
    if kind == "input":
        img = _frame(c, seed).long()
        gray = img if c["channels"] == 1 else (img[..., 2] * 4899 + img[..., 1] * 9617 + img[..., 0] * 1868 + 8192) >> 14
        levels = [gray.double()]
        for _ in range(c["levels"] - 1):
            p = levels[-1]
            p = torch.cat([p, p[-1:]], 0) if p.shape[0] % 2 else p
            p = torch.cat([p, p[:, -1:]], 1) if p.shape[1] % 2 else p
            levels.append((p[0::2, 0::2] + p[0::2, 1::2] + p[1::2, 0::2] + p[1::2, 1::2]) / 4)
        return {"levels": levels}
    return None  # whole runs of a randomised search: no value apart from the draws and decisions of the run


def _bearing(i, j, W, H):
    lat = -math.pi * (i.double() / H - 0.5)
    lon = 2 * math.pi * (j.double() / W - 0.5)
    return torch.stack([lat.cos() * lon.sin(), -lat.sin(), lat.cos() * lon.cos()], -1)


def _project(X, W, H):
    r = X.norm(dim=-1)
    lat = -torch.asin((X[..., 1] / r.clamp_min(1e-12)).clamp(-1, 1))
    lon = torch.atan2(X[..., 0], X[..., 2])
    return W * (0.5 + lon / (2 * math.pi)), H * (0.5 - lat / math.pi), r


def _pose(R0, t0, R1, t1):
    M = np.asarray(R1) @ np.asarray(R0).T
    return (torch.from_numpy(np.ascontiguousarray(M)).cuda(),
            torch.from_numpy(np.asarray(t1) - M @ np.asarray(t0)).cuda())


def _bilinear(img, u, v):
    H, W = img.shape
    u, v = u.clamp(0, W), v.clamp(0, H)
    x, y = u.floor(), v.floor()
    ax, ay = u - x, v - y
    x0, y0 = x.long().clamp(0, W - 1), y.long().clamp(0, H - 1)
    x1, y1 = (x.long() + 1).clamp(0, W - 1), (y.long() + 1).clamp(0, H - 1)
    top = img[y0, x0] * (1 - ax) + img[y0, x1] * ax
    return top * (1 - ay) + (img[y1, x0] * (1 - ax) + img[y1, x1] * ax) * ay


def _exact_hypotheses(c, seed):
    """Bilateral NCC of the 36 taps per source and its combination."""
    imgs, R, t, depth = _views(c, seed, c["S"] + 1)
    ij, planes = _hypotheses(c, seed, depth)
    ij, planes = torch.from_numpy(ij).cuda().long(), torch.from_numpy(planes).cuda().double()
    ref, src = imgs[0].double(), [i.double() for i in imgs[1:]]
    W, H, S = c["W"], c["H"], c["S"]
    poses = [_pose(R[0], t[0], R[k], t[k]) for k in range(1, S + 1)]

    def ncc(m, n):
        sw, sx, sxx = (v * n for v in (m[0], m[1], m[2]))
        mx, my = sx / sw, m[3] / sw
        vx, vy = sxx / sw - mx * mx, m[4] / sw - my * my
        return torch.where((vx < 0.1) | (vy < 0.1), -torch.ones_like(vx), (m[5] / sw - mx * my) / (vx * vy).sqrt())

    scores, per = [], []
    for q in range(0, c["n"], 1 << 17):
        p, pl = ij[q:q + (1 << 17)], planes[q:q + (1 << 17)]
        centre = ref[p[:, 0], p[:, 1]]
        mom = [[torch.zeros_like(centre) for _ in range(6)] for _ in range(S)]
        for k1 in range(-5, 6, 2):
            for k2 in range(-5, 6, 2):
                a, b = p[:, 0] + k1, p[:, 1] + k2
                x = ref[a, b] - centre
                w = torch.exp(-x * x / 5000.0 - (k1 * k1 + k2 * k2) / 50.0)
                bear = _bearing(a, b, W, H)
                X = bear / (pl * bear).sum(1, keepdim=True)
                for r, (M, cc) in enumerate(poses):
                    u, v, _ = _project(X @ M.T + cc, W, H)
                    y = _bilinear(src[r], u, v) - centre
                    for m, val in zip(mom[r], (w, w * x, w * x * x, w * y, w * y * y, w * x * y)):
                        m += val
        sep = [ncc(m, 1) for m in mom]
        per.append(torch.stack(sep, 1))
        mode = c["combine"]
        if mode == "max":
            scores.append(per[-1].max(1).values)
        elif mode == "top":
            k = min(3, S)
            scores.append(per[-1].topk(k, 1).values.mean(1))
        else:
            if mode == "fold":  # moments accumulated over sources 0..r
                run_, sep = [v.clone() for v in mom[0]], sep[:1]
                for r in range(1, S):
                    for k in (3, 4, 5):
                        run_[k] = run_[k] + mom[r][k]
                    sep.append(ncc(run_, r + 1))
            f = -torch.ones_like(sep[0])
            for s2 in sep:
                f = torch.where(((f - s2) / s2).abs() < 0.25, 0.5 * (f + s2), torch.maximum(f, s2))
            scores.append(f)
    return {"scores": torch.cat(scores), "best": None, "per_source": torch.cat(per)}


def _exact_clean(maps, R, t, center, thr, min_consistent, px):
    """Depths that enough views agree with within thr and a px-pixel round trip."""
    H, W = maps[0].shape
    i, j = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"), indexing="ij")
    d = maps[center]
    X0 = _bearing(i, j, W, H) * d[..., None]
    votes = torch.ones_like(d, dtype=torch.int64)
    for k in range(len(maps)):
        if k == center:
            continue
        M, c = _pose(R[center], t[center], R[k], t[k])
        x, y, r = _project(X0 @ M.T + c, W, H)
        ok = (r >= 1e-4) & (x >= 0) & (x < W - 1) & (y >= 0) & (y < H - 1)
        at = torch.where(ok, _bilinear(maps[k], x, y), torch.zeros_like(x))
        ok = ((at - r).abs() < r * thr) & (r >= 1e-4)
        lon, lat = 2 * math.pi * (x / W - 0.5), -math.pi * (y / H - 0.5)
        P = torch.stack([lat.cos() * lon.sin(), -lat.sin(), lat.cos() * lon.cos()], -1) * at[..., None]
        Mi, ci = _pose(R[k], t[k], R[center], t[center])
        xb, yb, rb = _project(P @ Mi.T + ci, W, H)
        ex = (xb - j).abs()
        ex = torch.where(ex > 0.5 * W, W - ex, ex)
        votes += (ok & (rb >= 1e-4) & (ex <= px) & ((yb - i).abs() <= px)).long()
    return torch.where((d > 1e-6) & (votes >= min_consistent), d, torch.zeros_like(d))
