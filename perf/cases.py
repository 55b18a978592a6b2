"""Measured cases: what a user of the library has it do, each through a public entry point.

A case is a plain dict; its "kind" picks the path:

  sam      one frame scored against a target library, then the detection list
           (score_frames + detect): the interactive tool and the per-frame stream
  video    a batch of frames of one shape: moments, FP64 statistics, SAM + CEM
           scores, one detection list per frame (the library's main workload)
  scores   SAM + CEM scoring alone of a batch whose filters are known
           (score_frames_batch; FP16 cubes take the tensor-core scorer)
  rxace    one frame: moments, FP64 statistics, RX and ACE maps
  stats    moments and FP64 statistics alone (a frame whose statistics score
           later frames; cubes above 127 bands)
  bip      SAM of a pixel-interleaved cube without a BSQ copy (hsi_sam_bip)
  train    one gradient step of the learned screen: batch, features, forward and
           backward (the optimiser after it is one elementwise launch)
  screen   the learned screen's logit for every pixel of an FP16 cube
  batch    uneven frames of 16 (mosaic) / 113 / 224 bands replayed as one graph

Scenes follow the library's own synthetic model (mixed endmembers, implanted
targets, anomalies, gain and noise), drawn here with torch from the seed alone.
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

# the package's folder is no Python name, so it goes on the path itself
sys.path.insert(1, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hsi-detectors-cuda_b200"))

import hsi_b200 as hsi  # noqa: E402

LOADING = 1e-6      # diagonal loading of the statistics
SAM_THRESHOLD = 0.10
ACE_THRESHOLD = 0.5
NMS_RADIUS = 2
CAPACITY = 4096
POS_WEIGHT = 2.0

F64 = torch.float64
DTYPES = {"f32": (hsi.F32, torch.float32, 4), "f16": (hsi.F16, torch.float16, 2)}


def listed():
    return [
        # smallest call: a thumbnail or a tracked window, where launches and latency count
        dict(name="sam_64x96_t4", kind="sam", height=64, width=96, bands=113, targets=4, dtype="f32", maps=True),
        # the reference tool's plain use: one target on a 520 x 696 camera frame, angle map and list
        dict(name="sam_520x696_t1", kind="sam", height=520, width=696, bands=113, targets=1, dtype="f32", maps=False),
        # SAM + CEM video, whole step (eight of the benchmark's frames)
        dict(name="video_8x1024_f32", kind="video", frames=8, height=1024, width=1024, bands=113, targets=8,
             dtype="f32"),
        # the FP16 variant's scoring (filters at hand), score maps of every target
        dict(name="scores_8x1024_f16", kind="scores", frames=8, height=1024, width=1024, bands=113, targets=8,
             dtype="f16"),
        # RX + ACE on a small ragged window, where the statistics' latency counts
        dict(name="rxace_250x331", kind="rxace", height=250, width=331, bands=113, targets=8, dtype="f32"),
        # RX + ACE on the precision configuration's frame
        dict(name="rxace_2048x1024", kind="rxace", height=2048, width=1024, bands=113, targets=8, dtype="f32"),
        # RX + ACE above 127 bands (the plain detector of the 224-band configurations)
        dict(name="rxace_1024x1024x224", kind="rxace", height=1024, width=1024, bands=224, targets=16, dtype="f16"),
        # statistics of a full 224-band FP16 frame
        dict(name="stats_2048x2048x224", kind="stats", height=2048, width=2048, bands=224, targets=16, dtype="f16"),
        # pixel-interleaved cube straight from a camera or file
        dict(name="bip_1024_t8", kind="bip", height=1024, width=1024, bands=113, targets=8),
        # screen training step: 8192 samples of a 512 x 512 x 224 frame
        dict(name="train_8192x224", kind="train", height=512, width=512, bands=224, samples=8192, dtype="f16"),
        # screen inference on a full 224-band frame
        dict(name="screen_2048x2048x224", kind="screen", height=2048, width=2048, bands=224),
        # batched stream of uneven frames in one graph
        dict(name="batch_12_uneven", kind="batch", frames=12, sizes_seed=20480),
    ]


# the largest listed cubes: elements of a scored cube, of a cube read once
_SCORED = 8 * 1024 * 1024 * 113
_FRAME = 1024 * 1024 * 224
_READ = 2048 * 2048 * 224


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, bands, least, most_elements, side=2048):
    """Height and width, log-uniform, odd ones among them, at least `least` pixels and at most so many elements."""
    while True:
        h, w = _log(rng, 32, side), _log(rng, 32, side)
        if rng.random() < 0.5:
            w = max(32, w // 8 * 8)
        if h * w >= least and h * w * bands <= most_elements:
            return h, w


def draw(rng: random.Random):
    kind = rng.choice(["sam", "sam", "video", "scores", "rxace", "rxace", "stats", "bip", "train", "screen", "batch"])
    dtype = rng.choice(["f32", "f16"])
    if kind == "sam":
        b = _log(rng, 8, 256)
        h, w = _shape(rng, b, 1024, _FRAME)
        return dict(kind=kind, height=h, width=w, bands=b, targets=rng.randint(1, 16), dtype=dtype,
                    maps=rng.random() < 0.5)
    if kind in ("video", "scores"):
        b, n = _log(rng, 16, 127), rng.randint(1, 8)
        h, w = _shape(rng, b * n, 8192, _SCORED, 1024)
        return dict(kind=kind, frames=n, height=h, width=w, bands=b, targets=rng.randint(1, 8), dtype=dtype)
    if kind == "rxace":
        b = _log(rng, 16, 254)
        h, w = _shape(rng, b, 16384, _FRAME)
        return dict(kind=kind, height=h, width=w, bands=b, targets=rng.randint(1, 16), dtype=dtype)
    if kind == "stats":
        b = _log(rng, 16, 254)
        h, w = _shape(rng, b, 16384, _READ if dtype == "f16" else _READ // 2)
        return dict(kind=kind, height=h, width=w, bands=b, targets=rng.randint(1, 16), dtype=dtype)
    if kind == "bip":
        b = _log(rng, 8, 256)
        h, w = _shape(rng, b, 1024, _FRAME)
        return dict(kind=kind, height=h, width=w, bands=b, targets=rng.randint(1, 16))
    if kind == "train":
        b = _log(rng, 16, 256)
        h, w = _shape(rng, b, 16384, 512 * 512 * 256, 512)
        return dict(kind=kind, height=h, width=w, bands=b, samples=_log(rng, 512, 8192), dtype=dtype)
    if kind == "screen":
        b = _log(rng, 16, 256)
        h, w = _shape(rng, b, 8192, _READ)
        return dict(kind=kind, height=h, width=w, bands=b)
    return dict(kind="batch", frames=rng.randint(3, 10), sizes_seed=rng.randrange(1 << 20))


# ---- inputs ---------------------------------------------------------------------------------------------------


def _spectra(gen, n, bands, dev):
    """n smooth spectra: three Gaussian bumps each (centre U(0, B), width U(5, 30) B / 113, height U(0.1, 0.9))."""
    u = torch.rand((n, 3, 3), generator=gen, device=dev, dtype=F64)
    c, w, h = u[..., 0] * bands, (5 + 25 * u[..., 1]) * bands / 113, 0.1 + 0.8 * u[..., 2]
    b = torch.arange(bands, device=dev, dtype=F64)
    return (h[..., None] * torch.exp(-0.5 * ((b - c[..., None]) / w[..., None]) ** 2)).sum(1).float()


def _library(seed, bands, targets, dev):
    """Endmembers, targets and one anomaly spectrum of a seed."""
    gen = torch.Generator(device=dev).manual_seed(7919 * seed + 13)
    s = _spectra(gen, 6 + targets + 1, bands, dev)
    return s[:6], s[6:6 + targets].contiguous(), s[-1]


def _pixels(seed, P, bands, library, dev, target_frac=0.003, anomaly_frac=0.001):
    """A scene of P pixels as (bands, P) floats: Dirichlet mixes, implants, gain, noise, clipped at zero."""
    ends, targets, anomaly = library
    T = targets.shape[0]
    gen = torch.Generator(device=dev).manual_seed(104729 * seed + 1)
    cube = torch.empty((bands, P), device=dev)
    for p0 in range(0, P, 1 << 20):
        n = min(1 << 20, P - p0)
        a = -torch.log(torch.rand((6, n), generator=gen, device=dev).clamp_min(2.0 ** -25))
        a /= a.sum(0)
        x = ends.t() @ a
        u, gain = (torch.rand(n, generator=gen, device=dev) for _ in range(2))
        alpha = torch.rand(n, generator=gen, device=dev)
        t = (u / target_frac).long()
        hit = t < T
        odd = ~hit & (u > 1 - anomaly_frac)
        mixed = torch.where(hit, 0.2 + 0.6 * alpha, torch.where(odd, 0.5 + 0.5 * alpha, torch.zeros_like(alpha)))
        at = torch.nonzero(hit | odd).squeeze(1)
        other = torch.cat([targets, anomaly[None]])[torch.where(hit, t, torch.full_like(t, T))[at]].t()
        x[:, at] = (1 - mixed[at]) * x[:, at] + mixed[at] * other
        x *= 0.3 + 0.9 * gain
        x += 0.005 * torch.randn((bands, n), generator=gen, device=dev)
        cube[:, p0:p0 + n] = x.clamp_min_(0)
    return cube


def _bsq(pixels, h, w, dtype):
    """A device BSQ cube at the library's plane stride."""
    stride = hsi.plane_stride(h, w)
    cube = torch.zeros((pixels.shape[0], stride), dtype=DTYPES[dtype][1], device=pixels.device)
    cube[:, :h * w] = pixels
    return cube


def _scene(case, seed, k=0):
    """(BSQ cube, targets, norms) of frame k; all frames of a case share the library."""
    h, w, b = case["height"], case["width"], case["bands"]
    lib = _library(seed, b, case.get("targets", 4), "cuda")
    cube = _bsq(_pixels(1009 * seed + k, h * w, b, lib, "cuda"), h, w, case.get("dtype", "f32"))
    norms = lib[1].double().square().sum(1).sqrt().float()
    return cube, lib[1], norms


def _vp(t):
    return C.c_void_p(t.data_ptr())


def _empty(n, dtype=torch.uint8):
    return torch.empty(max(int(n), 256), dtype=dtype, device="cuda")


# ---- sam ------------------------------------------------------------------------------------------------------


def _prepare_sam(case, seed):
    cube, tg, norms = _scene(case, seed)
    h, w = case["height"], case["width"]
    P, T = h * w, tg.shape[0]
    s = dict(cube=cube, tg=tg, norms=norms, h=h, w=w, best=torch.empty(P, device="cuda"),
             target=torch.empty(P, dtype=torch.int32, device="cuda"),
             maps=torch.empty((T, P), device="cuda") if case["maps"] else None,
             found=torch.zeros((CAPACITY, 4), dtype=torch.int32, device="cuda"),
             count=torch.zeros(1, dtype=torch.int32, device="cuda"), ws=_empty(hsi.detect_workspace_bytes(h, w)))
    s["frames"] = [hsi.make_frame(cube, h, w, case["bands"], DTYPES[case["dtype"]][0], sam_targets=tg, sam_norms=norms,
                                  sam_maps=s["maps"], sam_best=s["best"], sam_best_target=s["target"], map_stride=P)]
    return s


def _run_sam(s):
    hsi.score_frames(s["frames"])
    s["count"].zero_()
    hsi.detect(s["best"], s["target"], s["h"], s["w"], SAM_THRESHOLD, NMS_RADIUS, hsi.LOWER_IS_BETTER, CAPACITY,
               out=s["found"], count=s["count"], workspace=s["ws"])
    return [s["best"], s["target"], s["maps"], s["found"], s["count"]]


def _angles(x, targets):
    """Spectral angles, (T, P), of (B, P) pixels in 64 bits."""
    t = targets.double()
    nx = x.square().sum(0).sqrt()
    d = nx * t.square().sum(1).sqrt()[:, None]
    a = torch.acos((t @ x / torch.where(d > 0, d, torch.ones_like(d))).clamp(-1, 1))
    return torch.where(d > 0, a, torch.full_like(a, math.pi / 2))


def _exact_sam(case, seed):
    cube, tg, _ = _scene(case, seed)
    a = _angles(cube[:, :case["height"] * case["width"]].double(), tg)
    return [a.min(0).values, None, a if case["maps"] else None, None, None]


# ---- video and scores -----------------------------------------------------------------------------------------


def _prepare_video(case, seed):
    F, h, w, b = case["frames"], case["height"], case["width"], case["bands"]
    P, T, dt = h * w, case["targets"], DTYPES[case["dtype"]][0]
    scenes = [_scene(case, seed, k) for k in range(F)]
    tg, norms = scenes[0][1:]
    s = dict(cubes=[c for c, _, _ in scenes], tg=tg, norms=norms, bands=b, n=F,
             sam=torch.empty((F, T, P), device="cuda"), cem=torch.empty((F, T, P), device="cuda"),
             best=torch.empty((2, F, P), device="cuda"), which=torch.empty((2, F, P), dtype=torch.int32, device="cuda"),
             weights=torch.zeros((F, T, b), device="cuda"), status=torch.zeros(F, dtype=torch.int32, device="cuda"),
             moments=torch.zeros((F, hsi.moments_elements(b)), dtype=F64, device="cuda"),
             found=torch.zeros((F, CAPACITY, 4), dtype=torch.int32, device="cuda"),
             counts=torch.zeros(F, dtype=torch.int32, device="cuda"))
    if case["kind"] == "scores":  # filters of an earlier frame's statistics: smooth, of the library's scale
        gen = torch.Generator(device="cuda").manual_seed(31 * seed + 5)
        r = torch.randn((F, T, b), generator=gen, device="cuda") * 0.05
        s["weights"].copy_(r + tg / tg.square().sum(1, keepdim=True))
    s["moment_jobs"] = [hsi.moments_job(c, h, w, b, s["moments"][k], dtype=dt) for k, c in enumerate(s["cubes"])]
    arr = (hsi.MomentsJob * F)(*s["moment_jobs"])
    s["moments_ws"] = _empty(hsi.lib().hsi_scene_moments_batch_workspace_bytes(arr, F))
    s["frames"] = [hsi.make_frame(c, h, w, b, dt, sam_targets=tg, sam_norms=norms, sam_maps=s["sam"][k],
                                  sam_best=s["best"][0, k], sam_best_target=s["which"][0, k],
                                  cem_weights=s["weights"][k], cem_maps=s["cem"][k], cem_best=s["best"][1, k],
                                  cem_best_target=s["which"][1, k], map_stride=P) for k, c in enumerate(s["cubes"])]
    s["detect_jobs"] = [hsi.detect_job(s["best"][0, k], s["which"][0, k], h, w, SAM_THRESHOLD, NMS_RADIUS,
                                       hsi.LOWER_IS_BETTER, CAPACITY, s["found"][k], s["counts"][k:k + 1])
                        for k in range(F)]
    s["detect_ws"] = _empty(hsi.detect_batch_workspace_bytes(s["detect_jobs"]))
    return s


def _run_video(s):
    hsi.scene_moments_batch(s["moment_jobs"], s["moments_ws"])
    hsi.build_statistics(s["moments"], s["bands"], s["tg"], LOADING, want64=False, cem_weights=s["weights"],
                         status=s["status"])
    hsi.score_frames_batch(s["frames"])
    s["counts"].zero_()
    hsi.detect_batch(s["detect_jobs"], s["detect_ws"])
    return [s["moments"], s["weights"], s["sam"], s["cem"], s["best"], s["which"], s["found"], s["counts"]]


def _run_scores(s):
    hsi.score_frames_batch(s["frames"])
    return [s["sam"], s["cem"], s["best"]]


def _moments(x):
    """Raw moments, packed as the library packs them, of (B, P) pixels in 64 bits."""
    return torch.cat([x.sum(1), (x @ x.t()).reshape(-1), torch.tensor([float(x.shape[1])], dtype=F64, device=x.device)])


def _statistics(m, b, targets):
    """(mean, whitener, whitened targets (T, B), their squared norms, CEM weights) from raw moments in 64 bits."""
    n = m[-1]
    mean, R = m[:b] / n, m[b:b + b * b].reshape(b, b) / n
    eye = torch.eye(b, dtype=F64, device=m.device)
    L = torch.linalg.cholesky(R - mean[:, None] * mean[None] + LOADING * eye)
    W = torch.linalg.solve_triangular(L, eye, upper=False)
    t = targets.double()
    u = (W @ (t - mean).t()).t().contiguous()
    solved = torch.cholesky_solve(t.t(), torch.linalg.cholesky(R + LOADING * eye)).t()
    return mean, W, u, u.square().sum(1), solved / (solved * t).sum(1, keepdim=True)


def _exact_video(case, seed):
    P, b = case["height"] * case["width"], case["bands"]
    F, T = case["frames"], case["targets"]
    known = _prepare_video(case, seed)["weights"].double() if case["kind"] == "scores" else None
    moments, weights = [], []
    sam = torch.empty((F, T, P), dtype=F64, device="cuda")
    cem = torch.empty((F, T, P), dtype=F64, device="cuda")
    for k in range(F):
        cube, tg, _ = _scene(case, seed, k)
        x = cube[:, :P].double()
        if known is None:
            moments.append(_moments(x))
            weights.append(_statistics(moments[-1], b, tg)[4])
        else:
            weights.append(known[k])
        sam[k] = _angles(x, tg)
        cem[k] = weights[-1] @ x
    best = torch.stack([sam.min(1).values, cem.max(1).values])
    if known is not None:
        return [sam, cem, best]
    return [torch.stack(moments), torch.stack(weights), sam, cem, best, None, None, None]


# ---- rxace and stats ------------------------------------------------------------------------------------------


def _prepare_rxace(case, seed):
    cube, tg, _ = _scene(case, seed)
    h, w, b = case["height"], case["width"], case["bands"]
    P, T = h * w, tg.shape[0]
    plain = b > 127  # the tensor-core scorer holds at most 127 bands
    L = hsi.lib()
    return dict(cube=cube, tg=tg, h=h, w=w, bands=b, dt=DTYPES[case["dtype"]][0], plain=plain,
                moments=torch.empty(hsi.moments_elements(b), dtype=F64, device="cuda"),
                moments_ws=_empty(hsi.stats_workspace_bytes(h, w, b)),
                ws=_empty((L.hsi_rx_ace_simt_workspace_bytes if plain else L.hsi_rx_ace_workspace_bytes)(b, T)),
                rx=torch.empty(P, device="cuda"), best=torch.empty(P, device="cuda"),
                which=torch.empty(P, dtype=torch.int32, device="cuda"), maps=torch.empty((T, P), device="cuda"))


def _run_stats(s):
    hsi.scene_moments(s["cube"], s["h"], s["w"], s["bands"], dtype=s["dt"], out=s["moments"],
                      workspace=s["moments_ws"])
    s["stats"], _, status = hsi.build_statistics(s["moments"], s["bands"], s["tg"], LOADING)
    return [s["moments"], s["stats"], status]


def _run_rxace(s):
    _run_stats(s)
    hsi.rx_ace(s["cube"], s["h"], s["w"], s["bands"], s["stats"][0], s["tg"].shape[0], dtype=s["dt"], rx=s["rx"],
               ace_best=s["best"], ace_target=s["which"], ace_maps=s["maps"], simt=s["plain"], workspace=s["ws"])
    return [s["rx"], s["best"], s["which"], s["maps"]]


def _exact_rxace(case, seed):
    cube, tg, _ = _scene(case, seed)
    P, b = case["height"] * case["width"], case["bands"]
    m = _moments(cube[:, :P].double())
    mean, W, u, uu, cem = _statistics(m, b, tg)
    if case["kind"] == "stats":
        return [m, torch.cat([v.reshape(-1) for v in (mean, W, u, uu, cem)])[None], None]
    rx = torch.empty(P, dtype=F64, device="cuda")
    ace = torch.empty((tg.shape[0], P), dtype=F64, device="cuda")
    for p0 in range(0, P, 1 << 20):
        z = W @ (cube[:, p0:min(P, p0 + (1 << 20))].double() - mean[:, None])
        n = z.shape[1]
        rx[p0:p0 + n] = z.square().sum(0)
        ace[:, p0:p0 + n] = (u @ z).square() / (uu[:, None] * rx[p0:p0 + n])
    return [rx, ace.max(0).values.clamp(0, 1), None, ace]


# ---- bip ------------------------------------------------------------------------------------------------------


def _prepare_bip(case, seed):
    h, w, b, T = case["height"], case["width"], case["bands"], case["targets"]
    lib = _library(seed, b, T, "cuda")
    P = h * w
    return dict(cube=_pixels(1009 * seed, P, b, lib, "cuda").t().contiguous(), tg=lib[1], h=h, w=w, bands=b,
                norms=lib[1].double().square().sum(1).sqrt().float(), maps=torch.empty((T, P), device="cuda"),
                best=torch.empty(P, device="cuda"), which=torch.empty(P, dtype=torch.int32, device="cuda"))


def _run_bip(s):
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    hsi.check(hsi.lib().hsi_sam_bip(_vp(s["cube"]), s["h"], s["w"], s["bands"], _vp(s["tg"]), _vp(s["norms"]),
                                    s["tg"].shape[0], _vp(s["maps"]), s["h"] * s["w"], _vp(s["best"]),
                                    _vp(s["which"]), stream), "hsi_sam_bip")
    return [s["maps"], s["best"], s["which"]]


def _exact_bip(case, seed):
    s = _prepare_bip(case, seed)
    a = _angles(s["cube"].t().double(), s["tg"])
    return [a, a.min(0).values, None]


# ---- the learned screen ---------------------------------------------------------------------------------------


def _network(seed, b):
    """Parameters W1[64][Bp] | b1 | W2[32][64] | b2 | w3 | b3 of a screen some way into its training."""
    bp = (b + 63) // 64 * 64
    gen = torch.Generator(device="cuda").manual_seed(17 * seed + 3)

    def r(*shape):
        return torch.rand(shape, generator=gen, device="cuda") * 2 - 1

    w1 = torch.zeros((64, bp), device="cuda")
    w1[:, :b] = r(64, b) * math.sqrt(6 / b)
    parts = [w1, 0.1 * r(64), r(32, 64) * math.sqrt(6 / 64), 0.1 * r(32), r(32) * math.sqrt(6 / 32), r(1)]
    return torch.cat([p.reshape(-1) for p in parts]), bp


def _layers(p, b, bp):
    """The same parameters as 64-bit layers, the weights as the network uses them (rounded to bfloat16)."""
    p = p.double()
    q = [64 * bp, 64, 2048, 32, 32, 1]
    w1, b1, w2, b2, w3, b3 = torch.split(p, q)

    def r(t):
        return t.to(torch.bfloat16).double()

    return r(w1).reshape(64, bp)[:, :b], b1, r(w2).reshape(32, 64), b2, r(w3), b3


def _normaliser(cube, P, b, bp):
    """Per band: mean and a power of two near 1 / sigma."""
    norm = torch.zeros(2 * bp, device="cuda")
    for k in range(b):
        x = cube[k, :P].double()
        norm[k] = x.mean()
        norm[bp + k] = torch.exp2(torch.round(-torch.log2(x.std().clamp(2.0 ** -12, 2.0 ** 14))))
    return norm


def _prepare_train(case, seed):
    cube = _scene(case, seed)[0]
    h, w, b, n = case["height"], case["width"], case["bands"], case["samples"]
    P = h * w
    p, bp = _network(seed, b)
    gen = torch.Generator(device="cuda").manual_seed(seed + 99)
    score = torch.rand(P, generator=gen, device="cuda") ** 4  # a detector's scores: few above the threshold
    at = torch.nonzero(score >= ACE_THRESHOLD).squeeze(1)[:1 << 16].int()
    pos = torch.stack([at % w, at // w, torch.zeros_like(at), score[at.long()].view(torch.int32)], 1).contiguous()
    L = hsi.lib()
    return dict(cube=cube, dt=DTYPES[case["dtype"]][0], h=h, w=w, bands=b, n=n, p=p, norm=_normaliser(cube, P, b, bp),
                score=score, pos=pos, count=torch.tensor([at.numel()], dtype=torch.int32, device="cuda"),
                index=torch.empty(n, dtype=torch.int32, device="cuda"), labels=torch.empty(n, device="cuda"),
                features=torch.empty((bp, n), device="cuda"), grads=torch.zeros_like(p),
                loss=torch.zeros(1, device="cuda"), ws=_empty(L.hsi_screen_train_workspace_bytes(b, n)), seed=seed)


def _run_train(s):
    L, n, b = hsi.lib(), s["n"], s["bands"]
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    hsi.check(L.hsi_screen_batch(_vp(s["pos"]), _vp(s["count"]), s["pos"].shape[0], s["h"], s["w"], _vp(s["score"]),
                                 ACE_THRESHOLD, s["seed"], n // 4, n, _vp(s["index"]), _vp(s["labels"]), stream))
    hsi.check(L.hsi_screen_gather(_vp(s["cube"]), s["dt"], s["cube"].shape[1], b, _vp(s["norm"]), _vp(s["index"]), n,
                                  _vp(s["features"]), stream))
    hsi.check(L.hsi_screen_gradients(_vp(s["p"]), b, _vp(s["features"]), _vp(s["labels"]), n, POS_WEIGHT,
                                     _vp(s["grads"]), _vp(s["loss"]), _vp(s["ws"]), s["ws"].numel(), stream))
    return [s["index"], s["labels"], s["features"], s["grads"], s["loss"]]


def _mix64(z):
    m = (1 << 64) - 1
    z = (z + 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def _exact_train(case, seed):
    s = _prepare_train(case, seed)
    n, b, P = s["n"], s["bands"], s["h"] * s["w"]
    bp = s["features"].shape[0]
    hashes = [_mix64((seed * 0x100000001B3 + k) & ((1 << 64) - 1)) for k in range(n)]
    at = (s["pos"][:, 1].long() * s["w"] + s["pos"][:, 0].long()).cpu().numpy()
    index = torch.from_numpy(np.array([at[v % len(at)] if k < n // 4 and len(at) else v % P
                                       for k, v in enumerate(hashes)], np.int64)).cuda()
    y = (s["score"][index] >= ACE_THRESHOLD).double()
    x = s["cube"][:, index].float()
    x = ((x - s["norm"][:b, None]) * s["norm"][bp:bp + b, None]).to(torch.bfloat16).double()
    w1, b1, w2, b2, w3, b3 = _layers(s["p"], b, bp)
    z1 = w1 @ x + b1[:, None]
    h1 = z1.clamp_min(0).float().to(torch.bfloat16).double()
    z2 = w2 @ h1 + b2[:, None]
    h2 = z2.clamp_min(0)
    z3 = w3 @ h2 + b3
    weight = torch.where(y > 0.5, POS_WEIGHT, 1.0)
    loss = (weight * (torch.nn.functional.softplus(z3, threshold=60) - y * z3)).mean()
    d3 = weight * (torch.sigmoid(z3) - y) / n
    d2 = torch.where(z2 > 0, w3[:, None] * d3, torch.zeros_like(z2))
    d1 = torch.where(h1 > 0, w2.t() @ d2, torch.zeros_like(z1))
    g1 = torch.zeros((64, bp), dtype=F64, device="cuda")
    g1[:, :b] = d1 @ x.t()
    grads = torch.cat([g1.reshape(-1), d1.sum(1), (d2 @ h1.t()).reshape(-1), d2.sum(1), h2 @ d3, d3.sum()[None]])
    features = torch.zeros((bp, n), dtype=F64, device="cuda")
    features[:b] = x
    return [None, y, features, grads, loss[None]]


def _prepare_screen(case, seed):
    cube = _scene(dict(case, dtype="f16"), seed)[0]
    h, w, b = case["height"], case["width"], case["bands"]
    net = hsi.Screen(b, seed=1)
    p, bp = _network(seed, b)
    net.params.copy_(p)
    return dict(net=net, cube=cube, h=h, w=w, norm=_normaliser(cube, h * w, b, bp),
                out=torch.empty(h * w, device="cuda"))


def _run_screen(s):
    return s["net"].logits(s["cube"], s["h"], s["w"], s["norm"], out=s["out"])


def _exact_screen(case, seed):
    cube = _scene(dict(case, dtype="f16"), seed)[0]
    b, P = case["bands"], case["height"] * case["width"]
    p, bp = _network(seed, b)
    norm = _normaliser(cube, P, b, bp).double()
    w1, b1, w2, b2, w3, b3 = _layers(p, b, bp)
    out = torch.empty(P, dtype=F64, device="cuda")
    for p0 in range(0, P, 1 << 20):
        x = cube[:, p0:min(P, p0 + (1 << 20))].double()
        h1 = (w1 @ ((x - norm[:b, None]) * norm[bp:bp + b, None]) + b1[:, None]).clamp_min(0)
        h2 = (w2 @ h1.float().to(torch.bfloat16).double() + b2[:, None]).clamp_min(0)
        out[p0:p0 + x.shape[1]] = w3 @ h2 + b3
    return out


# ---- batch ----------------------------------------------------------------------------------------------------


def _batch_specs(case):
    """(height, width, bands, targets) of each frame: sides log-uniform in 256..2048 x 256..1024, multiples of 8,
    bands 16 / 113 / 224 in turn, 1 to 16 targets."""
    rng = random.Random(case["sizes_seed"])
    return [(_log(rng, 256, 2048) // 8 * 8, _log(rng, 256, 1024) // 8 * 8, (16, 113, 224)[k % 3], rng.randint(1, 16))
            for k in range(case["frames"])]


class _Owned:
    """Device memory of the library as torch sees it."""

    def __init__(self, ptr, n, typestr, keep):
        self.keep = keep
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(ptr, False), version=3)


def _frame_of(seed, k, h, w, b, t):
    lib = _library(seed + k, b, t, "cuda")
    return _pixels(1009 * seed + k, h * w, b, lib, "cuda"), lib[1]


def _prepare_batch(case, seed):
    frames = []
    for k, (h, w, b, t) in enumerate(_batch_specs(case)):
        x, tg = _frame_of(seed, k, h, w, b, t)
        if b == 16:  # a 4 x 4 snapshot mosaic, demosaiced in the run
            raw = x.reshape(4, 4, h, w).permute(2, 0, 3, 1).reshape(4 * h, 4 * w).contiguous()
            frames.append(dict(raw=raw, period=4, bands=b, targets=tg.cpu().numpy()))
        else:
            frames.append(dict(cube=_bsq(x, h, w, "f32"), height=h, width=w, bands=b, dtype=hsi.F32,
                               targets=tg.cpu().numpy()))
    # fixed plan: the autotuner's choice may change from one creation to the next
    batch = hsi.Batch(frames, sam_threshold=SAM_THRESHOLD, ace_threshold=ACE_THRESHOLD, nms_radius=NMS_RADIUS,
                      capacity=CAPACITY, autotune=False)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    batch.run(stream)
    batch.capture(stream)
    torch.cuda.current_stream().wait_stream(stream)
    outs = []
    for k, (h, w, _, _) in enumerate(_batch_specs(case)):
        o = batch.outputs(k)
        for name, kind in (("sam_best", "<f4"), ("sam_target", "<i4"), ("rx", "<f4"), ("ace_best", "<f4"),
                           ("ace_target", "<i4")):
            outs.append(torch.as_tensor(_Owned(getattr(o, name), h * w, kind, batch), device="cuda"))
        if k == 0:  # the counts of every frame's three lists lie one after the other
            counts = torch.as_tensor(_Owned(o.counts, 3 * case["frames"], "<i4", batch), device="cuda")
    return dict(batch=batch, frames=frames, outs=outs + [counts])


def _run_batch(s):
    s["batch"].launch(torch.cuda.current_stream())
    return s["outs"]


def _exact_batch(case, seed):
    outs = []
    for k, (h, w, b, t) in enumerate(_batch_specs(case)):
        x, tg = _frame_of(seed, k, h, w, b, t)
        x = x.double()
        mean, W, u, uu, _ = _statistics(_moments(x), b, tg)
        z = W @ (x - mean[:, None])
        rx = z.square().sum(0)
        ace = ((u @ z).square() / (uu[:, None] * rx)).max(0).values.clamp(0, 1)
        outs += [_angles(x, tg).min(0).values, None, rx, ace, None]
    return outs + [None]


# ---- the interface --------------------------------------------------------------------------------------------

_PREPARE = dict(sam=_prepare_sam, video=_prepare_video, scores=_prepare_video, rxace=_prepare_rxace,
                stats=_prepare_rxace, bip=_prepare_bip, train=_prepare_train, screen=_prepare_screen,
                batch=_prepare_batch)
_RUN = dict(sam=_run_sam, video=_run_video, scores=_run_scores, rxace=_run_rxace, stats=_run_stats, bip=_run_bip,
            train=_run_train, screen=_run_screen, batch=_run_batch)
_EXACT = dict(sam=_exact_sam, video=_exact_video, scores=_exact_video, rxace=_exact_rxace, stats=_exact_rxace,
              bip=_exact_bip, train=_exact_train, screen=_exact_screen, batch=_exact_batch)


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def work(case):
    """Bytes: each input read once, each output written once.  Operations: a multiply and an add each count."""
    kind = case["kind"]
    if kind == "batch":
        size = [(h * w, b, t) for h, w, b, t in _batch_specs(case)]
        return dict(bytes=sum(4 * P * b + 20 * P for P, b, t in size),
                    flops=sum(P * (2 * b * t + 2 * b * b + 2 * b * t) for P, b, t in size))
    P, b, T = case["height"] * case["width"], case["bands"], case.get("targets", 0)
    e = DTYPES[case.get("dtype", "f16" if kind == "screen" else "f32")][2]
    if kind == "sam":
        return dict(bytes=P * (e * b + 8 + (4 * T if case["maps"] else 0)), flops=2 * P * b * (T + 1))
    if kind == "scores":
        return dict(bytes=case["frames"] * P * (e * b + 8 * T + 8), flops=case["frames"] * 2 * P * b * (2 * T + 1))
    if kind == "video":
        return dict(bytes=case["frames"] * P * (e * b + 8 * T + 16),
                    flops=case["frames"] * P * (b * b + 2 * b * (2 * T + 1)))
    if kind == "rxace":
        return dict(bytes=P * (e * b + 4 * T + 12), flops=P * (b * b + b * b + 2 * b * T))
    if kind == "stats":
        return dict(bytes=P * e * b + 8 * (2 * b * b + 2 * T * b), flops=P * b * b + b * b * b)
    if kind == "bip":
        return dict(bytes=P * (4 * b + 4 * T + 8), flops=2 * P * b * (T + 1))
    if kind == "screen":
        return dict(bytes=P * (2 * b + 4), flops=2 * P * (64 * b + 64 * 32 + 32))
    n, bp = case["samples"], (b + 63) // 64 * 64  # train: the pixels' spectra in; features, labels, indices, grads out
    return dict(bytes=n * (e * b + 4 * bp + 8) + 8 * 64 * bp, flops=2 * n * (2 * 64 * b + 3 * 64 * 32))
