"""The work the framework's users have it do, as cases that can be timed and
compared: renders, AOV passes, batches, the compositor's filters, the learned
denoiser (inference and training) and its convolution layers, each through the
public entry points of ``rendertoy_gb300.Context``.

A case is a dict of plain values.  ``listed()`` names the cases, ``draw(rng)``
gives more of the same ranges, ``prepare(case, seed)`` makes what a program has
in hand before the call, ``run(state)`` is one pass, ``work(case)`` the bytes
and operations a pass cannot do without and ``exact(case, seed)`` the outputs
in 64-bit arithmetic by plain torch.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import rendertoy_gb300 as rt
from rendertoy_gb300 import scenes

# The denoiser's layers: first source, read upsampled, skip source, output,
# padded and real output channels, real input channels, ReLU; its tensors:
# channels and level (resolution = full >> level).
TENSORS = {"X": (16, 0), "A0a": (32, 0), "S0": (32, 0), "P1": (32, 1), "A1a": (64, 1), "S1": (64, 1),
           "P2": (64, 2), "A2a": (96, 2), "S2": (96, 2), "P3": (96, 3), "A3a": (128, 3), "S3": (128, 3),
           "P4": (128, 4), "B": (160, 4), "U3": (128, 3), "U2": (96, 2), "U1": (64, 1), "U0": (32, 0)}
POOLED = {"P1": "S0", "P2": "S1", "P3": "S2", "P4": "S3"}
LAYERS = [("X", 0, None, "A0a", 32, 32, 11, 1), ("A0a", 0, None, "S0", 32, 32, 32, 1),
          ("P1", 0, None, "A1a", 64, 64, 32, 1), ("A1a", 0, None, "S1", 64, 64, 64, 1),
          ("P2", 0, None, "A2a", 96, 96, 64, 1), ("A2a", 0, None, "S2", 96, 96, 96, 1),
          ("P3", 0, None, "A3a", 128, 128, 96, 1), ("A3a", 0, None, "S3", 128, 128, 128, 1),
          ("P4", 0, None, "B", 160, 160, 128, 1), ("B", 1, "S3", "U3", 128, 128, 288, 1),
          ("U3", 1, "S2", "U2", 96, 96, 224, 1), ("U2", 1, "S1", "U1", 64, 64, 160, 1),
          ("U1", 1, "S0", "U0", 32, 32, 96, 1), ("U0", 0, None, None, 32, 25, 32, 0)]
TAPS, REL_EPS = 25, 1e-2
LR, STEP, SECOND_MOMENT = 3e-4, 1000, 1e-6  # a training run resumed in its middle


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one 5 x 5 edge kernel on a thumbnail, the library's default (synchronous) call: latency
        dict(name="convolve5_256", kind="convolve", W=256, H=256, k=5),
        # the bench frame's Gaussian blur in a frame loop that enqueues (sigma 8, 49 taps)
        dict(name="blur49_1024", kind="blur", W=1024, H=1024, size=49, sigma=8.0),
        # the bloom that follows the denoiser on a full-HD frame
        dict(name="bloom49_1080p", kind="bloom", W=1920, H=1080, size=49, sigma=8.0, threshold=1.0),
        # normal, albedo and depth passes of a smooth mesh at full HD: the denoiser's other inputs
        dict(name="aov_1080p", kind="aov", scene="icosphere", subdiv=6, W=1920, H=1080),
        # the Cornell box at its usual size: a preview frame of a scene that sits in the caches
        dict(name="render_cornell", kind="render", scene="cornell", subdiv=0, W=256, H=256, spp=16, depth=8),
        # glass, metal, clearcoat, sheen and subsurface together, an odd frame
        dict(name="render_mixed_odd", kind="render", scene="mixed", subdiv=0, W=517, H=389, spp=9, depth=8),
        # the headline frame: 1.3 M triangles, 1024 x 1024, 64 samples, depth 12
        dict(name="render_icosphere", kind="render", scene="icosphere", subdiv=8, W=1024, H=1024, spp=64, depth=12),
        # uneven textured scenes in one wavefront, replayed as a CUDA graph: how training pairs are made
        dict(name="batch_8_scenes", kind="batch", scenes=8, tris=60000, W=512, H=384, spp=8, depth=8),
        # one denoised full-HD frame (1080 rows: padded to 1088)
        dict(name="denoise_1080p", kind="denoise", W=1920, H=1080, spp=16),
        # one Adam step at the training configuration's minibatch
        dict(name="train_32x256", kind="train", N=32, H=256, W=256),
        # a decoder layer of a full-HD frame: upsampled source + skip connection
        dict(name="conv_fwd_decoder", kind="conv_fwd", N=1, H=544, W=960, C1=96, up=1, C2=64, Cout=64),
        # an encoder layer's backward pass: data and weight gradients
        dict(name="conv_bwd_encoder", kind="conv_bwd", N=8, H=128, W=128, C1=64, up=0, C2=0, Cout=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["convolve", "blur", "bloom", "aov", "render", "render", "batch", "denoise", "train",
                       "conv_fwd", "conv_bwd"])
    W, H = _log(rng, 64, 1920), _log(rng, 64, 1080)
    if kind == "convolve":
        return dict(kind=kind, W=W, H=H, k=rng.choice([3, 5, 5, 7]))
    if kind == "blur":
        size = rng.choice([3, 7, 15, 25, 49, 65])
        return dict(kind=kind, W=W, H=H, size=size, sigma=size / 6.0)
    if kind == "bloom":
        size = rng.choice([7, 15, 25, 49])
        return dict(kind=kind, W=W, H=H, size=size, sigma=size / 6.0, threshold=1.0)
    if kind == "aov":
        return dict(kind=kind, scene=rng.choice(["cornell", "mixed", "icosphere"]), subdiv=rng.randint(3, 7), W=W, H=H)
    if kind == "render":
        W, H = _log(rng, 64, 1024), _log(rng, 64, 1024)
        return dict(kind=kind, scene=rng.choice(["cornell", "mixed", "icosphere"]), subdiv=rng.randint(3, 7), W=W, H=H,
                    spp=_log(rng, 1, 32), depth=rng.randint(2, 12))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 8), tris=_log(rng, 2000, 60000), W=_log(rng, 96, 640),
                    H=_log(rng, 96, 480), spp=_log(rng, 1, 12), depth=rng.randint(3, 8))
    if kind == "denoise":
        return dict(kind=kind, W=W, H=H, spp=_log(rng, 1, 256))
    if kind == "train":
        return dict(kind=kind, N=_log(rng, 1, 16), H=16 * rng.randint(3, 16), W=16 * rng.randint(3, 16))
    up = rng.randint(0, 1)
    C1 = 32 * rng.randint(1, 4)
    return dict(kind=kind, N=rng.randint(1, 8), H=2 * _log(rng, 8, 128), W=2 * _log(rng, 8, 128), C1=C1, up=up,
                C2=32 * rng.randint(1, 3) if up else 0, Cout=rng.choice([32, 64, 96, 128]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=24)
def _scene(name, subdiv, geometry):
    if name == "cornell":
        return scenes.cornell_box()
    if name == "mixed":
        return scenes.cornell_mixed()
    return scenes.displaced_icosphere(subdiv, seed=1 + geometry)


@functools.lru_cache(maxsize=64)
def _procedural(seed, tris):
    return scenes.procedural_scene(seed, n_tris=tris)[0]


def _camera(seed):
    """The Cornell camera moved about: a frame of a walk through the room."""
    rng = np.random.RandomState(seed % (1 << 31))
    eye = np.asarray(scenes.CORNELL_EYE) + rng.uniform(-40.0, 40.0, 3) - scenes.ROOM_CENTER
    return scenes.fov_camera(tuple(eye), vfov_deg=40.0, near=700.0, far=1500.0)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _image(g, H, W, spp=4.0):
    """A path tracer's radiance: smooth light and shade, a few bright areas, sampling noise."""
    low = torch.rand((1, 3, H // 32 + 2, W // 32 + 2), generator=g, device="cuda")
    base = torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear", align_corners=True)[0].permute(1, 2, 0)
    base = 0.02 + 1.5 * base ** 3
    noise = torch.rand((H, W, 1), generator=g, device="cuda").clamp_min(1e-6).log().neg()
    w = 1.0 / math.sqrt(max(spp, 1.0))
    return (base * ((1.0 - w) + w * noise)).contiguous()


def _raw(seed, N, H, W, spp):
    """The denoiser's network input [N][H][W][11] and a clean target."""
    g = _gen(seed)
    raw = torch.empty((N, H, W, 11), device="cuda")
    tgt = torch.empty((N, H, W, 3), device="cuda")
    for n in range(N):
        raw[n, ..., 0:3] = _image(g, H, W, spp)
        raw[n, ..., 3:6] = _image(g, H, W, 1e6).clamp(0, 1)
        raw[n, ..., 6:9] = _image(g, H, W, 1e6).clamp(0, 1)
        raw[n, ..., 9] = _image(g, H, W, 1e6)[..., 0].clamp(0, 1)
        tgt[n] = _image(g, H, W, 1e6)
    raw[..., 10] = float(spp)
    return raw, tgt


def _layout():
    """Per layer: padded input channels, offsets of w [cout][9][cin] and b [cout] in the flat parameter array."""
    rows, off = [], 0
    for s1, up, s2, out, cop, co, ci, relu in LAYERS:
        c1 = TENSORS[s1][0]
        cip = c1 + (TENSORS[s2][0] if s2 else 0)
        w_off = off
        off = (off + cop * 9 * cip + 3) // 4 * 4
        b_off = off
        off = (off + cop + 3) // 4 * 4
        rows.append((cip, w_off, b_off))
    return rows, off


def _params(seed):
    """He-normal weights and small biases on the network's real entries, zeros in its padding."""
    rng = np.random.default_rng(seed % (1 << 31))
    rows, n = _layout()
    p = np.zeros(n, np.float32)
    for (s1, up, s2, out, cop, co, ci, relu), (cip, w_off, b_off) in zip(LAYERS, rows):
        real = ci if s2 is None else cip
        w = np.zeros((cop, 9, cip), np.float32)
        w[:co, :, :real] = rng.standard_normal((co, 9, real), np.float32) * math.sqrt(2.0 / (9 * ci))
        p[w_off:w_off + w.size] = w.ravel()
        p[b_off:b_off + co] = 0.02 * rng.standard_normal(co, np.float32)
    return p


def _conv_inputs(c, seed):
    g = _gen(seed)

    def act(*shape):  # ReLU outputs: about half zeros
        return torch.randn(shape, generator=g, device="cuda").clamp_min(0).to(torch.bfloat16)

    N, H, W, C1, C2, Cout, up = (c[k] for k in ("N", "H", "W", "C1", "C2", "Cout", "up"))
    x1 = act(N, H // 2, W // 2, C1) if up else act(N, H, W, C1)
    x2 = act(N, H, W, C2) if C2 else None
    s = math.sqrt(2.0 / (9 * (C1 + C2)))
    w = (torch.randn((Cout, 9, C1 + C2), generator=g, device="cuda") * s).to(torch.bfloat16)
    bias = 0.02 * torch.randn((Cout,), generator=g, device="cuda")
    dout = (1e-3 * torch.randn((N, H, W, Cout), generator=g, device="cuda")).to(torch.bfloat16)
    return x1, x2, w, bias, dout


def _kernel(c, seed):
    """An edge kernel's weights: positive and negative, summing to about zero."""
    k = np.random.RandomState(seed % (1 << 31)).normal(0.0, 1.0, (c["k"], c["k"]))
    return (k - k.mean()).astype(np.float32)


def _mean_spp(seed):
    return float(2 ** (2 + seed % 4))


def prepare(case, seed):
    c = case
    kind = c["kind"]
    ctx = rt.Context(0)
    st = {"kind": kind, "case": c, "ctx": ctx, "seed": int(seed)}
    new = lambda *s, dtype=torch.float32: torch.empty(s, device="cuda", dtype=dtype)  # noqa: E731
    if kind in ("convolve", "blur", "bloom"):
        st["img"] = _image(_gen(seed), c["H"], c["W"])
        st["out"] = new(c["H"], c["W"], 3)
        if kind == "convolve":
            st["kernel"] = _kernel(c, seed)
        else:
            ctx.set_option(rt.OPT_ASYNC, 1)  # a frame loop: device images, one wait at its end
    elif kind in ("aov", "render"):
        ctx.upload(_scene(c["scene"], c["subdiv"], seed & 1))
        st["camera"] = _camera(seed)
        st["out"] = (tuple(new(c["H"], c["W"], 3) for _ in range(3)) if kind == "aov" else new(c["H"], c["W"], 3))
    elif kind == "batch":
        rng = np.random.RandomState(seed % (1 << 31))
        st["jobs"], scs = [], []
        for k in range(c["scenes"]):
            # uneven: triangle counts over a factor of 30, frames over a factor of 4
            scs.append(_procedural(8 * (seed & 1) + k, max(64, int(c["tris"] * (k + 1) ** 2 / c["scenes"] ** 2))))
            f = 0.5 + 0.5 * (k % 3)
            st["jobs"].append(dict(scene=k, W=int(c["W"] * f), H=int(c["H"] * f), spp=c["spp"] + k % 3,
                                   seed=int(rng.randint(1 << 30))))
        ctx.batch_upload(scs)
        ctx.set_option(rt.OPT_GRAPH, 1)
        st["out"] = new(3 * sum(j["W"] * j["H"] for j in st["jobs"]))
    elif kind == "denoise":
        ctx.dn_init(0)
        ctx.dn_set_params(_params(seed))
        raw, _ = _raw(seed, 1, c["H"], c["W"], c["spp"])
        st["passes"] = [raw[0, ..., 0:3].contiguous(), raw[0, ..., 3:6].contiguous(), raw[0, ..., 6:9].contiguous(),
                        raw[0, ..., 9:10].expand(-1, -1, 3).contiguous()]
        st["out"] = new(c["H"], c["W"], 3)
    elif kind == "train":
        ctx.dn_init(0)
        p = _params(seed)
        ctx.dn_set_params(p)
        ctx.dn_set_adam(np.zeros_like(p), np.full_like(p, SECOND_MOMENT), STEP)
        st["raw"], st["target"] = _raw(seed, c["N"], c["H"], c["W"], _mean_spp(seed))
    else:
        st["x1"], st["x2"], st["w"], st["bias"], st["dout"] = _conv_inputs(c, seed)
        N, H, W, Cin, Cout = c["N"], c["H"], c["W"], c["C1"] + c["C2"], c["Cout"]
        if kind == "conv_fwd":
            st["out"] = new(N, H, W, Cout)
        else:
            st["wt"] = st["w"].permute(2, 1, 0).contiguous()
            st["out"] = (new(N, H, W, Cin, dtype=torch.bfloat16), new(Cout, 9, Cin))
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    c, ctx, kind = st["case"], st["ctx"], st["kind"]
    if kind == "convolve":
        return ctx.convolve(st["img"], st["kernel"], out=st["out"])
    if kind == "blur":
        return ctx.gaussian_blur(st["img"], c["size"], c["sigma"], out=st["out"])
    if kind == "bloom":
        return ctx.bloom(st["img"], c["size"], c["sigma"], c["threshold"], out=st["out"])
    if kind == "aov":
        return ctx.aov(c["W"], c["H"], 700.0, 1500.0, camera=st["camera"], out=st["out"])
    if kind == "render":
        return ctx.render_pt(c["W"], c["H"], c["spp"], c["depth"], seed=st["seed"], camera=st["camera"], out=st["out"])
    if kind == "batch":
        return ctx.render_batch(st["jobs"], c["depth"], out=st["out"])
    if kind == "denoise":
        return ctx.denoise(*st["passes"], c["spp"], out=st["out"])
    if kind == "train":
        loss = ctx.dn_train_step(st["raw"], st["target"], lr=LR)
        return {"loss": loss, "params": ctx.dn_get_params(), "grads": ctx.dn_get_grads()}
    if kind == "conv_fwd":
        return ctx.conv3x3_fwd(st["x1"], st["w"], c["Cout"], x2=st["x2"], up1=bool(c["up"]), bias=st["bias"],
                               relu=True, out=st["out"])
    din, dw = st["out"]
    ctx.conv3x3_dgrad(st["dout"], st["wt"], st["x1"], x2=st["x2"], up1=bool(c["up"]), mask_relu=True, out=din)
    ctx.conv3x3_wgrad(st["dout"], st["x1"], x2=st["x2"], up1=bool(c["up"]), out=dw)
    return {"din": din, "dw": dw}


def _network_flops(P, train):
    f = 0
    for s1, up, s2, out, cop, co, ci, relu in LAYERS:
        level = TENSORS[out][1] if out else 0
        f += 2 * 9 * ci * co * (P >> (2 * level)) * (3 if train else 1)
    return f


def work(case):
    c = case
    kind = c["kind"]
    px = c.get("W", 0) * c.get("H", 0)
    if kind == "convolve":
        return {"bytes": 24 * px, "flops": 6 * c["k"] ** 2 * px}
    if kind in ("blur", "bloom"):
        return {"bytes": 24 * px, "flops": 12 * c["size"] * px}
    tris = {"cornell": 36, "mixed": 500, "icosphere": 20 * 4 ** c.get("subdiv", 0)}.get(c.get("scene"), 0)
    # a triangle's record (48 B) once, the image once; about 40 operations per
    # primary ray for its camera ray and one intersection, about 2,900 FP32
    # operations of shading per sample
    if kind == "aov":
        return {"bytes": 48 * tris + 36 * px, "flops": 40 * px}
    if kind == "render":
        return {"bytes": 48 * tris + 12 * px, "flops": 2900 * px * c["spp"]}
    if kind == "batch":
        b = f = 0
        for k in range(c["scenes"]):
            s = 0.5 + 0.5 * (k % 3)
            p = int(c["W"] * s) * int(c["H"] * s)
            b += 12 * p + 48 * max(64, int(c["tris"] * (k + 1) ** 2 / c["scenes"] ** 2))
            f += 2900 * p * (c["spp"] + k % 3)
        return {"bytes": b, "flops": f}
    if kind == "denoise":
        return {"bytes": 60 * px + 4 * _layout()[1], "flops": _network_flops(px, False)}
    if kind == "train":
        return {"bytes": 56 * px * c["N"] + 24 * _layout()[1], "flops": _network_flops(px * c["N"], True)}
    P, Cin, Cout = c["N"] * px, c["C1"] + c["C2"], c["Cout"]
    src = (c["C1"] // (4 if c["up"] else 1) + c["C2"]) * P * 2
    f = 2 * 9 * Cin * Cout * P
    if kind == "conv_fwd":
        return {"bytes": src + 18 * Cin * Cout + 4 * P * Cout, "flops": f}
    return {"bytes": src + 2 * P * (Cin + Cout) + 54 * Cin * Cout, "flops": 2 * f}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _reflected(img, dy, dx):
    """The image moved by (dy, dx) under the compositor's edge rule: an index
    past an edge is mirrored (index == size maps to itself, so a column past
    the last reads the next row's first pixel) and a pixel past the image
    reads zero."""
    H, W = img.shape[:2]
    r = (torch.arange(H, device=img.device) + dy).abs()
    q = (torch.arange(W, device=img.device) + dx).abs()
    q = torch.where(q >= W, 2 * W - q, q)
    r = torch.where(r >= H, 2 * H - r, r)
    idx = r[:, None] * W + q[None, :]
    ok = (idx >= 0) & (idx < H * W)
    v = img.reshape(H * W, 3)[idx.clamp(0, H * W - 1).reshape(-1)].reshape(H, W, 3)
    return v * ok[..., None]


def _filter(img, k):
    out = torch.zeros_like(img)
    for i in range(k.shape[0]):
        for j in range(k.shape[1]):
            out += _reflected(img, i - k.shape[0] // 2, j - k.shape[1] // 2) * float(k[i, j])
    return out


def _gauss(img, size, sigma):
    x = np.arange(size, dtype=np.float64) - (size >> 1)
    g = np.exp(-x * x / (2.0 * sigma * sigma))
    g /= g.sum()
    return _filter(_filter(img, g[None, :]), g[:, None])


def _network(params, raw):
    """The U-Net's filter logits [N][H][W][25] for raw [N][H][W][11], FP64."""
    F = torch.nn.functional
    rows, _ = _layout()
    sane = raw[..., :3].clamp(0.0, 65504.0)
    x = torch.cat([torch.log1p(sane), raw[..., 3:10], raw[..., 10:11].clamp_min(1.0).log2() / 16.0], -1)
    act = {"X": F.pad(x, (0, 5)).permute(0, 3, 1, 2)}
    for (s1, up, s2, out, cop, co, ci, relu), (cip, w_off, b_off) in zip(LAYERS, rows):
        w = params[w_off:w_off + cop * 9 * cip].reshape(cop, 3, 3, cip).permute(0, 3, 1, 2)
        b = params[b_off:b_off + cop]
        if s1 in POOLED:
            act[s1] = F.avg_pool2d(act[POOLED[s1]], 2)
        h = act[s1]
        if up:
            h = h.repeat_interleave(2, 2).repeat_interleave(2, 3)
        if s2:
            h = torch.cat([h, act[s2]], 1)
        z = F.conv2d(h, w, b, padding=1)
        if out is None:
            return z.permute(0, 2, 3, 1)[..., :TAPS]
        act[out] = F.relu(z) if relu else z


def _filtered(logits, rad):
    """The predicted 5 x 5 filters applied to the radiance, taps clamped to the frame."""
    H, W = rad.shape[1:3]
    w = torch.softmax(logits, -1)
    out = torch.zeros_like(rad)
    ys, xs = torch.arange(H, device=rad.device), torch.arange(W, device=rad.device)
    for k in range(TAPS):
        y = (ys + k // 5 - 2).clamp(0, H - 1)
        x = (xs + k % 5 - 2).clamp(0, W - 1)
        out = out + w[..., k:k + 1] * rad[:, y][:, :, x]
    return out


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind in ("convolve", "blur", "bloom"):
        img = _image(_gen(seed), c["H"], c["W"]).double()
        if kind == "convolve":
            return _filter(img, _kernel(c, seed).astype(np.float64))
        if kind == "blur":
            return _gauss(img, c["size"], c["sigma"])
        luma = 0.2126 * img[..., 0] + 0.7152 * img[..., 1] + 0.0722 * img[..., 2]
        return img + _gauss(img * (luma > c["threshold"])[..., None], c["size"], c["sigma"])
    if kind == "denoise":
        H, W = c["H"], c["W"]
        raw, _ = _raw(seed, 1, H, W, c["spp"])
        pad = torch.zeros((1, (H + 15) // 16 * 16, (W + 15) // 16 * 16, 11), device="cuda", dtype=torch.float64)
        pad[:, :H, :W] = raw.double()
        with torch.no_grad():
            logits = _network(torch.from_numpy(_params(seed)).cuda().double(), pad)[:, :H, :W]
            return _filtered(logits, pad[:, :H, :W, :3].clamp(0.0, 65504.0))[0]
    if kind == "train":
        raw, tgt = _raw(seed, c["N"], c["H"], c["W"], _mean_spp(seed))
        p = torch.from_numpy(_params(seed)).cuda().double().requires_grad_(True)
        total, count = 0.0, c["N"] * c["H"] * c["W"] * 3
        for n in range(0, c["N"], 4):  # in parts: the sum of their gradients is the minibatch's
            x = raw[n:n + 4].double()
            o = _filtered(_network(p, x), x[..., :3].clamp(0.0, 65504.0))
            d = o - tgt[n:n + 4].double().clamp(0.0, 65504.0)
            loss = (d * d / (o.detach() ** 2 + REL_EPS)).sum() / count
            loss.backward()
            total += float(loss)
        # Adam with the moments of the resumed run (its divisor held constant in FP32: beta powers at this step)
        g, t = p.grad, STEP + 1
        m, v = 0.1 * g, 0.999 * SECOND_MOMENT + 0.001 * g * g
        q = p.detach() - LR * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
        return {"loss": total, "params": q, "grads": g}
    if kind in ("conv_fwd", "conv_bwd"):
        F = torch.nn.functional
        x1, x2, w, bias, dout = _conv_inputs(c, seed)
        x = x1.double().permute(0, 3, 1, 2)
        if c["up"]:
            x = x.repeat_interleave(2, 2).repeat_interleave(2, 3)
        if x2 is not None:
            x = torch.cat([x, x2.double().permute(0, 3, 1, 2)], 1)
        Cin, Cout = c["C1"] + c["C2"], c["Cout"]
        k = w.double().reshape(Cout, 3, 3, Cin).permute(0, 3, 1, 2)
        if kind == "conv_fwd":
            return F.relu(F.conv2d(x, k, bias.double(), padding=1)).permute(0, 2, 3, 1).contiguous()
        x, k = x.contiguous().requires_grad_(True), k.contiguous().requires_grad_(True)
        F.conv2d(x, k, padding=1).backward(dout.double().permute(0, 3, 1, 2).contiguous())
        din = torch.where(x.detach() > 0, x.grad, torch.zeros_like(x.grad)).permute(0, 2, 3, 1).contiguous()
        return {"din": din, "dw": k.grad.permute(0, 2, 3, 1).reshape(Cout, 9, Cin).contiguous()}
    return None  # Monte Carlo images and discrete hits: the start's own bits say more
