"""The framework's work as a user's program asks for it, one case per call pattern.

Kinds and what they stand for (sizes: the headline frame, the tracer, serving
and 1024^3 workloads of bench.py, the tests, and odd sizes between them):

* ``network`` -- predict_features on device tensors: the radiance predictor
  called on feature sets that a program holds (a handful up to a frame's worth
  of hits), in each arithmetic it offers, grey or coloured albedo.
* ``frame`` -- VolumeRender.Render of MRPNN frames of a resident volume under a
  fixed light, into a device buffer: a turntable, a thumbnail, a full frame.
* ``trace`` -- VolumeRender.Render of path-traced frames (the renderer's ground
  truth), the light's NEE grid already baked.
* ``relight`` -- the sun moves from frame to frame: each Render rebuilds the
  transmittance levels (MRPNN) or bakes the NEE grid (path tracer) first.
* ``animate`` -- a new density grid per frame (a simulation's next step, held on
  the device): set_data, Update, one MRPNN frame.
* ``phase`` -- the phase function changes: UpdateHGLut for another asymmetry,
  and the table read back (GetHGLut's host copy).
* ``tiles`` -- GatherData, the input of the tile network, to host memory.
"""
import math
import os
import struct

import numpy as np
import torch

import mrpnn_b200 as M

FOV = 45.0
CAMERA = (0.75, 0.75, 0.75)
PRECISION = {"fp32": M.FP32, "bf16": M.BF16, "fp8": M.FP8}
FLOPS_PER_HIT = 97072        # one evaluation of the network, grey albedo
FLOPS_PER_TAIL = 2 * (1200 + 96 + 24 + 16384 + 8192 + 2048 + 512 + 12 * 256 + 16)   # a further albedo channel's share
HIT_SHARE = 0.49             # pixels of the cloud's frames that hit it


def listed():
    return [
        # a frame's worth of feature sets through the drop-in network
        dict(name="network_fp32_200k", kind="network", n=200003, precision="fp32", coloured=False),
        # coloured albedo: the network's tail runs once per channel
        dict(name="network_bf16_100k_rgb", kind="network", n=100001, precision="bf16", coloured=True),
        # a few probes: launch and latency bound
        dict(name="network_fp8_300", kind="network", n=300, precision="fp8", coloured=False),
        # the headline frame, drop-in precision
        dict(name="frame_fp32_1024", kind="frame", res=512, width=1024, height=1024, launches=1, precision="fp32",
             coloured=False),
        # a full-HD frame in the fast form
        dict(name="frame_bf16_1080p", kind="frame", res=512, width=1920, height=1080, launches=1, precision="bf16",
             coloured=False),
        # a thumbnail of a small volume, four launches averaged
        dict(name="frame_fp8_thumb", kind="frame", res=100, width=163, height=97, launches=4, precision="fp8",
             coloured=False),
        # the tracer benchmark: 256^2, 16 samples per pixel, NEE from the default 768^3 grid
        dict(name="trace_256_spp16", kind="trace", res=128, size=256, spp=16, bounces=256, bake=768, texture=False),
        # a sun sweep over a resident cloud
        dict(name="relight_bf16_512", kind="relight", res=256, size=512, suns=4, tracer=False, precision="bf16",
             bake=0),
        # the same for the path tracer: every sun bakes its own default-size NEE grid
        dict(name="relight_trace_768", kind="relight", res=128, size=96, suns=2, tracer=True, precision="fp32",
             bake=768),
        # the next step of a simulation: ingest, pyramid, frame
        dict(name="animate_bf16_512", kind="animate", res=512, size=512, storage="fp32", precision="bf16"),
        # an asymmetry slider: two tables
        dict(name="phase_2", kind="phase", tables=2),
        # tile-network inputs of a 1024 x 1024 view
        dict(name="tiles_128", kind="tiles", res=256, width=128, height=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["network", "network", "frame", "frame", "trace", "relight", "relight", "animate", "phase",
                       "tiles"])
    prec = rng.choice(["fp32", "bf16", "fp8"])
    if kind == "network":
        return dict(kind=kind, n=_log_int(rng, 33, 262144), precision=prec, coloured=rng.random() < 0.3)
    if kind == "frame":
        return dict(kind=kind, res=rng.choice([64, 100, 128, 200, 256, 300, 512]), width=_log_int(rng, 64, 1920),
                    height=_log_int(rng, 48, 1080), launches=rng.choice([1, 1, 1, 2, 4]), precision=prec,
                    coloured=rng.random() < 0.2)
    if kind == "trace":
        return dict(kind=kind, res=rng.choice([48, 100, 128, 256]), size=_log_int(rng, 48, 320),
                    spp=_log_int(rng, 1, 16), bounces=rng.choice([1, 16, 256]), bake=_log_int(rng, 96, 768),
                    texture=rng.random() < 0.4)
    if kind == "relight":
        tracer = rng.random() < 0.5
        return dict(kind=kind, res=rng.choice([64, 100, 128, 256]), size=_log_int(rng, 64, 512),
                    suns=rng.choice([2, 3, 4]), tracer=tracer, precision=prec,
                    bake=_log_int(rng, 96, 512) if tracer else 0)
    if kind == "animate":
        return dict(kind=kind, res=_log_int(rng, 64, 512), size=_log_int(rng, 96, 768),
                    storage=rng.choice(["fp32", "fp16"]), precision=prec)
    if kind == "phase":
        return dict(kind=kind, tables=rng.choice([2, 3]), spread=round(rng.uniform(0.02, 0.2), 3))
    return dict(kind=kind, res=rng.choice([64, 100, 128, 256, 512]), width=_log_int(rng, 8, 160),
                height=_log_int(rng, 8, 128))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _unit(v):
    v = np.asarray(v, np.float32)
    return (v / np.float32(np.sqrt(np.float32(np.dot(v, v))))).astype(np.float32)


def _suns(seed, n):
    """n unit directions from above, the benchmark's sun among their neighbours."""
    r = np.random.default_rng(seed)
    return [_unit(np.array([0.3, 0.8, 0.5]) + r.uniform(-0.25, 0.25, 3)) for _ in range(n)]


def _camera():
    ori, up, right = M.camera_frame(CAMERA)
    s = np.float32(np.tan(np.deg2rad(FOV) / 2))
    return ori, (up * s).astype(np.float32), (right * s).astype(np.float32)


def _albedo(coloured):
    return (0.99, 0.97, 0.93) if coloured else 0.99


def _volume(case, seed, storage="fp32"):
    vol = M.VolumeRender(case["res"], storage=storage)
    vol.SetScatterRate(_albedo(case.get("coloured", False)))
    vol.SetSky(0.05)
    vol.SetPrecision(PRECISION[case.get("precision", "fp32")])
    return vol


def _cloud_volume(case, seed):
    vol = _volume(case, seed)
    vol.generate_fbm(seed, 6.0 if case["res"] >= 256 else 4.0)
    vol.Update()
    return vol


def _cloud_grid(res, seed):
    """A density grid as a simulation would hand it over: five octaves of
    smooth noise inside a ball, float32 [res, res, res] on the device."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    d = torch.zeros((1, 1, res, res, res), device="cuda")
    amp = 0.5
    for o in range(5):
        n = 6 << o
        d += amp * torch.nn.functional.interpolate(torch.rand((1, 1, n, n, n), generator=gen, device="cuda"),
                                                   size=(res,) * 3, mode="trilinear", align_corners=False)
        amp *= 0.5
    x = (torch.arange(res, device="cuda") + 0.5) / res - 0.5
    r = (x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2).sqrt()
    return (d[0, 0] * ((0.4 - r) / 0.08).clamp(0, 1)).clamp_(0, 1).contiguous()


def _features(n, seed):
    """Feature sets as the gather makes them: log(1 + alpha d / 64) of a
    density that varies slowly over the stencil, transmittances in (0, 1) and
    log(1 + HG factors) with their forward peak."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def u(*shape):
        return torch.rand(shape, generator=gen, device="cuda")

    dens = torch.log1p((u(n, 1) * 0.9 * (0.4 + 0.6 * u(n, 192)) - 0.1).clamp_(min=0.0))
    tr = (u(n, 1) * (0.5 + 0.5 * u(n, 192))).clamp_(0.0, 1.0)
    hg = torch.log1p(0.02 + 2.0 * u(n, 192) ** 8)
    return torch.cat([dens, tr, hg], 1), u(n) * math.pi


def _gs(case, seed):
    r = np.random.default_rng(seed)
    return [float(np.float32(0.85 + case.get("spread", 0.05) * (k + float(r.uniform(0.0, 0.5))) / case["tables"] - 0.05))
            for k in range(case["tables"])]


def prepare(case, seed):
    M.init()
    kind = case["kind"]
    s = {"case": case, "seed": seed}
    if kind == "network":
        s["feat"], s["gamma"] = _features(case["n"], seed)
        s["albedo"] = (0.99, 0.97, 0.93) if case["coloured"] else (0.99, 0.99, 0.99)
        s["out"] = torch.empty((case["n"], 3), device="cuda")
        return s
    s["ori"], s["up"], s["right"] = _camera()
    if kind == "frame":
        s["vol"] = _cloud_volume(case, seed)
        s["suns"] = _suns(seed, 1)
        s["vol"].UpdateHGLut(0.857)
        s["vol"].Update_TR(s["suns"][0], 64.0)
        s["out"] = torch.empty((case["height"], case["width"], 4), device="cuda")
    elif kind == "trace":
        s["vol"] = _cloud_volume(case, seed)
        s["suns"] = _suns(seed, 1)
        s["vol"].SetBakeResolution(case["bake"])
        s["vol"].SetTracerFilter(case["texture"])
        s["vol"].Update_CachedTR(s["suns"][0], 64.0)
        s["out"] = torch.empty((case["size"], case["size"], 4), device="cuda")
    elif kind == "relight":
        s["vol"] = _cloud_volume(case, seed)
        s["suns"] = _suns(seed, case["suns"])
        if case["tracer"]:
            s["vol"].SetBakeResolution(case["bake"])
        else:
            s["vol"].UpdateHGLut(0.857)
        s["out"] = [torch.empty((case["size"], case["size"], 4), device="cuda") for _ in s["suns"]]
    elif kind == "animate":
        s["vol"] = _volume(case, seed, case["storage"])
        s["suns"] = _suns(seed, 1)
        s["grid"] = _cloud_grid(case["res"], seed)
        s["vol"].UpdateHGLut(0.857)
        s["out"] = torch.empty((case["size"], case["size"], 4), device="cuda")
    elif kind == "phase":
        s["vol"] = M.VolumeRender(32)
        s["vol"].SetSeed(seed)
        s["gs"] = _gs(case, seed)
    else:   # tiles
        s["vol"] = _cloud_volume(case, seed)
        s["suns"] = _suns(seed, 1)
        s["vol"].UpdateHGLut(0.857)
        s["vol"].Update_TR(s["suns"][0], 64.0)
    return s


def run(s):
    case, kind, vol = s["case"], s["case"]["kind"], s.get("vol")
    if kind == "network":
        return M.predict_features(s["feat"], s["gamma"], 0.857, s["albedo"], PRECISION[case["precision"]],
                                  out=s["out"])
    if kind == "frame":
        return vol.Render((case["width"], case["height"]), s["ori"], s["up"], s["right"], s["suns"][0], vol.MRPNN,
                          0.857, 64.0, sampleNum=case["launches"], seed=s["seed"], out=s["out"])
    if kind == "trace":
        return vol.Render(case["size"], s["ori"], s["up"], s["right"], s["suns"][0], vol.PT, 0.857, 64.0,
                          multiScatter=case["bounces"], sampleNum=1, spp=case["spp"], seed=s["seed"], out=s["out"])
    if kind == "relight":
        for sun, out in zip(s["suns"], s["out"]):
            vol.Render(case["size"], s["ori"], s["up"], s["right"], sun, vol.PT if case["tracer"] else vol.MRPNN, 0.857,
                       64.0, multiScatter=64, sampleNum=1, spp=4, seed=s["seed"], out=out)
        return s["out"]
    if kind == "animate":
        vol.set_data(s["grid"])
        vol.Update()
        return vol.Render(case["size"], s["ori"], s["up"], s["right"], s["suns"][0], vol.MRPNN, 0.857, 64.0,
                          sampleNum=1, seed=s["seed"], out=s["out"])
    if kind == "phase":
        tables = []
        for g in s["gs"]:
            vol.UpdateHGLut(g)
            tables.append(vol.read(M.api.RES_LUT))
        return tables
    return vol.GatherData((case["width"], case["height"]), s["ori"], s["up"], s["right"], s["suns"][0], 64.0, 0.857,
                          seed=s["seed"])


def work(case):
    """Inputs read once, outputs written once; the arithmetic of the network
    (frames: for the pixels that hit), the rest of a path not counted."""
    kind = case["kind"]
    if kind == "network":
        tails = 2 * FLOPS_PER_TAIL if case["coloured"] else 0
        return {"bytes": case["n"] * (576 + 1 + 3) * 4, "flops": case["n"] * (FLOPS_PER_HIT + tails)}
    if kind == "phase":   # 1024 samples of the phase function per entry, about 30 operations each
        return {"bytes": case["tables"] * 512 * 512 * 4, "flops": case["tables"] * 512 * 512 * 1024 * 30}
    grid = case["res"] ** 3 * 4
    if kind == "frame":
        px = case["width"] * case["height"]
        return {"bytes": grid + px * 16, "flops": case["launches"] * px * HIT_SHARE * FLOPS_PER_HIT}
    if kind == "trace":   # the grid and the baked grid, the image
        return {"bytes": grid + case["bake"] ** 3 * 4 + case["size"] ** 2 * 16, "flops": 0}
    if kind == "relight":
        px = case["size"] ** 2
        if case["tracer"]:   # each sun's grid is written once and read once
            return {"bytes": case["suns"] * (grid + 2 * case["bake"] ** 3 * 4 + px * 16), "flops": 0}
        return {"bytes": case["suns"] * (grid + 128 ** 3 * 4 + px * 16),
                "flops": case["suns"] * px * HIT_SHARE * FLOPS_PER_HIT}
    if kind == "animate":
        px = case["size"] ** 2
        return {"bytes": 2 * grid + 256 ** 3 * 4 + px * 16, "flops": px * HIT_SHARE * FLOPS_PER_HIT}
    return {"bytes": grid + case["width"] * case["height"] * 773 * 4, "flops": 0}


# ---------------------------------------------------------------------------
# values in 64 bits.  Network outputs and phase tables have them.  A frame is
# one draw of jittered rays and random frames (or of random paths) through
# decisions taken in float, so its pixels have no value of their own.
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "network":
        feat, gamma = _features(case["n"], seed)
        sr = (0.99, 0.97, 0.93) if case["coloured"] else (0.99, 0.99, 0.99)
        net = _Network64()
        return torch.cat([net(feat[i:i + 32768].double(), gamma[i:i + 32768].double(), 0.857, sr)
                          for i in range(0, case["n"], 32768)])
    if case["kind"] == "phase":
        return [_phase_table64(g, seed).cpu().numpy().ravel() for g in _gs(case, seed)]
    return None


def _model():
    path = os.path.join(os.path.dirname(os.path.abspath(M.__file__)), "data", "mrpnn_model.bin")
    with open(path, "rb") as f:
        data = f.read()
    count, off, out = struct.unpack_from("<I", data, 8)[0], 12, {}
    for _ in range(count):
        ln = struct.unpack_from("<H", data, off)[0]
        name = data[off + 2:off + 2 + ln].decode()
        n = struct.unpack_from("<I", data, off + 2 + ln)[0]
        off += 6 + ln
        out[name] = torch.from_numpy(np.frombuffer(data, "<f4", n, off).astype(np.float64)).cuda()
        off += 4 * n
    return out


class _Network64:
    """The SE-gated network: eight main blocks and four light-ray blocks of
    gated branch layers, then the gated tail per albedo value."""
    MAIN = [(0, 8), (8, 8), (16, 16), (32, 16), (48, 16), (64, 32), (96, 32), (128, 32)]

    def __init__(self):
        self.t = _model()

    def lin(self, x, name):
        b = self.t[name + "B"]
        return torch.relu(x @ self.t[name + "W"].view(b.numel(), -1).T + b)

    def chain(self, X, gg, blocks, gate, layer):
        prev, avgs, maxs = None, [], []
        for k, (at, w) in enumerate(blocks):
            sl = X[:, :, at:at + w]
            avg, mx = sl.mean(-1), sl.amax(-1)
            avgs.append(avg)
            maxs.append(mx)
            h = torch.relu(torch.cat([avg, mx, gg], 1) @ self.t[f"{gate}{k}1W"].view(8, 8).T)
            a = torch.sigmoid(h @ self.t[f"{gate}{k}2W"].view(3, 8).T)
            x = sl * a[:, :, None]
            if prev is not None:
                x = x + torch.stack(prev, 1)
            o = [self.lin(x[:, c], layer.format(("", "_Tr", "_Hg")[c], f"{k}1")) for c in range(3)]
            widen = k + 1 < len(blocks) and blocks[k + 1][1] > w
            prev = [torch.cat([o[c], sl[:, c]], 1) if widen else o[c] + sl[:, c] for c in range(3)]
        last = f"{len(blocks)}1"
        return [self.lin(prev[c], layer.format(("", "_Tr", "_Hg")[c], last)) for c in range(3)], avgs, maxs

    def __call__(self, feat, gamma, g, sr):
        n = feat.shape[0]
        X = feat.view(n, 3, 192)
        g = float(np.float32(g))
        gg = torch.stack([torch.full_like(gamma, g), gamma], 1)
        main, a1, m1 = self.chain(X, gg, self.MAIN, "LSE", "L{}{}")
        di, a2, m2 = self.chain(X, gg, [(160 + 8 * k, 8) for k in range(4)], "LDSE", "LD{}{}")
        pool = torch.cat(a1 + a2 + m1 + m2 + [gg], 1)
        out = []
        for r in sr:
            s4 = float(np.float32(r)) ** 4
            p = torch.cat([pool, torch.full_like(gamma, s4)[:, None]], 1)
            a = torch.sigmoid(torch.relu(p @ self.t["LSEFin1W"].view(16, 75).T) @ self.t["LSEFin2W"].view(6, 16).T)
            x = [v * a[:, k:k + 1] for k, v in enumerate(main + di)]
            x = torch.cat(x + [self.lin(p[:, 72:75], "LGGS")], 1)
            for name in ("LC0", "LC1", "LC2", "LX"):
                x = self.lin(x, name)
            for k in range(0, 12, 2):
                x = x + self.lin(self.lin(x, f"LX{k}"), f"LX{k + 1}")
            y = torch.relu(x @ self.t["LX12W"] + self.t["LX12B"])
            out.append(torch.expm1(y) * s4)
        return torch.stack(out, 1)


def _philox_first(ids, k1, kind):
    """First word of Philox-4x32-10 at counter (0, 0, 0, kind), key (ids, k1)."""
    m = 0xFFFFFFFF
    z = torch.zeros_like(ids)
    c0, c1, c2, c3 = z, z, z, z + kind
    a, b = ids.clone(), z + k1
    for r in range(10):
        if r:
            a, b = (a + 0x9E3779B9) & m, (b + 0xBB67AE85) & m

        def wide(mul, c):   # 32 x 32 -> (high, low) within int64
            lo16 = mul * (c & 0xFFFF)
            hi16 = mul * (c >> 16) + (lo16 >> 16)
            return hi16 >> 16, ((hi16 & 0xFFFF) << 16) | (lo16 & 0xFFFF)

        h0, l0 = wide(0xD2511F53, c0)
        h1, l1 = wide(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ a, l1, h0 ^ c3 ^ b, l0
    return c0


def _radical_inverse(base, perm, count):
    """Scrambled radical inverse of 0..count-1: permuted digits, then the
    permuted zeros that follow them for good."""
    out = []
    for a in range(count):
        v, scale = 0.0, 1.0
        while a:
            scale /= base
            v = v * base + perm[a % base]
            a //= base
        out.append(min(scale * (v + perm[0] / (base - 1)), 0.99999994))
    return torch.tensor(out, dtype=torch.float64, device="cuda")


def _phase_table64(g, seed):
    """The phase function averaged over a cone around a direction, 512 cone
    angles x 512 cosines: one-sample mixture of solid-angle and phase sampling
    with 1024 shifted Halton points per entry."""
    n, samples = 512, 1024
    g = float(np.float32(g))
    digits = _model()["HALTON_PERMS"].tolist()
    table = {b: _radical_inverse(b, digits[o:o + b], samples) for b, o in ((2, 0), (3, 2), (5, 5), (11, 17))}
    ids = torch.arange(n * n, device="cuda", dtype=torch.int64)
    word = _philox_first(ids, (seed ^ 0x9E3779B9) & 0xFFFFFFFF, 1)
    shift = (((word >> 9) << 1) | 1).double() * 2.0 ** -24
    cosine = ((ids % n).double() + 0.5) / n * 2 - 1
    radius = torch.tan(((ids // n).double() + 0.5) / n * (math.pi / 3))
    sine = (1 - cosine ** 2).clamp(min=0).sqrt()
    p = radius ** 2 - 1 + cosine ** 2
    w = p.clamp(min=0).sqrt()
    toward = cosine if g > 0 else -cosine
    d0, d1 = (toward - w).clamp(min=0) / radius, (toward + w) / radius
    mix = torch.where(p > 0, torch.where(d1 > d0, d1 ** 3 - d0 ** 3, torch.zeros_like(p)), torch.zeros_like(p))
    mix = mix.clamp(1e-8, 1.0)
    a = abs(g)
    a = 0.0 if a < 0.6 else (a - 0.6) * 9 if a < 0.7 else ((a - 0.7) / 0.3) ** 0.05 * 0.1 + 0.9
    mix = 1 - 1 / (1 + a * mix / (1 - a))
    out = torch.empty(n * n, dtype=torch.float64, device="cuda")
    for i in range(0, n * n, 8192):
        c, s, r, t = (v[i:i + 8192, None] for v in (cosine, sine, radius, shift))
        x, y, z, pick = ((table[b][None] + t) % 1.0 for b in (2, 3, 5, 11))
        # phase sampling: a direction l around the view axis
        q = (1 - g * g) / (1 - g + 2 * g * x)
        cl = (1 + g * g - q * q) / (2 * g)
        sl = (1 - cl ** 2).clamp(min=0).sqrt()
        sd = c * cl - s * sl * torch.sin(2 * math.pi * y)
        pp = r ** 2 - 1 + sd ** 2
        ww = pp.clamp(min=0).sqrt()
        e0, e1 = (sd - ww).clamp(min=0) / r, (sd + ww) / r
        h1 = torch.where(pp > 0, ((e1 ** 3 - e0 ** 3) / 4).clamp(min=0), torch.zeros_like(pp))
        # solid-angle sampling: a point of the ball of that radius around the direction
        cp = 2 * y - 1
        sp = (1 - cp ** 2).clamp(min=0).sqrt()
        rr = r * z ** (1 / 3)
        px, py, pz = rr * sp * torch.cos(2 * math.pi * x) + c, rr * sp * torch.sin(2 * math.pi * x) + s, rr * cp
        h2 = (1 - g * g) / (1 + g * g - 2 * g * px / (px ** 2 + py ** 2 + pz ** 2).sqrt()) ** 1.5 / 4
        out[i:i + 8192] = torch.where(pick < mix[i:i + 8192, None], h1, h2).mean(1)
    return out
