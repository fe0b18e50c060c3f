"""Timed workloads of the cloud renderer, through its public entry points.

A case is a dict of plain values. `prepare` makes what a program has in hand
before the call (volume, network, trainer, device buffers), `run` is one call
or one frame, `work` the bytes and operations it cannot do without, and
`exact` the result in 64-bit arithmetic where the outputs have one (a path
tracer's image is an estimate over a fixed random stream and has none).

Kinds:
  frame        one neural (MRPNN) frame: trace, descriptor gather, network
  batch        one frame of a batch of views over several clouds (CUDA graph)
  track        offline delta tracking of the solid sphere
  interactive  one progressive delta-tracking frame with the histogram denoiser
  scene        a new cloud: density upload, pyramids, and the light and phase
               tables and descriptors of two media (training-data set-up)
  labels       multiple-scattering training labels
  train        loss and gradient of a training batch
  predict      the radiance-predictor network on a table of descriptors
"""
import ctypes as C
import math

import numpy as np
import torch

import internship_b200 as mr
from internship_b200 import _lib, scenes
from internship_b200.train import Trainer

PRECISION = {"fp32": _lib.PREC_FP32, "bf16": _lib.PREC_BF16, "fp8": _lib.PREC_FP8}
SAMPLER = {"exact": _lib.SAMPLER_EXACT, "texture": _lib.SAMPLER_TEXTURE}
NETWORK_FLOP = 97072  # per row: 48,536 multiply-adds, one albedo channel
IN_VIEW = 0.155       # share of a frame's pixels that meet the cloud at the camera used here
ALPHA, G, ALBEDO = 64.0, 0.857, 0.99


def listed():
    return [
        # a thumbnail or viewport preview through the Python API, image on the host
        {"name": "preview_160x90_fp32", "kind": "frame", "res": 64, "width": 160, "height": 90, "precision": "fp32",
         "sampler": "exact", "host": True},
        # the benchmark's headline frame: 1080p, 512^3 cloud, fp32 network, exact sampler
        {"name": "frame_1080p_fp32", "kind": "frame", "res": 512, "width": 1920, "height": 1080, "precision": "fp32",
         "sampler": "exact", "host": False},
        # the fast form of a frame, at a size that no tile divides
        {"name": "frame_1283x719_bf16", "kind": "frame", "res": 256, "width": 1283, "height": 719, "precision": "bf16",
         "sampler": "texture", "host": False},
        # batched serving: clouds of uneven resolution seen at uneven sizes
        {"name": "batch_8_views_bf16", "kind": "batch", "views": 8, "max_side": 1024, "precision": "bf16",
         "sampler": "texture"},
        # reference delta tracking: 128^3 sphere, 256 x 256, 64 samples per pixel
        {"name": "track_256_64spp", "kind": "track", "res": 128, "side": 256, "spp": 64},
        # the interactive viewer at full HD after eight accumulated frames
        {"name": "interactive_1080p", "kind": "interactive", "res": 256, "width": 1920, "height": 1080, "history": 8},
        # set-up of a training scene
        {"name": "scene_512", "kind": "scene", "res": 512, "points": 16384},
        # training labels of one scene
        {"name": "labels_4096_256spp", "kind": "labels", "res": 256, "points": 4096, "spp": 256},
        # training steps: the default precision on an uneven last batch, BF16 at the default batch size
        {"name": "train_20011_fp32", "kind": "train", "rows": 20011, "precision": "fp32"},
        {"name": "train_65536_bf16", "kind": "train", "rows": 65536, "precision": "bf16"},
        # held-out evaluation of a training run, and a handful of probe points
        {"name": "predict_262144_fp32", "kind": "predict", "rows": 262144, "precision": "fp32", "channels": 1},
        {"name": "predict_1000_bf16", "kind": "predict", "rows": 1000, "precision": "bf16", "channels": 1},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame", "batch", "track", "interactive", "scene", "labels", "train", "train", "predict",
                       "predict"])
    res = rng.choice([64, 128, 256, 512])
    if kind == "frame":
        host = rng.random() < 0.3
        width = log_int(96, 640 if host else 1920)
        return {"kind": kind, "res": res, "width": width, "height": max(16, min(1080, int(width * rng.uniform(0.5, 1.0)))),
                "precision": rng.choice(["fp32", "bf16", "fp8"]),
                "sampler": "exact" if host else rng.choice(["exact", "texture"]), "host": host}
    if kind == "batch":
        return {"kind": kind, "views": rng.randint(2, 8), "max_side": log_int(256, 1024),
                "precision": rng.choice(["fp32", "bf16"]), "sampler": rng.choice(["exact", "texture"])}
    if kind == "track":
        return {"kind": kind, "res": rng.choice([64, 96, 128]), "side": log_int(48, 256), "spp": log_int(1, 64)}
    if kind == "interactive":
        width = log_int(160, 1920)
        return {"kind": kind, "res": res, "width": width, "height": max(90, min(1080, int(width * rng.uniform(0.5, 1.0)))),
                "history": rng.randint(1, 12)}
    if kind == "scene":
        return {"kind": kind, "res": rng.choice([64, 100, 128, 200, 256, 400, 512]), "points": log_int(1000, 16384)}
    if kind == "labels":
        return {"kind": kind, "res": rng.choice([64, 128, 256]), "points": log_int(100, 4096), "spp": log_int(16, 256)}
    if kind == "train":
        return {"kind": kind, "rows": log_int(500, 65536), "precision": rng.choice(["fp32", "bf16"])}
    return {"kind": kind, "rows": log_int(200, 262144), "precision": rng.choice(["fp32", "bf16", "fp8"]),
            "channels": rng.choice([1, 1, 3])}


# ---- inputs -----------------------------------------------------------------------

def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * seed + 17)
    return g


def _cloud(res, seed):
    """A seeded fBm cloud, res^3 floats on the device."""
    dens = torch.empty(res ** 3, device="cuda")
    scenes.generate_cloud_device(res, 500 + seed, dens.data_ptr())
    return dens


def _volume(res, dens):
    v = mr.VolumeRender(res)
    _lib.check(_lib.load().mr_volume_set_data_device(v.handle, _ptr(dens), dens.numel(), None))
    _lib.check(_lib.load().mr_volume_update(v.handle, None))
    return v


def _points(dens, res, n, gen):
    """n points in the medium (voxel centres, jittered) and unit directions."""
    inside = torch.nonzero(dens > 0.02).squeeze(1)
    pick = inside[torch.randint(len(inside), (n,), device="cuda", generator=gen)]
    ijk = torch.stack([pick // (res * res), (pick // res) % res, pick % res], 1).float()
    pos = (ijk + torch.rand(n, 3, device="cuda", generator=gen)) / res - 0.5
    d = torch.randn(n, 3, device="cuda", generator=gen)
    return pos.contiguous(), (d / d.norm(dim=1, keepdim=True)).contiguous()


_PAIRS = ([("LD%s%d1" % (t, i), 8, 8) for t in ("", "_Tr", "_Hg") for i in range(5)]
          + [("L%s%d1" % (t, i), s, s) for t in ("", "_Tr", "_Hg")
             for i, s in enumerate((8, 8, 16, 16, 16, 32, 32, 32, 32))])
_SQUEEZE = [(p + "%d1W" % i, p + "%d2W" % i) for p, k in (("LDSE", 4), ("LSE", 8)) for i in range(k)]
_HEAD = ([("LGGS", 8, 3), ("LC0", 128, 128), ("LC1", 64, 128), ("LC2", 32, 64), ("LX", 16, 32)]
         + [("LX%d" % i, 16, 16) for i in range(12)] + [("LX12", 1, 16)])


def _layout():
    """(name, shape) of the network's arrays in the order of a weight file."""
    out = []
    for name, o, i in _PAIRS:
        out += [(name + "W", (o, i)), (name + "B", (o,))]
    for a, b in _SQUEEZE:
        out += [(a, (8, 8)), (b, (3, 8))]
    out += [("LSEFin1W", (16, 75)), ("LSEFin2W", (6, 16))]
    for name, o, i in _HEAD:
        out += [(name + "W", (o, i)), (name + "B", (o,))]
    return out


def _weights(seed):
    """Xavier-uniform weights with small positive biases and a live output unit."""
    rng = np.random.default_rng(seed)
    out = []
    for name, shape in _layout():
        if len(shape) == 1:
            out.append(rng.uniform(0.0, 0.05, shape))
        else:
            b = math.sqrt(6.0 / (shape[0] + shape[1]))
            w = rng.uniform(-b, b, shape)
            out.append(np.abs(w) if name == "LX12W" else w)
    return np.concatenate([a.ravel() for a in out]).astype(np.float32)


def _rows(n, seed, channels=1):
    """Descriptor rows with the value ranges of gathered ones: sparse log
    densities, transmittances in [0, 1], skewed phase terms."""
    gen = _gen(seed)

    def u(*shape):
        return torch.rand(*shape, device="cuda", generator=gen)

    desc = torch.cat([1.2 * u(n, 192) ** 2 * (u(n, 192) > 0.3), u(n, 192), 1.5 * u(n, 192) ** 6], 1).contiguous()
    srp = 0.65 + 0.35 * u(n, 1)
    srp = srp.expand(n, 3) if channels == 1 else 0.65 + 0.35 * u(n, 3)
    aux = torch.cat([0.7 + 0.2 * u(n, 1), math.pi * u(n, 1), srp], 1).contiguous()
    label = (0.01 + 2.0 * u(n)).contiguous()
    return desc, aux, label


def _shipped_weights():
    import os
    return np.load(os.path.join(os.path.dirname(mr.__file__), "data", "mrpnn_trained.npy"))


class _Batch:
    def __init__(self):
        self.handle = C.c_void_p()
        _lib.check(_lib.load().mr_batch_create(C.byref(self.handle)))

    def __del__(self):
        _lib.load().mr_batch_destroy(self.handle)


def _light(seed, k=0):
    return scenes.seeded_light(seed + 7919 * k)


def _prepare_frame(c, seed):
    dens = _cloud(c["res"], seed)
    v = _volume(c["res"], dens)
    s = {"kind": "frame", "volume": v, "host": c["host"]}
    if c["host"]:
        v.SetWeights(_shipped_weights())
        v.SetScatterRate(ALBEDO)
        ori, up, right = scenes.camera_vectors(scenes.CAMERA_DIR * 2.5, 40.0)
        s["call"] = dict(size=(c["width"], c["height"]), ori=ori, up=up, right=right, lightDir=_light(seed),
                         rt=mr.MRPNN, g=G, alpha=ALPHA, sampleNum=1, precision=PRECISION[c["precision"]])
        return s
    s["net"] = mr.Network(_shipped_weights())
    s["params"] = scenes.cloud_scene_params(c["width"], c["height"], precision=PRECISION[c["precision"]],
                                            sampler=SAMPLER[c["sampler"]], light_seed=seed)
    s["out"] = torch.zeros(c["height"], c["width"], 3, device="cuda")
    return s


def _prepare_batch(c, seed):
    L = _lib.load()
    stream = torch.cuda.Stream()
    s = {"kind": "batch", "stream": stream, "net": mr.Network(_shipped_weights()), "volumes": [], "out": []}
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(c["views"] * 4099 + c["max_side"])
    for k, res in enumerate((64, 128, 256)):
        s["volumes"].append(_volume(res, _cloud(res, seed + 31 * k)))
    torch.cuda.synchronize()
    b = _Batch()
    s["batch"] = b
    for k in range(c["views"]):
        w, h = (max(16, int(c["max_side"] * f)) for f in sizes.uniform(0.25, 1.0, 2))
        p = scenes.make_params(w, h, 1, rt=_lib.RT_MRPNN, precision=PRECISION[c["precision"]],
                               sampler=SAMPLER[c["sampler"]], light_seed=seed)
        d = rng.normal(size=3)
        ori, up, right = scenes.camera_vectors(d / np.linalg.norm(d) * 2.5, 40.0)
        p.ori, p.up, p.right = _lib.f3(ori), _lib.f3(up), _lib.f3(right)
        s["out"].append(torch.zeros(h, w, 3, device="cuda"))
        _lib.check(L.mr_batch_add(b.handle, s["volumes"][k % 3].handle, C.byref(p), _ptr(s["out"][-1])))
    torch.cuda.synchronize()
    sp = C.c_void_p(stream.cuda_stream)
    _lib.check(L.mr_batch_prepare(b.handle, s["net"].handle, 0, sp))
    _lib.check(L.mr_batch_capture(b.handle, s["net"].handle, sp))
    return s


def _prepare_track(c, seed):
    v = mr.VolumeRender(c["res"])
    v.SetDatas(scenes.sphere_density(c["res"]))
    v.Update()
    v.SetScatterRate(ALBEDO)
    v.SetSeed(seed)
    ori, up, right = scenes.camera_vectors(scenes.CAMERA_DIR * 2.5, 40.0)
    return {"kind": "track", "volume": v,
            "call": dict(size=(c["side"], c["side"]), ori=ori, up=up, right=right, lightDir=_light(seed), rt=mr.PT, g=G,
                         alpha=ALPHA, multiScatter=512, sampleNum=c["spp"])}


def _prepare_interactive(c, seed):
    v = _volume(c["res"], _cloud(c["res"], seed))
    v.SetScatterRate(ALBEDO)
    v.SetSeed(seed)
    ori, up, right = scenes.camera_vectors(scenes.CAMERA_DIR * 2.5, 40.0)
    w, h = c["width"], c["height"]
    s = {"kind": "interactive", "volume": v, "frame": 0, "accum": torch.zeros(h, w, 3, device="cuda"),
         "hist": torch.zeros(h, w, 33, device="cuda"), "bgra": torch.zeros(h, w, dtype=torch.int32, device="cuda"),
         "call": dict(size=(w, h), ori=ori, up=up, right=right, lightDir=_light(seed), alpha=ALPHA, multiScatter=512,
                      g=G, denoise=True)}
    for _ in range(c["history"]):
        run(s)
    return s


def _prepare_scene(c, seed):
    gen = _gen(seed)
    dens = _cloud(c["res"], seed)
    v = _volume(c["res"], dens)
    n = c["points"]
    pos, dirs = _points(dens, c["res"], n, gen)
    net = mr.Network(_weights(seed))  # the gather uses its stencil
    media = []
    for k, (alpha, g) in enumerate(((ALPHA, G), (150.0, 0.78))):
        frames = torch.empty(n, 12, device="cuda")
        light = _light(seed, k)
        _lib.check(_lib.load().mr_train_frames(_ptr(dirs), n, _lib.f3(light), seed, _ptr(frames), None))
        media.append({"light": light, "alpha": alpha, "g": g, "frames": frames,
                      "desc": torch.zeros(n, 576, device="cuda"), "aux": torch.zeros(n, 5, device="cuda")})
    return {"kind": "scene", "volume": v, "net": net, "density": dens, "pos": pos, "media": media, "seed": seed}


def _prepare_labels(c, seed):
    gen = _gen(seed)
    dens = _cloud(c["res"], seed)
    v = _volume(c["res"], dens)
    pos, dirs = _points(dens, c["res"], c["points"], gen)
    return {"kind": "labels", "volume": v,
            "call": dict(points=pos.cpu().numpy(), dirs=dirs.cpu().numpy(), lightDir=_light(seed), alpha=ALPHA, g=G,
                         scatter=0.95, multiScatter=512, spp=c["spp"], seed=seed)}


def _prepare_train(c, seed):
    return {"kind": "train", "trainer": Trainer(_weights(seed), c["precision"]), "rows": _rows(c["rows"], seed)}


def _prepare_predict(c, seed):
    desc, aux, _ = _rows(c["rows"], seed, c["channels"])
    return {"kind": "predict", "net": mr.Network(_weights(seed)), "precision": PRECISION[c["precision"]], "desc": desc,
            "aux": aux, "out": torch.zeros(c["rows"], 3, device="cuda")}


def prepare(case, seed):
    return {"frame": _prepare_frame, "batch": _prepare_batch, "track": _prepare_track,
            "interactive": _prepare_interactive, "scene": _prepare_scene, "labels": _prepare_labels,
            "train": _prepare_train, "predict": _prepare_predict}[case["kind"]](case, seed)


# ---- one pass ----------------------------------------------------------------------

def run(s):
    L = _lib.load()
    kind = s["kind"]
    if kind == "frame":
        if s["host"]:
            return s["volume"].Render(**s["call"])
        _lib.check(L.mr_render(s["volume"].handle, s["net"].handle, C.byref(s["params"]), _ptr(s["out"]), None))
        return s["out"]
    if kind == "batch":
        _lib.check(L.mr_batch_launch(s["batch"].handle, C.c_void_p(s["stream"].cuda_stream)))
        return s["out"]
    if kind == "track":
        return s["volume"].Render(**s["call"])
    if kind == "interactive":
        s["volume"].RenderInteractive(s["accum"], s["hist"], s["bgra"], randseed=s["frame"], **s["call"])
        s["frame"] += 1
        return [s["accum"], s["hist"], s["bgra"]]
    if kind == "scene":
        v, n = s["volume"].handle, len(s["pos"])
        _lib.check(L.mr_volume_set_data_device(v, _ptr(s["density"]), s["density"].numel(), None))
        _lib.check(L.mr_volume_update(v, None))
        for m in s["media"]:
            _lib.check(L.mr_volume_update_tr(v, _lib.f3(m["light"]), m["alpha"], None))
            _lib.check(L.mr_volume_update_hglut(v, m["g"], s["seed"], None))
            _lib.check(L.mr_gather_descriptors(v, s["net"].handle, _ptr(s["pos"]), _ptr(m["frames"]), n, m["alpha"],
                                               m["g"], _lib.f3((ALBEDO,) * 3), _ptr(m["desc"]), _ptr(m["aux"]), None))
        # density, transmittance and phase columns of each medium's descriptors
        return [[m["desc"][:, :192], m["desc"][:, 192:384], m["desc"][:, 384:]] for m in s["media"]]
    if kind == "labels":
        return s["volume"].GetSamples(**s["call"])
    if kind == "train":
        grad, loss = s["trainer"].gradient(*s["rows"])
        return {"gradient": grad, "loss": loss}
    _lib.check(L.mr_radiance_predict(s["net"].handle, s["precision"], _ptr(s["desc"]), _ptr(s["aux"]), len(s["desc"]),
                                     _ptr(s["out"]), None))
    return s["out"]


def work(case):
    k = case["kind"]
    if k in ("frame", "batch"):
        if k == "frame":
            px, cells = case["width"] * case["height"], case["res"] ** 3
        else:
            px, cells = case["views"] * (0.625 * case["max_side"]) ** 2, 64 ** 3 + 128 ** 3 + 256 ** 3
        # the density and the table texels near the visible points, and the image
        return {"bytes": 12 * px + 4 * cells, "flops": IN_VIEW * px * NETWORK_FLOP}
    if k == "track":
        n = case["side"] ** 2
        return {"bytes": 12 * n + 4 * case["res"] ** 3, "flops": n * case["spp"] * 24 * 60}  # 24 collisions a path
    if k == "interactive":
        n = case["width"] * case["height"]  # colour, histogram and moments read and written, packed pixel written
        return {"bytes": n * (2 * 12 + 2 * 132 + 2 * 40 + 4) + 4 * case["res"] ** 3, "flops": IN_VIEW * n * 121 * 30 * 6}
    if k == "scene":
        pyramid, light = 4 * 8 * 256 ** 3 // 7, 4 * 8 * 128 ** 3 // 7
        out = 2 * case["points"] * 4 * (576 + 5)
        return {"bytes": 8 * case["res"] ** 3 + 2 * pyramid + 2 * (light + 4 * 512 ** 2) + out,
                "flops": 2 * (light / 4 * 128 * 25 + 512 ** 2 * 1024 * 25)}
    if k == "labels":
        n = case["points"]
        return {"bytes": 4 * case["res"] ** 3 + n * 32, "flops": n * case["spp"] * 60 * 60}
    if k == "train":
        return {"bytes": case["rows"] * 4 * 582, "flops": 3.0 * NETWORK_FLOP * case["rows"]}
    return {"bytes": case["rows"] * 4 * (576 + 5 + 3), "flops": 1.0 * NETWORK_FLOP * case["rows"] * (
        1 + 0.63 * (case["channels"] - 1))}


# ---- 64-bit results ------------------------------------------------------------------

def _forward64(w, desc, aux, channel):
    """Head output X of the network for one albedo channel, float64 rows."""
    relu, sig, lin = torch.relu, torch.sigmoid, torch.nn.functional.linear
    n = len(desc)
    d = desc.view(n, 3, 192)
    g, gamma, srp = aux[:, 0:1], aux[:, 1:2], aux[:, 2 + channel:3 + channel]
    mean, peak, comb = [], [], {}
    blocks = [("L", "LSE", i, s, f, m) for i, (s, f, m) in enumerate(zip(
        (8, 8, 16, 16, 16, 32, 32, 32), (0, 8, 16, 32, 48, 64, 96, 128), (0, 2, 1, 1, 2, 1, 1, 1)))]
    blocks += [("LD", "LDSE", i, 8, 160 + 8 * i, min(i, 1)) for i in range(4)]
    y = None
    for p, se, i, s, f, mode in blocks:
        x = d[:, :, f:f + s]
        av, mx = x.mean(2), x.amax(2)
        mean.append(av)
        peak.append(mx)
        gate = sig(lin(relu(lin(torch.cat([av, mx, g, gamma], 1), w["%s%d1W" % (se, i)])), w["%s%d2W" % (se, i)]))
        z = []
        for br, t in enumerate(("", "_Tr", "_Hg")):
            a = x[:, br] * gate[:, br:br + 1]
            a = a if mode == 0 else a + y[br]
            h = relu(lin(a, w["%s%s%d1W" % (p, t, i)], w["%s%s%d1B" % (p, t, i)]))
            z.append(torch.cat([h, x[:, br]], 1) if mode == 2 else h + x[:, br])
        y = z
        if (p, i) in (("L", 7), ("LD", 3)):
            comb[p] = [relu(lin(y[br], w["%s%s%d1W" % (p, t, i + 1)], w["%s%s%d1B" % (p, t, i + 1)]))
                       for br, t in enumerate(("", "_Tr", "_Hg"))]
    pool = torch.cat(mean + peak + [g, gamma, srp], 1)
    gates = sig(lin(relu(lin(pool, w["LSEFin1W"])), w["LSEFin2W"]))
    parts = [c * gates[:, i:i + 1] for i, c in enumerate(comb["L"] + comb["LD"])]
    a = torch.cat(parts + [relu(lin(torch.cat([g, gamma, srp], 1), w["LGGSW"], w["LGGSB"]))], 1)
    for name in ("LC0", "LC1", "LC2", "LX"):
        a = relu(lin(a, w[name + "W"], w[name + "B"]))
    for i in range(0, 12, 2):
        h = relu(lin(a, w["LX%dW" % i], w["LX%dB" % i]))
        a = a + relu(lin(h, w["LX%dW" % (i + 1)], w["LX%dB" % (i + 1)]))
    return relu(lin(a, w["LX12W"], w["LX12B"]))[:, 0]


def _weights64(seed):
    flat = torch.from_numpy(_weights(seed)).double().cuda()
    out, at = {}, 0
    for name, shape in _layout():
        k = int(np.prod(shape))
        out[name] = flat[at:at + k].view(shape)
        at += k
    return flat, out


def _exact_predict(c, seed):
    desc, aux, _ = _rows(c["rows"], seed, c["channels"])
    _, w = _weights64(seed)
    out = torch.empty(c["rows"], 3, dtype=torch.float64, device="cuda")
    for a in range(0, c["rows"], 32768):
        d, x = desc[a:a + 32768].double(), aux[a:a + 32768].double()
        for ch in range(3):
            if ch and c["channels"] == 1:
                out[a:a + 32768, ch] = out[a:a + 32768, 0]
            else:
                out[a:a + 32768, ch] = torch.clamp(torch.exp(_forward64(w, d, x, ch)) - 1, min=0) * x[:, 2 + ch]
    return out


def _exact_train(c, seed):
    desc, aux, label = (t.double() for t in _rows(c["rows"], seed))
    flat, w = _weights64(seed)
    flat.requires_grad_(True)
    grad, loss = torch.zeros_like(flat), 0.0
    for a in range(0, c["rows"], 16384):
        at, w = 0, {}
        for name, shape in _layout():
            k = int(np.prod(shape))
            w[name] = flat[at:at + k].view(shape)
            at += k
        x = _forward64(w, desc[a:a + 16384], aux[a:a + 16384], 0)
        part = ((x - torch.log1p(torch.clamp(label[a:a + 16384], min=0) / aux[a:a + 16384, 2])) ** 2).sum() / c["rows"]
        grad += torch.autograd.grad(part, flat)[0]
        loss += float(part)
    return {"gradient": grad.detach(), "loss": loss}


def _trilinear64(grid, uv, clamp):
    """Trilinear lookup of an x-major r^3 grid at uv in texture space; zero
    outside, or clamped to the edge."""
    r = grid.shape[0]
    p = uv * r - 0.5
    i = torch.floor(p)
    f = p - i
    i = i.long()
    flat = grid.reshape(-1)
    out = 0.0
    for dx in (0, 1):
        for dy in (0, 1):
            for dz in (0, 1):
                j = [i[..., a] + o for a, o in enumerate((dx, dy, dz))]
                cl = [q.clamp(0, r - 1) for q in j]
                v = flat[(cl[0] * r + cl[1]) * r + cl[2]]
                if not clamp:
                    ok = sum(((q >= 0) & (q < r)).int() for q in j) == 3
                    v = v * ok
                for a, o in enumerate((dx, dy, dz)):
                    v = v * (f[..., a] if o else 1 - f[..., a])
                out = out + v
    return out


def _centres(r):
    t = (torch.arange(r, device="cuda", dtype=torch.float64) + 0.5) / r
    return torch.stack(torch.meshgrid(t, t, t, indexing="ij"), -1)


def _box_exit(p, d, half):
    inv = 1.0 / d
    return torch.maximum(-p * inv + half * inv, -p * inv - half * inv).amin(-1)


def _box_entry(p, d, half):
    inv = 1.0 / d
    a, b = -p * inv + half * inv, -p * inv - half * inv
    lo, hi = torch.minimum(a, b).amax(-1), torch.maximum(a, b).amin(-1)
    return torch.where(hi >= lo, lo.clamp(min=0), torch.full_like(lo, -1.0))


def _exact_scene(c, seed):
    """Density and transmittance columns (the phase columns read a table that
    is a Monte Carlo estimate)."""
    s = _prepare_scene(c, seed)
    dens = s["density"].double().view((c["res"],) * 3)
    mips = [torch.cat([_trilinear64(dens.clamp(min=0), x, False) for x in _centres(256).split(32)])]
    for k in range(8):
        r = 128 >> k
        mips.append(mips[-1].view(r, 2, r, 2, r, 2).mean((1, 3, 5)))
    del dens
    pos = s["pos"].double()
    stencil = torch.from_numpy(mr.builtin_stencil()).double().cuda().view(160, 3)
    offset, level = [], []
    for k, m in enumerate((1, 1, 2, 2, 2, 4, 4, 4)):
        base = (1.0, 2.5, 5.5, 11.5, 23.5, 47.5, 95.5, 191.5)[k]
        t = max(0.0, 1.0 - 0.2 * k)
        offset += [base / 256 * (0.6 * (1 - t) + t)] * (8 * m)
        level += [k] * (8 * m)
    along = ([(i + 1) / 256 for i in range(8)] + [(9.5 + 2 * i) / 256 for i in range(8)]
             + [(26.5 + 4 * i) / 256 for i in range(8)] + [(60.5 + 8 * i) / 256 for i in range(8)])
    offset = torch.tensor(offset, dtype=torch.float64, device="cuda")
    along = torch.tensor(along, dtype=torch.float64, device="cuda")
    level = torch.tensor(level + [0] * 8 + [1] * 8 + [2] * 8 + [3] * 8, device="cuda")
    out = []
    for m in s["media"]:
        ldir = torch.tensor(np.asarray(m["light"]), dtype=torch.float64, device="cuda")
        ldir = ldir / ldir.norm()
        tr = []
        for k in range(8):
            r = 128 >> k
            rows = []
            for o in _centres(r).split(32):
                o = o - 0.5
                step = _box_exit(o, ldir, 0.5) / 128
                total = 0.0
                for q in range(1, 129):
                    total = total + _trilinear64(mips[k + 1], o + ldir * (step * q)[..., None] + 0.5, False)
                rows.append(torch.exp(-total * (m["alpha"] / 1.73 ** (k + 1)) * step))
            tr.append(torch.cat(rows))
        f = m["frames"].double().view(-1, 4, 3)
        # the along-light points follow the light axis of the frame
        ball = torch.einsum("nax,pa->npx", f[:, :3], stencil) * offset[:, None]
        p = pos[:, None] + torch.cat([ball, f[:, 3:4] * along[:, None]], 1)
        density = torch.empty(p.shape[:2], dtype=torch.float64, device="cuda")
        light = torch.empty_like(density)
        outside = ((p < -0.5) | (p > 0.5)).any(-1)
        entry = _box_entry(p, f[:, 3:4].expand_as(p), 0.4999)
        q = torch.where((outside & (entry >= 0))[..., None], p + f[:, 3:4] * entry[..., None], p)
        for k in range(8):
            at = level == k
            if at.any():
                density[:, at] = torch.log1p(m["alpha"] * _trilinear64(mips[k], p[:, at] + 0.5, False) / 64)
                light[:, at] = _trilinear64(tr[max(k - 1, 0)], q[:, at] + 0.5, True)
        light[outside & (entry < 0)] = 1.0
        out.append([density, light, None])
    return out


def exact(case, seed):
    fn = {"predict": _exact_predict, "train": _exact_train, "scene": _exact_scene}.get(case["kind"])
    return fn(case, seed) if fn else None
