"""Performance cases of the neural-radiance-cache library: what a renderer that
embeds it calls, through the public binding (vknrc_gb300.nrc), from one small
query to a whole frame.

listed() names the cases, draw(rng) makes more of the same ranges, prepare()
builds what the program holds before the call, run() makes one pass, work() says
what a pass cannot do without, and exact() computes the results in 64 bits with
plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vknrc_gb300 import nrc, synthetic

P = nrc.P
BATCHES = nrc.TRAIN_BATCH_COUNT
LR, BETA1, BETA2, EPS, EMA = 1e-3, 0.9, 0.99, 1e-8, 0.99
MLP_FLOPS = 2 * (5 * 64 * 64 + 3 * 64)          # one record forward
TRAIN_FLOPS = 3 * MLP_FLOPS - 2 * 64 * 64       # forward, dW and dA (none for the input)
PARAM_BYTES = P * (2 * 16 + 2 * 2)              # Adam entries read and written, two 16-bit vectors
BATCHED_QUERIES = [256 * 256, 640 * 360, 960 * 540, 1280 * 720, 1600 * 900, 1920 * 1080, 2048 * 1152, 2560 * 1440]
BATCHED_TRAIN = [4096, 8192, 16384, 24576, 32768, 40960, 49152, 65536]


def listed():
    return [
        # a probe or tile of a few pixels: the call's latency
        {"name": "query_1k", "kind": "query", "fmt": "fp16", "n": 1000},
        # every pixel of a 1080p frame, the reference's query pass
        {"name": "query_1080p", "kind": "query", "fmt": "fp16", "n": 1920 * 1080},
        # a 720p frame with some escaped paths (a ragged count), in the bf16 form
        {"name": "query_720p_bf16", "kind": "query", "fmt": "bf16", "n": 911_487},
        # the largest frame of the serving mix, in the FP8 form
        {"name": "query_1440p_fp8", "kind": "query", "fmt": "fp8", "n": 2560 * 1440},
        # one training step on a few paths, as a low-rate updater runs it, bf16
        {"name": "train_1k_bf16", "kind": "train", "fmt": "bf16", "n": 1000, "steps": 1},
        # the four chained training steps of a frame
        {"name": "train_4x16k", "kind": "train", "fmt": "fp16", "n": 16384, "steps": 4},
        # the largest training batch of the batched configuration, one step
        {"name": "train_64k", "kind": "train", "fmt": "fp16", "n": 65536, "steps": 1},
        # a 1080p frame: queries and four training steps, unpacked records
        {"name": "frame_1080p", "kind": "frame", "n": 1920 * 1080, "train": 16384},
        # the same frame from the reference's packed records of a 522,254-triangle scene
        {"name": "frame_packed_1080p", "kind": "packed", "n": 1920 * 1080, "train": 16384, "grid": 512},
        # a rendered 1080p frame with the cache: path trace, query into the image, screen pass
        {"name": "render_1080p", "kind": "render", "width": 1920, "height": 1080, "grid": 512},
        # the path tracer without the cache (reference images), full-length paths
        {"name": "trace_540p", "kind": "trace", "width": 960, "height": 540, "grid": 512, "method": 0},
        # eight caches with uneven counts, one batched launch per phase
        {"name": "many_8", "kind": "many", "jobs": 8, "scale": 1.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "train", "frame", "packed", "render", "trace", "many"])
    if kind == "query":
        return {"kind": kind, "fmt": rng.choice(["fp16", "bf16", "fp8"]), "n": _log(rng, 100, 2560 * 1440)}
    if kind == "train":
        return {"kind": kind, "fmt": rng.choice(["fp16", "bf16"]), "n": _log(rng, 200, 65536), "steps": rng.randint(1, 4)}
    if kind == "frame":
        return {"kind": kind, "n": _log(rng, 256 * 256, 2560 * 1440), "train": _log(rng, 2048, 16384)}
    if kind == "packed":
        return {"kind": kind, "n": _log(rng, 256 * 256, 1920 * 1080), "train": _log(rng, 2048, 16384),
                "grid": rng.randint(64, 512)}
    if kind == "render":
        h = rng.randint(200, 1080)
        return {"kind": kind, "width": int(h * rng.uniform(1.0, 1.77)), "height": h, "grid": rng.randint(64, 512)}
    if kind == "trace":
        h = rng.randint(120, 540)
        return {"kind": kind, "width": int(h * rng.uniform(1.0, 1.77)), "height": h, "grid": rng.randint(64, 512),
                "method": rng.randint(0, 2)}
    return {"kind": kind, "jobs": rng.randint(2, 8), "scale": round(rng.uniform(0.05, 0.9), 3)}


# ------------------------------------------------------------------- inputs --
def _gen(seed, stream=0):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + stream * 7919 + 17) & 0x7FFFFFFFFFFF)


def _weights(seed):
    """He-normal weights, as a cache starts with, in fp32 on the host."""
    return np.random.default_rng([seed, 5]).normal(0.0, math.sqrt(2.0 / 64), P).astype(np.float32)


def _w16(seed, fmt):
    w = torch.from_numpy(_weights(seed)).to(torch.bfloat16 if fmt == "bf16" else torch.float16)
    return w


def _cache(seed, fmt="fp16", batch=nrc.TRAIN_BATCH_SIZE):
    c = nrc.Cache(seed=seed, learning_rate=LR, beta1=BETA1, beta2=BETA2, epsilon=EPS, ema_alpha=EMA,
                  train_batch_size=max(batch, nrc.TRAIN_BATCH_SIZE),
                  precision=nrc.PRECISION_BF16 if fmt == "bf16" else nrc.PRECISION_FP16,
                  fp8_inference=1 if fmt == "fp8" else 0)
    if fmt == "fp8":  # one step, so that the activations' scales are those of real records
        c.train(_train(seed, 9, 16384), _count(16384), write_use=True)
    c.set_weights(_w16(seed, fmt).view(torch.int16).numpy().view(np.uint16))
    return c


def _queries(seed, stream, n):
    """(n, 14) unpacked records: positions and albedos uniform, directions on the sphere."""
    return synthetic.train_records_device(_gen(seed, stream), n)[:, 6:20].contiguous()


def _train(seed, stream, n):
    """(n, 20) training records: a smooth radiance field times lognormal noise (of a few samples a path)."""
    return synthetic.train_records_device(_gen(seed, stream), n, sigma=0.5)


def _count(n):
    return torch.tensor([n], dtype=torch.int32, device="cuda")


def _rgb(n):
    return torch.zeros((n, 3), dtype=torch.float32, device="cuda")


class _Buffer:
    """A device buffer of a cache, for torch.as_tensor; keeps the cache alive while a view of it is."""

    def __init__(self, cache, ptr, shape, typestr):
        self.cache = cache
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3, "strides": None}


def _views(c, fmt="fp16"):
    """The cache's own parameter buffers: weights, rendering weights, Adam entries, step state."""
    w, u, e, s = c.device_buffers()
    t = torch.bfloat16 if fmt == "bf16" else torch.float16

    def view(ptr, shape, typestr):
        return torch.as_tensor(_Buffer(c, ptr, shape, typestr), device="cuda")

    return {"weights": view(w, (P // 2,), "<i4").view(t), "use_weights": view(u, (P // 2,), "<i4").view(t),
            "entries": view(e, (P, 4), "<f4"), "state": view(s, (5,), "<i4")}


def _scene_arrays(seed, grid):
    return synthetic.terrain_scene(np.random.default_rng([seed, 3]), grid)


def _packed(seed, stream, n, sc):
    """(n, 4) packed inputs over the scene's primitives (both instances), uniform barycentrics and directions."""
    g = _gen(seed, stream)
    prims, inst = sc["vertex_indices"].shape[0], sc["transforms"].shape[0]
    out = torch.empty((n, 4), dtype=torch.int32, device="cuda")

    def word(lo, hi):
        w = lo.long() | (hi.long() << 16)
        return torch.where(w >= 2**31, w - 2**32, w).int()

    out[:, 0] = torch.randint(0, prims, (n,), generator=g, device="cuda", dtype=torch.int32)
    flip = torch.randint(0, 2, (n,), generator=g, device="cuda")
    out[:, 1] = word(torch.randint(0, inst, (n,), generator=g, device="cuda"), flip << 15)
    b = torch.rand((n, 2), generator=g, device="cuda")
    b = torch.where(b.sum(1, keepdim=True) > 1, 1 - b, b)
    bq = torch.round(b * 65535)
    out[:, 2] = word(bq[:, 0], bq[:, 1])
    v = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    d = torch.round(_sph(v / v.norm(dim=1, keepdim=True)) * 65535)
    out[:, 3] = word(d[:, 0], d[:, 1])
    return out


def _eval_records(seed, n, sc):
    r = torch.empty((n, 5), dtype=torch.int32, device="cuda")
    r[:, 0] = -1  # no destination
    r[:, 1:] = _packed(seed, 21, n, sc)
    return r


def _packed_train(seed, b, n, sc):
    r = torch.empty((n, 10), dtype=torch.int32, device="cuda")
    f = r.view(torch.float32)
    f[:, 0:3] = torch.exp(0.5 * torch.randn((n, 3), generator=_gen(seed, 40 + b), device="cuda"))
    f[:, 3:6] = 1.0
    r[:, 6:] = _packed(seed, 30 + b, n, sc)
    return r


def _many_sizes(case):
    jobs, s = case["jobs"], case["scale"]
    return ([max(1, int(q * s)) for q in BATCHED_QUERIES[8 - jobs:]], [max(1, int(t * s)) for t in BATCHED_TRAIN[8 - jobs:]])


def _camera(case, seed):
    p = nrc.TraceParams()
    r = np.random.default_rng([seed, 4])
    p.origin[:] = (float(r.uniform(-0.3, 0.3)), float(r.uniform(0.25, 0.4)), float(r.uniform(-1.9, -1.6)))
    p.look[:] = (float(r.uniform(-0.1, 0.1)), -0.25, 1.0)
    p.side[:] = (0.8, 0.0, 0.0)
    p.up[:] = (0.0, 0.8 * case["height"] / case["width"], 0.0)
    p.width, p.height = case["width"], case["height"]
    p.seed = seed * 65536
    p.left_method = p.right_method = case.get("method", 1)
    p.train_probability = min(0.03, 6000.0 / (case["width"] * case["height"]))  # the frame's training paths
    return p


# -------------------------------------------------------------------- cases --
def prepare(case, seed):
    k = case["kind"]
    if k == "query":
        n = case["n"]
        return {"k": k, "fmt": case["fmt"], "c": _cache(seed, case["fmt"]), "x": _queries(seed, 1, n), "cnt": _count(n),
                "out": _rgb(n)}
    if k == "train":
        n = case["n"]
        c = _cache(seed, case["fmt"], n)
        return {"k": k, "c": c, "rec": [_train(seed, 10 + b, n) for b in range(case["steps"])],
                "cnt": [_count(n) for _ in range(case["steps"])], "views": _views(c, case["fmt"])}
    if k == "frame":
        n, t = case["n"], case["train"]
        c = _cache(seed)
        return {"k": k, "c": c, "x": _queries(seed, 1, n), "cnt": _count(n), "out": _rgb(n),
                "rec": [_train(seed, 10 + b, t) for b in range(BATCHES)], "tcnt": [_count(t) for _ in range(BATCHES)],
                "views": _views(c)}
    if k == "packed":
        n, t = case["n"], case["train"]
        sc = _scene_arrays(seed, case["grid"])
        c = _cache(seed)
        return {"k": k, "c": c, "scene": nrc.DeviceScene(sc).prepare(), "x": _eval_records(seed, n, sc),
                "cnt": _count(n), "out": _rgb(n), "rec": [_packed_train(seed, b, t, sc) for b in range(BATCHES)],
                "tcnt": [_count(t) for _ in range(BATCHES)], "views": _views(c)}
    if k in ("render", "trace"):
        w, h = case["width"], case["height"]
        scene = nrc.DeviceScene(_scene_arrays(seed, case["grid"])).prepare()
        s = {"k": k, "scene": scene, "bvh": nrc.Bvh(scene), "p": _camera(case, seed), "buf": nrc.TraceBuffers(w, h)}
        if k == "render":
            b = s["buf"]
            s["c"] = _cache(seed)
            s["targets"] = nrc.scatter_targets(b.bias_factor_r, b.factor_gb, b.train)
            s["acc"] = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")
            s["rgba8"] = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
            s["frame"] = 0
        return s
    qs, ts = _many_sizes(case)
    s = {"k": k, "c": [], "q": [], "t": [], "out": [], "views": []}
    for j, (q, t) in enumerate(zip(qs, ts)):
        c = _cache(seed * 16 + j, "fp16", t)
        out = _rgb(q)
        s["c"].append(c)
        s["out"].append(out)
        s["views"].append(_views(c))
        s["q"].append(nrc.query_job(c, _queries(seed, 50 + j, q), _count(q), out))
        s["t"].append(nrc.train_job(c, [_train(seed, 60 + j * BATCHES + b, t) for b in range(BATCHES)],
                                    [_count(t) for _ in range(BATCHES)]))
    return s


def run(s):
    k = s["k"]
    if k == "query":
        (s["c"].infer_fp8 if s["fmt"] == "fp8" else s["c"].infer)(s["x"], s["cnt"], s["out"])
        return s["out"]
    if k == "train":
        if len(s["rec"]) == 1:
            s["c"].train(s["rec"][0], s["cnt"][0], write_use=True)
        else:
            s["c"].train_batches(s["rec"], s["cnt"], write_use_last=True)
        return s["views"]
    if k == "frame":
        s["c"].frame_overlapped(s["x"], s["cnt"], s["out"], s["rec"], s["tcnt"])
        return {"rgb": s["out"], **s["views"]}
    if k == "packed":
        s["c"].frame_packed(s["scene"], s["x"], s["cnt"], s["out"], s["rec"], s["tcnt"])
        return {"rgb": s["out"], **s["views"]}
    if k in ("render", "trace"):
        b = s["buf"]
        b.reset()
        nrc.path_trace(s["scene"], s["bvh"], s["p"], b)
        images = {"bias_factor_r": b.bias_factor_r, "factor_gb": b.factor_gb, "eval_count": b.eval_count,
                  "train_counts": b.train_counts}
        if k == "trace":
            return images
        s["c"].infer_scatter_packed(s["scene"], b.eval, b.eval_count, s["targets"])
        nrc.screen(b.bias_factor_r, s["acc"], s["frame"], out_rgba8=s["rgba8"])
        s["frame"] += 1
        s["p"].seed += 1
        return {**images, "accumulated": s["acc"], "rgba8": s["rgba8"]}
    nrc.infer_many(s["q"])
    nrc.train_many(s["t"])
    return {"rgb": s["out"], "caches": s["views"]}


def work(case):
    k = case["kind"]
    if k == "query":
        return {"bytes": case["n"] * 68, "flops": case["n"] * MLP_FLOPS}
    if k == "train":
        n = case["n"] * case["steps"]
        return {"bytes": n * 80 + PARAM_BYTES, "flops": n * TRAIN_FLOPS}
    if k in ("frame", "packed"):
        t = case["train"] * BATCHES
        scene = 2 * (case["grid"] - 1) ** 2 * 64 if k == "packed" else 0
        return {"bytes": case["n"] * (68 if k == "frame" else 32) + t * (80 if k == "frame" else 40) + PARAM_BYTES + scene,
                "flops": case["n"] * MLP_FLOPS + t * TRAIN_FLOPS}
    if k in ("render", "trace"):
        # a ray: a path from the tree's root to a triangle, 20 operations a node; the images written once
        px, tris = case["width"] * case["height"], 2 * (case["grid"] - 1) ** 2
        rays = 8 if case.get("method", 1) == 0 else 2
        flops, nbytes = px * rays * 20 * math.log2(tris), px * 24 + tris * 48
        if k == "render":
            flops, nbytes = flops + px * MLP_FLOPS, nbytes + px * (40 + 24 + 16 + 36)
        return {"bytes": nbytes, "flops": flops}
    qs, ts = _many_sizes(case)
    return {"bytes": sum(qs) * 68 + BATCHES * sum(ts) * 80 + len(qs) * PARAM_BYTES,
            "flops": sum(qs) * MLP_FLOPS + BATCHES * sum(ts) * TRAIN_FLOPS}


# ----------------------------------------------------------- 64-bit results --
def _sph(d):
    u = 0.5 + torch.atan2(d[:, 1], d[:, 0]) / (2 * math.pi)
    u = torch.where((d[:, 0] == 0) & (d[:, 1] == 0), torch.full_like(u, 0.5), u)
    return torch.stack([u, torch.arccos(d[:, 2].clamp(-1, 1)) / math.pi], 1)


def _encode(x):
    """64 features: 12 triangle waves a coordinate, one-blobs of directions, normal and roughness, albedos, ones."""
    f = [2 * (torch.remainder(x[:, c:c + 1] * 2.0 ** torch.arange(12, device=x.device, dtype=x.dtype) - 0.5, 2) - 1).abs() - 1
         for c in range(3)]
    edges = torch.arange(5, device=x.device, dtype=x.dtype) / 4

    def blob(v):
        u = (edges[None, :] - v[:, None]) * 4
        cdf = ((15 / 16) * u * (1 - 2 / 3 * u * u + 0.2 * u ** 4) + 0.5).clamp(0, 1)
        return cdf[:, 1:] - cdf[:, :-1]

    f += [blob(x[:, c]) for c in range(3, 7)] + [blob(1 - torch.exp(-x[:, 7])), x[:, 8:14], torch.ones_like(x[:, :2])]
    return torch.cat(f, 1)


def _layers(w):
    return [w[l * 4096:(l + 1) * 4096].view(64, 64) for l in range(5)] + [w[5 * 4096:].view(3, 64)]


def _forward(w, x, clamp=True):
    parts = []
    for i in range(0, x.shape[0], 1 << 18):
        a = _encode(x[i:i + (1 << 18)].double())
        for l, m in enumerate(_layers(w)):
            a = a @ m.T
            a = a.clamp_min(0) if l < 5 else a
        parts.append(a.clamp_min(0) if clamp else a)
    return torch.cat(parts)


def _gradient(w, rec):
    """The weight-gradient sum under the relative-L2 luminance loss, the denominator held constant."""
    total = torch.zeros(P, dtype=torch.float64, device=rec.device)
    ms = _layers(w)
    for i in range(0, rec.shape[0], 1 << 16):
        r = rec[i:i + (1 << 16)].double()
        acts = [_encode(r[:, 6:20])]
        for m in ms[:5]:
            acts.append((acts[-1] @ m.T).clamp_min(0))
        p = acts[5] @ ms[5].T
        lum = p.clamp_min(0) @ torch.tensor([0.299, 0.587, 0.114], dtype=torch.float64, device=rec.device)
        g = 2 * (p - r[:, 0:3]) / (lum * lum + 0.01)[:, None]
        parts = []
        for l in range(5, -1, -1):
            parts.append((g.T @ acts[l]).reshape(-1))
            g = (g @ ms[l]) * (acts[l] > 0) if l > 0 else g
        total += torch.cat(parts[::-1])
    return total


def _trained(w, batches):
    """The chained Adam and EMA steps: (weights, rendering weights, entries)."""
    w = w.clone()
    m, v, ema = torch.zeros_like(w), torch.zeros_like(w), w.clone()
    for t, rec in enumerate(batches, 1):
        g = _gradient(w, rec) / rec.shape[0]
        m = BETA1 * m + (1 - BETA1) * g
        v = BETA2 * v + (1 - BETA2) * g * g
        w = w - LR * (m / (1 - BETA1 ** t)) / ((v / (1 - BETA2 ** t)).sqrt() + EPS)
        ema = (1 - EMA) / (1 - EMA ** t) * w + EMA * (1 - EMA ** (t - 1)) / (1 - EMA ** t) * ema
    # after several steps the squared gradients of a few bright records, which 16 bits round coarsely, outweigh the rest
    entries = torch.stack([m, v, w, ema], 1) if len(batches) == 1 else None
    return {"weights": w, "use_weights": w, "entries": entries, "state": None}


def _unpack(packed, sc):
    """The 14 input floats of packed records, from the scene's arrays."""
    dev = {k: torch.from_numpy(np.ascontiguousarray(v.view(np.int32) if v.dtype == np.uint32 else v)).cuda()
           for k, v in sc.items() if k not in ("textures", "instance_ranges")}
    word = packed.long() & 0xFFFFFFFF
    prim, inst, flip = word[:, 0], word[:, 1] & 0x7FFFFFFF, (word[:, 1] >> 31) == 1
    T = dev["transforms"].double()[inst]
    vi, ti = dev["vertex_indices"].long()[prim], dev["texcoord_indices"].long()[prim]
    v = dev["vertices"].double()[vi]
    v = torch.einsum("nij,nkj->nki", T[:, :, :3], v) + T[:, None, :, 3]
    n = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    n = n / n.norm(dim=1, keepdim=True)
    n = torch.where(flip[:, None], -n, n)
    b1, b2 = (word[:, 2] & 0xFFFF).double() / 65535, (word[:, 2] >> 16).double() / 65535
    b = torch.stack([1 - b1 - b2, b1, b2], 1)
    pos = (v * b[:, :, None]).sum(1)
    tc = (dev["texcoords"].double()[ti] * b[:, :, None]).sum(1)
    mat = dev["materials"][dev["material_ids"].long()[prim]]
    out = [pos, torch.stack([(word[:, 3] & 0xFFFF).double(), (word[:, 3] >> 16).double()], 1) / 65535, _sph(n),
           mat[:, 13:14].double()]
    for col, tex in ((0, 3), (4, 7)):
        ids = mat.view(torch.int32)[:, tex].long() & 0xFFFFFFFF
        c = mat[:, col:col + 3].double()
        for t, img in enumerate(sc["textures"]):
            h, w = img.shape[:2]
            lin = torch.from_numpy(img[:, :, :3].astype(np.float64) / 255).cuda()
            lin = torch.where(lin <= 0.04045, lin / 12.92, ((lin + 0.055) / 1.055) ** 2.4)
            u, q = tc[:, 0] * w - 0.5, tc[:, 1] * h - 0.5
            i, j = u.floor(), q.floor()
            a, e = (u - i)[:, None], (q - j)[:, None]
            i0, j0 = i.long() % w, j.long() % h
            i1, j1 = (i0 + 1) % w, (j0 + 1) % h
            s = (lin[j0, i0] * (1 - a) + lin[j0, i1] * a) * (1 - e) + (lin[j1, i0] * (1 - a) + lin[j1, i1] * a) * e
            c = torch.where((ids == t)[:, None], s, c)
        out.append(c)
    return torch.cat(out, 1)


def exact(case, seed):
    k = case["kind"]
    if k == "query" and case["fmt"] == "fp8":
        return None  # its result is the quantised network's, 14% from the unquantised one's
    if k == "query":
        return _forward(_w16(seed, case["fmt"]).double().cuda(), _queries(seed, 1, case["n"]))
    if k == "train":
        w = _w16(seed, case["fmt"]).double().cuda()
        return _trained(w, [_train(seed, 10 + b, case["n"]) for b in range(case["steps"])])
    if k == "frame":
        w = _w16(seed, "fp16").double().cuda()
        return {"rgb": _forward(w, _queries(seed, 1, case["n"])),
                **_trained(w, [_train(seed, 10 + b, case["train"]) for b in range(BATCHES)])}
    if k == "packed":
        sc = _scene_arrays(seed, case["grid"])
        w = _w16(seed, "fp16").double().cuda()
        rec = _eval_records(seed, case["n"], sc)
        rgb = torch.cat([_forward(w, _unpack(rec[i:i + (1 << 18), 1:], sc)) for i in range(0, case["n"], 1 << 18)])
        batches = []
        for b in range(BATCHES):
            r = _packed_train(seed, b, case["train"], sc)
            batches.append(torch.cat([r.view(torch.float32)[:, :6].double(), _unpack(r[:, 6:], sc)], 1))
        return {"rgb": rgb, **_trained(w, batches)}
    if k == "many":
        qs, ts = _many_sizes(case)
        rgb, caches = [], []
        for j, (q, t) in enumerate(zip(qs, ts)):
            w = _w16(seed * 16 + j, "fp16").double().cuda()
            rgb.append(_forward(w, _queries(seed, 50 + j, q)))
            caches.append(_trained(w, [_train(seed, 60 + j * BATCHES + b, t) for b in range(BATCHES)]))
        return {"rgb": rgb, "caches": caches}
    return None  # a traced path: rounding decides which triangle a ray meets
