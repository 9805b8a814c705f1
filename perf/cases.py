"""Performance cases of the reconstruction library: what its users have it do,
through the Python binding, over the ranges it is used in.

A case is a dict of plain values; `kind` says which entry points it goes through:

  frame    a new sample buffer in device memory: hierarchy rebuild and
           reconstruction into a device image (TreeGather.rebuild,
           reconstruct_to_device)
  host     the same with host buffers: upload, rebuild, reconstruction, image
           back in host memory (TreeGather.rebuild_from, reconstructDofMotion)
  batch    several built buffers of uneven size reconstructed as one graph
  sweep    one hierarchy under several output settings as one graph (a movie)
  routed   a frame with the learned router on
  network  the router's network alone: inference over an image's pixels, and
           loss and gradient over labelled rows

Records come from the library's own scene generator, whose scenes have the
sizes, depths, motion and circles of confusion of the configurations.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "temporal-lightfield-reconstruction_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import tlfr  # noqa: E402

# largest empty circle radius by samples per pixel, as the method uses it
_DISPERSION = {1: 2.0, 2: 1.34, 4: 1.1, 8: 0.8, 16: 0.5}

_FEATURE_MEAN = [1.5, 0.5, 6.0, 1.0, 1.5, 0.5, 10.0, 0.3]
_FEATURE_STD = [1.0, 0.6, 5.0, 0.8, 1.0, 0.6, 12.0, 0.3]


def _frame(name, scene, width, height, spp, **more):
    c = {"name": name, "kind": "frame", "scene": scene, "width": width, "height": height, "spp": spp,
         "output_spp": 128, "pinhole": False, "gaussian": False, "aperture": 1.0, "focus": 1.0, "toggle": False}
    c.update(more)
    return c


def listed():
    planes, cards, large = tlfr.SCENE_PLANES, tlfr.SCENE_CARDS, tlfr.SCENE_CARDS_LARGE
    return [
        # a preview or a unit test: launches and synchronisations count
        _frame("preview_64x48x4", cards, 64, 48, 4),
        # defocus only, densely sampled, half the output samples
        _frame("defocus_256x256x16", planes, 256, 256, 16, output_spp=64),
        # defocus and motion at an odd size
        _frame("motion_962x543x4", cards, 962, 543, 4),
        # the full-size frame with strong blur
        _frame("strong_1920x1080x8", large, 1920, 1080, 8),
        # the sharp t = 1 image: one output sample per pixel, so the hierarchy build dominates
        _frame("pinhole_1280x720x8", large, 1280, 720, 8, pinhole=True),
        # sparse input, refocused, Gaussian lens and shutter
        _frame("refocus_481x271x1", cards, 481, 271, 1, gaussian=True, aperture=0.7, focus=1.3),
        # the reference's GPU algorithm (its toggle)
        _frame("toggle_200x150x4", cards, 200, 150, 4, toggle=True),
        # a host program: records in host memory, image back in host memory
        _frame("host_640x480x4", cards, 640, 480, 4, kind="host"),
        # a mixed job: buffers of several sizes and sampling rates
        {"name": "batch_6_uneven", "kind": "batch", "scene": cards, "frames": 6, "width": 640, "height": 480,
         "spp": 16},
        # a (u, v, t) movie of one buffer
        {"name": "sweep_8_of_640x480x4", "kind": "sweep", "scene": cards, "frames": 8, "width": 640, "height": 480,
         "spp": 4},
        # the learned router in front of a frame
        _frame("routed_640x360x8", large, 640, 360, 8, kind="routed"),
        # the router's network: inference over a 1080p image, gradient over a training set
        {"name": "network_1080p", "kind": "network", "pixels": 1920 * 1080, "rows": 262144},
    ]


def _size(rng, lo, hi):
    """(width, height) with a log-uniform pixel count in [lo, hi]; widths and heights of any parity."""
    pixels = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = rng.uniform(1.0, 2.0)
    return max(8, int(math.sqrt(pixels * aspect))), max(8, int(math.sqrt(pixels / aspect)))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "pinhole", "refocus", "toggle", "host", "batch", "sweep", "routed",
                       "network"])
    scene = rng.choice([tlfr.SCENE_PLANES, tlfr.SCENE_CARDS, tlfr.SCENE_CARDS_LARGE])
    spp = rng.choice([1, 2, 4, 8, 16])
    if kind == "network":
        return {"kind": "network", "pixels": int(math.exp(rng.uniform(math.log(3e3), math.log(2e6)))),
                "rows": int(math.exp(rng.uniform(math.log(1e3), math.log(2.5e5))))}
    if kind in ("batch", "sweep"):
        w, h = _size(rng, 100 * 75, 640 * 480)
        return {"kind": kind, "scene": scene, "frames": rng.randint(2, 8), "width": w, "height": h, "spp": spp}
    most = {"frame": 1280 * 720, "pinhole": 1920 * 1080, "refocus": 640 * 480, "toggle": 200 * 150,
            "host": 960 * 540, "routed": 640 * 360}[kind]
    w, h = _size(rng, 64 * 48, most)
    more = {}
    if kind == "pinhole":
        more["pinhole"] = True
    if kind == "refocus":
        more.update(gaussian=rng.random() < 0.5, aperture=rng.uniform(0.5, 1.2), focus=rng.uniform(0.8, 1.5))
    if kind == "toggle":
        more["toggle"] = True
    if kind in ("host", "routed"):
        more["kind"] = kind
    if kind == "frame":
        more["output_spp"] = rng.choice([128, 128, 64, 32, rng.randint(8, 127)])
    c = _frame("", scene, w, h, spp, **more)
    del c["name"]
    return c


def _params(case):
    g = case["gaussian"]
    return tlfr.CameraParams(lensFilter=tlfr.LENS_GAUSSIAN if g else tlfr.LENS_BOX,
                             timeFilter=tlfr.TIME_GAUSSIAN if g else tlfr.TIME_BOX,
                             overrideUVT=(0.0, 0.0, 1.0) if case["pinhole"] else None,
                             enableCuda=case["toggle"], outputSpp=0 if case["pinhole"] else case["output_spp"])


def _uneven(case):
    """The sizes of a batch's buffers: from the case's largest down, sampling rates cycling."""
    rates = [1, 2, 4, 8, 16]
    out = []
    for k in range(case["frames"]):
        f = 1.0 / (1.0 + 0.45 * k)
        out.append((max(16, int(case["width"] * f)), max(16, int(case["height"] * f)),
                    rates[(rates.index(case["spp"]) + k) % 5]))
    return out


def _records(scene, width, height, spp, seed):
    rec, coc = tlfr.synth_scene(scene, width, height, spp, seed + 1)
    return torch.from_numpy(rec).cuda(), coc


def _image(width, height):
    return torch.empty((height, width, 4), dtype=torch.float32, device="cuda")


def prepare(case, seed):
    seed = int(seed) & 0x3FFFFFFF
    kind = case["kind"]
    if kind == "network":
        gen = torch.Generator().manual_seed(seed)
        n = max(case["pixels"], case["rows"])
        feats = torch.randn((n, 8), generator=gen) * torch.tensor(_FEATURE_STD) + torch.tensor(_FEATURE_MEAN)
        labels = (torch.rand(case["rows"], generator=gen) < 0.65).float()
        router = tlfr.Router(0, seed=seed + 1, mean=np.float32(_FEATURE_MEAN), inv_std=1 / np.float32(_FEATURE_STD))
        return {"kind": kind, "router": router, "feats": feats.cuda(), "labels": labels.cuda(),
                "pixels": case["pixels"], "rows": case["rows"],
                "prob": torch.empty(case["pixels"], dtype=torch.float32, device="cuda")}
    if kind == "batch":
        trees, outs, keep = [], [], []
        for k, (w, h, s) in enumerate(_uneven(case)):
            rec, coc = _records(case["scene"], w, h, s, seed + 1000 * k)
            trees.append(tlfr.TreeGather(None, tlfr.CameraParams(), device_records=(rec.data_ptr(), (w, h, s), coc)))
            outs.append(_image(w, h))
            keep.append(rec)
        batch = tlfr.Batch(trees, [o.data_ptr() for o in outs])
        return {"kind": kind, "batch": batch, "outs": outs, "keep": (trees, keep)}
    w, h, s = case["width"], case["height"], case["spp"]
    if kind == "sweep":
        rec, coc = _records(case["scene"], w, h, s, seed)
        tree = tlfr.TreeGather(None, tlfr.CameraParams(), device_records=(rec.data_ptr(), (w, h, s), coc))
        n = case["frames"]
        params = [tlfr.CameraParams(overrideUVT=(0.7 * math.cos(2 * math.pi * k / n),
                                                 0.7 * math.sin(2 * math.pi * k / n), k / n)) for k in range(n)]
        outs = [_image(w, h) for _ in params]
        batch = tlfr.Batch([tree] * n, [o.data_ptr() for o in outs], params=params)
        return {"kind": kind, "batch": batch, "outs": outs, "keep": (tree, rec)}
    if kind == "host":
        rec, coc = tlfr.synth_scene(case["scene"], w, h, s, seed + 1)
        buf = tlfr.UVTSampleBuffer(records=rec, coc=coc)
        tree = tlfr.TreeGather(buf, _params(case), case["aperture"], case["focus"])
        return {"kind": kind, "tree": tree, "buf": buf, "image": np.empty((h, w, 4), np.float32)}
    rec, coc = _records(case["scene"], w, h, s, seed)
    tree = tlfr.TreeGather(None, _params(case), case["aperture"], case["focus"],
                           device_records=(rec.data_ptr(), (w, h, s), coc))
    state = {"kind": kind, "tree": tree, "records": rec, "image": _image(w, h)}
    if kind == "routed":
        # a network with this scene's standardisation; about half the pixels take the fast path
        feats = torch.empty((h * w, 8), dtype=torch.float32, device="cuda")
        tree.route_features(feats.data_ptr())
        f = feats.cpu().numpy()
        state["router"] = tlfr.Router(0, seed=3, mean=f.mean(0), inv_std=1.0 / np.maximum(f.std(0), 1e-6))
        tree.set_routing(state["router"], 0.5)
    return state


def run(state):
    kind = state["kind"]
    if kind == "network":
        r, f = state["router"], state["feats"].data_ptr()
        r.predict(f, state["pixels"], state["prob"].data_ptr())
        grad, loss = r.gradient(f, state["labels"].data_ptr(), state["rows"])
        return {"prob": state["prob"], "grad": grad, "loss": loss}
    if kind in ("batch", "sweep"):
        state["batch"].run()
        return state["outs"]
    if kind == "host":
        state["tree"].rebuild_from(state["buf"])
        return state["tree"].reconstructDofMotion(state["image"])
    state["tree"].rebuild(state["records"].data_ptr())
    state["tree"].reconstruct_to_device(state["image"].data_ptr())
    return state["image"]


def _query_work(pixels, spp, output_spp):
    """Image written; per output sample the input samples within the dispersion radius reprojected and filtered."""
    accepted = math.pi * _DISPERSION[spp] ** 2 * spp
    return 16.0 * pixels, 40.0 * accepted * pixels * output_spp


def work(case):
    kind = case["kind"]
    if kind == "network":
        # weights are small; forward 2 flops a weight, backward twice that
        weights = 8 * 64 + 64 * 64 + 64
        return {"bytes": case["pixels"] * 36.0 + case["rows"] * 36.0,
                "flops": 2.0 * weights * case["pixels"] + 6.0 * weights * case["rows"]}
    if kind == "batch":
        b = f = 0.0
        for w, h, s in _uneven(case):
            qb, qf = _query_work(w * h, s, 128)
            b += qb + 48.0 * w * h * s
            f += qf
        return {"bytes": b, "flops": f}
    pixels, s = case["width"] * case["height"], case["spp"]
    if kind == "sweep":
        qb, qf = _query_work(pixels, s, 1)
        return {"bytes": case["frames"] * qb + 48.0 * pixels * s, "flops": case["frames"] * qf}
    qb, qf = _query_work(pixels, s, 1 if case["pinhole"] else case["output_spp"])
    # each record read once; about 200 operations a sample to bound and place it
    return {"bytes": 64.0 * pixels * s + qb, "flops": 200.0 * pixels * s + qf}


def exact(case, seed):
    """The network in 64 bits.  A reconstruction has no such value: which samples it
    accepts, how it separates surfaces and in which order it adds are decisions taken
    on 32-bit values, and the images are defined by them."""
    if case["kind"] != "network":
        return None
    s = prepare(case, seed)
    p = s["router"].params().astype(np.float64)
    w1 = p[:1024].reshape(64, 16)[:, :8]
    b1, w2, b2 = p[1024:1088], p[1088:5184].reshape(64, 64), p[5184:5248]
    w3, b3 = p[5248:5312], p[5312]
    mean, inv_std = p[5313:5321], p[5321:5329]
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (w1, b1, w2, b2, w3, mean, inv_std)]
    w1, b1, w2, b2, w3, mean, inv_std = t

    def forward(f):
        x = (f.double() - mean) * inv_std
        h1 = torch.relu(x @ w1.T + b1)
        h2 = torch.relu(h1 @ w2.T + b2)
        return x, h1, h2, torch.sigmoid(h2 @ w3 + b3)

    prob = torch.cat([forward(f)[3] for f in s["feats"][:case["pixels"]].split(1 << 18)])
    n = case["rows"]
    x, h1, h2, q = forward(s["feats"][:n])
    y = s["labels"].double()
    q1 = q.clamp(1e-7, 1 - 1e-7)
    loss = -(y * q1.log() + (1 - y) * (1 - q1).log()).mean()
    dy = (q - y) / n
    d2 = dy[:, None] * w3 * (h2 > 0)
    d1 = (d2 @ w2) * (h1 > 0)
    g1 = torch.zeros((64, 16), dtype=torch.float64, device="cuda")
    g1[:, :8] = d1.T @ x
    grad = torch.cat([g1.reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), dy @ h2, dy.sum()[None]])
    return {"prob": prob, "grad": grad, "loss": float(loss)}
