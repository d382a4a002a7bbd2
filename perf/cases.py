"""Performance cases: the work a user of the renderer has it do, through its
public entry points, from the smallest calls to the largest.

A case is a dict with a "kind":

  tile     sundog_session_render_tile_noalloc: a worker renders a few samples
           of a tile into device memory it owns
  session  Session.render and copy_film: the film of a resident scene on the
           device, as a viewer, a sweep over cameras or a training loop wants it
  denoise  Session.render with AOVs, then Session.denoise: a preview of few
           samples, cleaned up and read back with its AOVs
  oneshot  Scene.render_film: the drop-in render of a scene, from its
           description to the film on the host, nothing resident before it
  serve    Server.submit and Job.wait: a handful of mixed jobs on a server
  guide    sundog_guide_outputs and sundog_guide_gradients: the guiding
           network's mixtures at query points and one training batch's
           loss and gradient

The scenes are the repository's own workloads. A seed sets each render's
random streams and moves its camera a little, so two seeds give other rays.
"""

import ctypes
import math
import shutil
import tempfile

import numpy as np
import torch

from sundog_b200 import abi, scene as sc, serve, workloads

_assets = None


class _Assets(object):
    """A folder for the workloads' .obj / .hdr / image files, removed with
    the process."""

    def __init__(self):
        self.path = tempfile.mkdtemp(prefix="sundog_perf_")

    def __del__(self):
        shutil.rmtree(self.path, ignore_errors=True)


def _asset_dir():
    global _assets
    if _assets is None:
        _assets = _Assets()
    return _assets.path


# Per scene: rays (radiance + shadow) per camera path, and the operations of a
# ray that no structure saves: a root-to-leaf descent of box tests (18
# operations each), the primitive tests at its end and the shading of its
# vertex, with the flame march and the wave normals of the volumes scene.
SCENES = {
    "cornell": (6.0, 1100.0),
    "textured": (3.4, 1200.0),
    "features": (3.6, 1400.0),
    "instancing": (1.9, 1500.0),
    "volumes": (3.6, 4200.0),
}


def _scene(name, seed, width, height, spp):
    d = _asset_dir()
    if name == "cornell":
        s = workloads.cornell(width=width, height=height, spp=spp)
    elif name == "textured":
        s = workloads.textured(d, width=width, height=height, spp=spp)
    elif name == "features":
        s = workloads.features()
        s.render(width=width, height=height, spp=spp)
    elif name == "instancing":
        s = workloads.instancing(d, width=width, height=height, spp=spp)
    else:
        s = workloads.volumes(d, width=width, height=height, spp=spp)
    rng = np.random.default_rng(seed)
    lookfrom, lookat, up, vfov, aperture, focus = s._camera
    lookfrom = [float(v) * float(f) for v, f in zip(lookfrom, rng.uniform(0.98, 1.02, 3))]
    s.camera(lookfrom=lookfrom, lookat=lookat, up=up, vfov=vfov, aperture=aperture,
             focus_dist=focus)
    s.render(seed=int(rng.integers(1, 1 << 31)))
    return s


def listed():
    return [
        # The smallest call: a worker's preview tile of a small scene.
        {"name": "tile_32", "kind": "tile", "scene": "cornell", "size": 32, "spp": 4},
        # An interactive viewport's frame of a small scene: latency counts.
        {"name": "view_96", "kind": "session", "scene": "cornell", "width": 96, "height": 96,
         "spp": 4},
        # The Cornell box at its own size and sample count.
        {"name": "cornell_256", "kind": "session", "scene": "cornell", "width": 256,
         "height": 256, "spp": 16},
        # Every primitive and material at an odd frame size.
        {"name": "features_427x283", "kind": "session", "scene": "features", "width": 427,
         "height": 283, "spp": 9},
        # Image textures and cutouts: a few samples, denoised for a preview.
        {"name": "textured_denoise", "kind": "denoise", "scene": "textured", "width": 960,
         "height": 540, "spp": 4},
        # A thumbnail of the instanced scene at a ragged size.
        {"name": "instancing_333x217", "kind": "session", "scene": "instancing", "width": 333,
         "height": 217, "spp": 5},
        # The instanced scene under the sky at its own size and sample count.
        {"name": "instancing_1080p", "kind": "session", "scene": "instancing", "width": 1920,
         "height": 1080, "spp": 64},
        # Flame, water and glass: a preview, and its own size at an eighth of
        # its samples (a render's time is linear in them from there on).
        {"name": "volumes_640x360", "kind": "session", "scene": "volumes", "width": 640,
         "height": 360, "spp": 8},
        {"name": "volumes_1440p", "kind": "session", "scene": "volumes", "width": 2560,
         "height": 1440, "spp": 32},
        # One drop-in call with nothing resident: scene build, render, film.
        {"name": "oneshot_cornell", "kind": "oneshot", "scene": "cornell", "width": 256,
         "height": 256, "spp": 16},
        # Six jobs of three scenes on one server, small ones among large.
        {"name": "serve_6_jobs", "kind": "serve", "jobs": 6, "size": 512, "spp": 16},
        # The guiding network on one training batch of its default size.
        {"name": "guide_16384", "kind": "guide", "records": 16384},
    ]


# Sizes over which each scene is rendered: (least, most) camera paths of a
# drawn session, up to what the listed frames of that scene take.
_DRAW_PATHS = {
    "cornell": (1 << 12, 1 << 24),
    "textured": (1 << 12, 1 << 23),
    "features": (1 << 12, 1 << 23),
    "instancing": (1 << 14, 1 << 26),
    "volumes": (1 << 14, 1 << 26),
}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["session"] * 6 + ["tile", "denoise", "oneshot", "serve", "guide"])
    if kind == "tile":
        size = _log_int(rng, 8, 64)
        return {"kind": kind, "scene": rng.choice(sorted(SCENES)), "size": size,
                "spp": _log_int(rng, 1, 64)}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(2, 8), "size": _log_int(rng, 128, 640),
                "spp": _log_int(rng, 4, 24)}
    if kind == "guide":
        return {"kind": kind, "records": _log_int(rng, 1024, 32768)}
    scene = rng.choice(sorted(SCENES))
    lo, hi = _DRAW_PATHS[scene]
    if kind == "oneshot":
        hi = min(hi, 1 << 22)
    if kind == "denoise":
        lo, hi = 1 << 16, min(hi, 1 << 23)
    paths = _log_int(rng, lo, hi)
    spp = _log_int(rng, 1, 8 if kind == "denoise" else 64)
    pixels = max(paths // spp, 64)
    width = max(8, min(2560, int(math.sqrt(pixels * rng.uniform(0.8, 2.2)))))
    height = max(8, min(1600, pixels // width))
    return {"kind": kind, "scene": scene, "width": width, "height": height, "spp": spp}


# The kinds of job a server case submits, in turn: a scene and its share of
# the case's edge length and samples.
_JOBS = [("cornell", 0.5, 1.0), ("instancing", 1.0, 1.0), ("volumes", 0.75, 0.5),
         ("cornell", 0.25, 0.25), ("volumes", 0.4, 1.0), ("instancing", 0.3, 0.5),
         ("cornell", 1.0, 0.5), ("instancing", 0.6, 0.25)]


def _job_sizes(case):
    for k in range(case["jobs"]):
        name, edge, share = _JOBS[k % len(_JOBS)]
        size = max(16, int(case["size"] * edge))
        yield name, size, max(8, size * 9 // 16), max(1, int(case["spp"] * share))


# Guiding network: 48 inputs, three hidden layers of 64, 48 outputs (40 used).
_LAYERS = [(64, 48), (64, 64), (64, 64), (48, 64)]
_N_WEIGHTS = sum(o * i for o, i in _LAYERS)
_FREQS, _LOBES = 5, 8


def _guide_inputs(n, seed):
    """Parameters spread like a network in training, queries over the guide
    box, and records with the renderer's mixture of bright and dark."""
    rng = np.random.default_rng(seed)
    p = np.zeros(abi.GUIDE_PARAMS, np.float32)
    at = 0
    for k, (o, i) in enumerate(_LAYERS):
        sd = 0.05 if k == 3 else math.sqrt(2.0 / (35 if k == 0 else i))
        p[at:at + o * i] = rng.standard_normal(o * i) * sd
        at += o * i
    p[at:at + 192] = rng.standard_normal(192) * 0.05
    b3 = p[at + 192:]
    d = 1.0 / math.sqrt(3.0)
    for k in range(_LOBES):
        b3[5 * k:5 * k + 3] = [d if k & 1 else -d, d if k & 2 else -d, d if k & 4 else -d]
        b3[5 * k + 3] = math.log(math.exp(1.95) - 1.0)

    def units(m, near=None):
        v = rng.standard_normal((m, 3))
        if near is not None:
            v += 0.8 * near
        return v / np.linalg.norm(v, axis=1, keepdims=True)

    q = np.concatenate([rng.random((n, 3)), units(n)], 1).astype(np.float32)
    lo, hi = np.array([-2.0, -1.0, -3.0]), np.array([3.0, 2.0, 1.0])
    rec = np.zeros((n, 12), np.float32)
    rec[:, 0:3] = lo + (hi - lo) * rng.random((n, 3))
    rec[:, 3] = rng.exponential(1.0, n) * (rng.random(n) < 0.8) + 1e-3
    rec[:, 4:7] = units(n)
    rec[:, 8:11] = units(n, rec[:, 4:7])
    box = np.concatenate([lo, 1.0 / (hi - lo)]).astype(np.float32)
    return p, q, rec, box


def prepare(case, seed):
    lib = abi.load()
    kind = case["kind"]
    if kind == "guide":
        n = case["records"]
        p, q, rec, box = _guide_inputs(n, seed)
        return {"case": case, "lib": lib, "params": p, "queries": q, "records": rec, "box": box,
                "outputs": np.zeros((n, 40), np.float32),
                "grads": np.zeros(abi.GUIDE_PARAMS, np.float32)}
    if kind == "serve":
        jobs = [(_scene(name, seed * 16 + k, w, h, spp), dict(width=w, height=h, spp=spp))
                for k, (name, w, h, spp) in enumerate(_job_sizes(case))]
        return {"case": case, "server": serve.Server(), "jobs": jobs}
    if kind == "oneshot":
        return {"case": case, "scene": _scene(case["scene"], seed, case["width"], case["height"],
                                              case["spp"])}
    if kind == "tile":
        # A tile of a 256x256 frame of 64 samples, at an offset of its own.
        frame = 256
        s = _scene(case["scene"], seed, frame, frame, 64)
        rng = np.random.default_rng(seed + 1)
        span = frame - case["size"]
        return {"case": case, "lib": lib, "session": sc.Session(s, base_dir=_asset_dir()),
                "x0": int(rng.integers(0, span + 1)), "y0": int(rng.integers(0, span + 1)),
                "film": torch.zeros(case["size"], case["size"], 4, device="cuda")}
    s = _scene(case["scene"], seed, case["width"], case["height"], case["spp"])
    aov = kind == "denoise"
    return {"case": case, "session": sc.Session(s, base_dir=_asset_dir(), aov=aov),
            "film": None if aov else torch.zeros(case["height"], case["width"], 4, device="cuda")}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "session":
        ses, film = state["session"], state["film"]
        ses.render()
        ses.copy_film(film.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return film
    if kind == "tile":
        ses, lib, film = state["session"], state["lib"], state["film"]
        film.zero_()
        abi.check(lib.sundog_session_render_tile_noalloc(
            ses.handle, state["x0"], state["y0"], case["size"], case["size"], 0, case["spp"],
            film.data_ptr(), None, torch.cuda.current_stream().cuda_stream), "tile", lib)
        return film
    if kind == "denoise":
        ses = state["session"]
        ses.render()
        film, albedo, normal = ses.read()
        return {"denoised": ses.denoise(), "film": film, "albedo": albedo, "normal": normal}
    if kind == "oneshot":
        return state["scene"].render_film(_asset_dir())[0]
    if kind == "serve":
        jobs = [state["server"].submit(s, base_dir=_asset_dir(), **o) for s, o in state["jobs"]]
        return [j.wait() for j in jobs]
    lib, n = state["lib"], case["records"]
    abi.check(lib.sundog_guide_outputs(state["params"].ctypes.data, state["queries"].ctypes.data, n,
                                       state["outputs"].ctypes.data), "guide outputs", lib)
    loss = ctypes.c_float(0.0)
    abi.check(lib.sundog_guide_gradients(state["params"].ctypes.data, state["records"].ctypes.data,
                                         n, state["box"].ctypes.data, state["grads"].ctypes.data,
                                         ctypes.byref(loss)), "guide gradients", lib)
    return {"outputs": state["outputs"], "grads": state["grads"], "loss": float(loss.value)}


def work(case):
    """What a pass cannot do without: each film written once (16 bytes a
    pixel) and the operations of its rays; the network's matrix products."""
    kind = case["kind"]
    if kind == "guide":
        n = case["records"]
        # Forward twice (outputs and the batch), and the batch's backward:
        # weight gradients and the three hidden gradients.
        fwd = 2.0 * _N_WEIGHTS
        bwd = fwd + 2.0 * sum(o * i for o, i in _LAYERS[1:])
        return {"bytes": n * (24 + 160 + 48) + 8.0 * abi.GUIDE_PARAMS,
                "flops": n * (2 * fwd + bwd)}
    if kind == "serve":
        paths = [(name, w * h, spp) for name, w, h, spp in _job_sizes(case)]
    elif kind == "tile":
        paths = [(case["scene"], case["size"] ** 2, case["spp"])]
    else:
        paths = [(case["scene"], case["width"] * case["height"], case["spp"])]
    flops = sum(SCENES[name][0] * SCENES[name][1] * px * spp for name, px, spp in paths)
    px = sum(p for _, p, _ in paths)
    if kind == "denoise":
        # Film, two AOVs and the denoised film; four passes of 25 taps.
        return {"bytes": 64.0 * px, "flops": flops + px * 4 * 25 * 30.0}
    return {"bytes": 16.0 * px, "flops": flops}


def _unflatten(p):
    W, at = [], 0
    for o, i in _LAYERS:
        W.append(p[at:at + o * i].reshape(o, i))
        at += o * i
    b = []
    for o, _ in _LAYERS:
        b.append(p[at:at + o])
        at += o
    return W, b


def _forward(p, pos, nrm):
    f = torch.zeros(pos.shape[0], 48, dtype=torch.float64)
    for i in range(3):
        for j in range(_FREQS):
            v = math.pi * pos[:, i] * (1 << j)
            f[:, 10 * i + 2 * j] = torch.sin(v)
            f[:, 10 * i + 2 * j + 1] = torch.cos(v)
    f[:, 32:35] = nrm
    W, b = _unflatten(p)
    for k in range(3):
        f = torch.relu(f @ W[k].T + b[k])
    return f @ W[3].T + b[3]


def exact(case, seed):
    """The guiding network in 64 bits: its outputs, and the loss
    sum_i -c_i log q(w_i), c_i = min(F_i / mean F, 100) / n, q the mixture of
    von Mises-Fisher lobes, with its gradient. A path-traced film has no such
    value: rounding decides which way a path goes."""
    if case["kind"] != "guide":
        return None
    params, q, rec, box = _guide_inputs(case["records"], seed)
    p = torch.tensor(params, dtype=torch.float64, requires_grad=True)
    q, rec, box = (torch.tensor(a, dtype=torch.float64) for a in (q, rec, box))
    with torch.no_grad():
        outputs = _forward(p, q[:, :3], q[:, 3:])[:, :40]
    pos = ((rec[:, :3] - box[:3]) * box[3:]).clamp(0.0, 1.0)
    o = _forward(p, pos, rec[:, 4:7])[:, :40].reshape(-1, _LOBES, 5)
    mu = o[..., :3] / o[..., :3].norm(dim=-1, keepdim=True).clamp_min(1e-4)
    kappa = (torch.nn.functional.softplus(o[..., 3]) + 0.05).clamp_max(500.0)
    cosm = (mu * rec[:, None, 8:11]).sum(-1)
    norm = kappa.log() - math.log(2.0 * math.pi) - torch.log1p(-torch.exp(-2.0 * kappa))
    logq = torch.logsumexp(torch.log_softmax(o[..., 4], -1) + norm + kappa * (cosm - 1.0), -1)
    c = (rec[:, 3] / rec[:, 3].mean()).clamp_max(100.0) / rec.shape[0]
    loss = -(c * logq).sum()
    loss.backward()
    return {"outputs": outputs, "grads": p.grad, "loss": float(loss.detach())}
