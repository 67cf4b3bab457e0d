"""Performance cases of visualtur_b200: what a program that uses the ray
caster spends its time on, through the package's public entry points.

`listed()` names the standing cases, `draw(rng)` makes more of the same
ranges.  `prepare(case, seed)` makes what the program holds before the call
(volume, octree, renderer, network, camera path), `run(state)` is one pass,
`work(case)` the bytes and operations the pass cannot do without and
`exact(case, seed)` the pass's result in 64 bits where one can be had without
the library.  Volumes are the library's seeded generators at the proportions
of the benchmark workloads (blobs, noisy sphere, uint8 fractal).

Kinds of case:
  frame    one view per call (visualTur.updateVisibleCubes), every brick or
           the whole volume on the device
  views    many views of mixed sizes per call (visualTur.render_batch)
  path     a fly-through from a cold or too small brick cache
  octree   building the octree file of a volume on the device
  train    training steps of the prefetch network, then its weights
  forward  predictions of the prefetch network
  cube     rayCaster.renderCube of a single brick
"""
import math
import os
import random
import shutil
import tempfile

import numpy as np
import torch

import visualtur_b200 as vt
from visualtur_b200 import prefetch as pf

LIGHT = (0.0, 512.0, 0.0)      # the renderer's light
RATE = 2e-5                    # a late learning rate: the network stays near its start however often a stretch is run
FOV, DIST = 30.0, 50.0         # half-angle in degrees, screen distance
VIEW_SIZES = ((256, 256), (512, 512), (1024, 1024), (1920, 1080))


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a preview window on a small scalar field: the shortest call a viewer makes
        dict(name="frame_preview", kind="frame", gen="sphere", nx=64, ny=64, nz=64, node=4, brick=8, resident=1,
             W=96, H=96, r=2.4, refine=0, persistent=0),
        # the resident benchmark scene: 128^3 noisy sphere at 512 x 512
        dict(name="frame_resident", kind="frame", gen="sphere", nx=128, ny=128, nz=128, node=4, brick=8, resident=1,
             W=512, H=512, r=2.4, refine=0, persistent=0),
        # an interactive full-HD viewer with the default options, bricks on the device
        dict(name="frame_hd", kind="frame", gen="blobs", nx=512, ny=512, nz=512, node=4, brick=16, resident=0,
             W=1920, H=1080, r=1.5, refine=0, persistent=0),
        # uint8 data of ragged extents, odd screen, bisection refinement, the camera near the data
        dict(name="frame_u8_ragged", kind="frame", gen="fractal", nx=401, ny=290, nz=333, node=4, brick=32, resident=0,
             W=1277, H=719, r=0.8, refine=5, persistent=1),
        # offline rendering: 16 views of mixed sizes in one call
        dict(name="views_mixed", kind="views", gen="blobs", nx=512, ny=512, nz=512, node=4, brick=16, views=16, r=1.5,
             size=0),
        # a fly-through's first frames: everything paged in from a cold cache, no lookahead
        dict(name="path_cold", kind="path", gen="blobs", nx=512, ny=512, nz=512, node=4, brick=16, frames=8, batch=4,
             W=960, H=540, r=1.5, share=1.0, cold=1, skip=0, lookahead=0),
        # steady paging: uint8 fractal surfaces, the device cache smaller than the path needs
        dict(name="path_paging", kind="path", gen="fractal", nx=512, ny=512, nz=512, node=4, brick=32, frames=8, batch=2,
             W=960, H=540, r=0.9, share=0.5, cold=0, skip=2, lookahead=2),
        # a new data set is opened: its octree
        dict(name="octree_f32", kind="octree", gen="blobs", nx=512, ny=512, nz=512),
        dict(name="octree_u8_ragged", kind="octree", gen="fractal", nx=201, ny=333, nz=129),
        # the prefetch network: one stretch of training, and the poses of the coming frames
        dict(name="train_256", kind="train", batch=256, steps=16, hidden=512, out=4096),
        dict(name="forward_8", kind="forward", batch=8, hidden=512, out=4096),
        # one brick in a brick viewer
        dict(name="cube_512", kind="cube", edge=32, W=512, H=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "views", "path", "octree", "octree", "train", "forward", "cube"])
    if kind == "train":
        return dict(kind=kind, batch=_log(rng, 16, 512), steps=rng.randint(4, 16), hidden=_log(rng, 96, 512),
                    out=rng.choice([512, 4096]))
    if kind == "forward":
        return dict(kind=kind, batch=_log(rng, 1, 512), hidden=_log(rng, 96, 512), out=rng.choice([512, 4096]))
    if kind == "cube":
        return dict(kind=kind, edge=_log(rng, 8, 64), W=_log(rng, 64, 1024), H=_log(rng, 64, 1024))
    gen = rng.choice(["sphere", "blobs", "fractal"])
    # cubes and boxes of any extents: the longest side over 48..512, the others down to half of it
    n = _log(rng, 48, 512)
    nx, ny, nz = (n, n, n) if rng.random() < 0.3 else [max(33, int(n * rng.uniform(0.5, 1.0))) for _ in range(3)]
    c = dict(kind=kind, gen=gen, nx=nx, ny=ny, nz=nz)
    if kind == "octree":
        return c
    c.update(node=rng.choice([2, 4, 4, 4, 8]), brick=rng.choice([8, 16, 16, 32]), r=round(rng.uniform(0.3, 2.5), 3))
    c["node"] = min(c["node"], c["brick"])
    if kind == "frame":
        c.update(resident=rng.choice([0, 0, 1]), W=_log(rng, 64, 1920), H=_log(rng, 64, 1080),
                 refine=rng.choice([0, 0, 0, 5]), persistent=rng.choice([0, 1]))
    elif kind == "views":
        c.update(views=rng.randint(2, 16), size=_log(rng, 64, 1024))
    else:
        cold = rng.choice([0, 1])
        c.update(frames=rng.randint(2, 8), batch=rng.choice([1, 2, 4]), W=_log(rng, 160, 960), H=_log(rng, 120, 540),
                 share=1.0 if cold else round(rng.uniform(0.5, 0.9), 2), cold=cold, skip=rng.choice([0, 0, 2]),
                 lookahead=rng.choice([0, 2]))
    return c


# ------------------------------------------------------------------ inputs
def _iso(case):
    if case["gen"] == "sphere":
        return 0.3125 * max(case["nx"], case["ny"], case["nz"])
    return 0.6 if case["gen"] == "blobs" else 128.0


def _device_volume(case, seed):
    dims = (case["nx"], case["ny"], case["nz"])
    n = float(max(dims))
    u8 = case["gen"] == "fractal"
    vol = torch.empty(dims, dtype=torch.uint8 if u8 else torch.float32, device="cuda")
    kind, prm = {
        "sphere": (vt.VT_GEN_SPHERE, ((dims[0] - 1) / 2, (dims[1] - 1) / 2, (dims[2] - 1) / 2, 0.25)),
        "blobs": (vt.VT_GEN_BLOBS, (256, n / 102.4, n / 17.0667, 0.5, 1.5, 0.05)),
        "fractal": (vt.VT_GEN_FRACTAL_U8, (32, n / 81.92, n / 10.24, 200.0)),
    }[case["gen"]]
    vt.generate_volume(kind, 1000 + int(seed), dims, prm, device_ptr=vol.data_ptr())
    return vol


def _build_octree(vol, iso, path):
    vt.build_octree_device(vol.data_ptr(), vt.VT_U8 if vol.dtype == torch.uint8 else vt.VT_F32, vol.shape, iso, path)


def _scene(case, seed):
    vol = _device_volume(case, seed)
    d = tempfile.mkdtemp()
    try:
        path = os.path.join(d, "v.oct")
        _build_octree(vol, _iso(case), path)
        oc = vt.Octree(path)
    finally:
        shutil.rmtree(d)
    return vt.FileManager.wrap(vol.cpu().numpy()), oc


def _bricks_of(oc, level):
    """bricks of `level` that hold parts of the surface"""
    e = oc.level(level).reshape(-1, 2)
    return int((e[:, 1] - e[:, 0] + np.uint64(1)).sum())


def _renderer(case, fm, oc, W, H, dev, host, **opt):
    levelO = max(1, oc.nLevels - int(math.log2(case["node"])))
    levelC = min(levelO, max(0, oc.nLevels - int(math.log2(case["brick"]))))
    p = vt.make_params(W=W, H=H, octreeFile=None, hdf5File=None, octreeLevel=levelO, levelCubes=levelC,
                       dimCube=1 << (oc.nLevels - levelC), distance=DIST, fov_H=FOV, fov_W=FOV, maxElementsCache=dev,
                       maxElementsCache_CPU=host)
    return vt.visualTur(p, vt.default_options(**opt), volume=fm, octree=oc)


def _brick_level(case, oc):
    return max(0, oc.nLevels - int(math.log2(case["brick"])))


def _cameras(case, seed, sizes):
    """Cameras at `r` volume extents from the centre, on an orbit of 1.2
    degrees a view from a seeded start, looking near the centre."""
    rng = np.random.RandomState(77 + int(seed))
    dims = np.array([case["nx"], case["ny"], case["nz"]], float)
    c, n = (dims - 1) / 2, dims.max()
    a0, tilt, off = rng.uniform(0, 2 * math.pi), rng.uniform(-0.5, 0.5), rng.uniform(-0.05, 0.05, 3) * n
    out = []
    for k, (W, H) in enumerate(sizes):
        a = a0 + math.radians(1.2) * k
        pos = c + case["r"] * n * np.array([math.cos(a) * math.cos(tilt), math.sin(tilt), math.sin(a) * math.cos(tilt)])
        out.append(pf.look_at(W, H, DIST, FOV, pos, c + off))
    return out


def _network(case, seed):
    rng = np.random.RandomState(5 + int(seed))
    d = (12, case["hidden"], case["hidden"], case["out"])
    layers = [((rng.standard_normal((d[l], d[l + 1])) * math.sqrt(2.0 / d[l])).astype(np.float32),
               (rng.standard_normal(d[l + 1]) * 0.1).astype(np.float32)) for l in range(3)]
    return d, layers, rng


def _poses(rng, n):
    """pose features as the renderer's cameras give them"""
    x = np.empty((n, 12), np.float32)
    v = rng.standard_normal((n, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    r = rng.uniform(1.2, 1.7, (n, 1))
    x[:, 0:3], x[:, 3:6] = v * r, -v
    u = np.cross(np.cross(-v, (0.0, 1.0, 0.0)), -v)
    x[:, 6:9] = u / np.linalg.norm(u, axis=1, keepdims=True)
    x[:, 9] = FOV / 90.0
    x[:, 10:11], x[:, 11:12] = np.maximum(r - 0.866, 0), r + 0.866
    return x


def _targets(rng, x, out):
    """nodes on the camera's side of a random plane each: about a quarter of them"""
    proj = rng.standard_normal((12, out))
    z = x @ proj
    return (z > np.quantile(z[:256], 0.75)).astype(np.float32)


def _train_data(case, seed):
    d, layers, rng = _network(case, seed)
    n = case["batch"] * case["steps"]
    x = _poses(rng, n)
    return d, layers, x, _targets(rng, x, case["out"])


def _cube(case, seed):
    rng = np.random.RandomState(11 + int(seed))
    D = case["edge"] + 6
    g = np.arange(D, dtype=np.float32) - (D - 1) / 2
    v = np.sqrt(g[:, None, None] ** 2 + g[None, :, None] ** 2 + g[None, None, :] ** 2)
    v = (v + 0.25 * rng.standard_normal((D, D, D))).astype(np.float32)
    cam = vt.Camera(case["H"], case["W"], DIST, FOV, FOV)
    e = case["edge"]
    cam.Move((100.0 + e / 2 + rng.uniform(-1, 1), 60.0 + e / 2 + rng.uniform(-1, 1), 40.0 + 2.4 * e + rng.uniform(0, 1)))
    return v, cam, (100, 60, 40), 0.3125 * e


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "octree":
        s["vol"], s["dir"] = _device_volume(case, seed), tempfile.TemporaryDirectory()
        # the file's bytes, in room enough for any surface of this volume
        s["file"] = np.zeros((1 << 16) + case["nx"] * case["ny"] * case["nz"] // 2, np.uint8)
        return s
    if kind in ("train", "forward"):
        if kind == "train":
            d, layers, x, y = _train_data(case, seed)
            s["y"] = torch.from_numpy(y).cuda()
        else:
            d, layers, rng = _network(case, seed)
            x = _poses(rng, case["batch"])
            s["p"] = torch.empty(case["batch"], case["out"], device="cuda")
        s["net"] = vt.MLP(d, seed=1)
        s["net"].set_weights(layers)
        s["x"] = torch.from_numpy(x).cuda()
        return s
    if kind == "cube":
        v, cam, s["min"], iso = _cube(case, seed)
        s["cam"], s["rc"], s["cube"] = cam, vt.rayCaster(iso, LIGHT), torch.from_numpy(v).cuda()
        s["rgba"] = torch.empty(case["H"] * case["W"], 4, device="cuda")
        return s
    fm, oc = _scene(case, seed)
    bricks = max(16, _bricks_of(oc, _brick_level(case, oc)))
    if kind == "frame":
        W, H = case["W"], case["H"]
        s["r"] = _renderer(case, fm, oc, W, H, bricks, bricks, resident=case["resident"], refine=case["refine"],
                           persistent=case["persistent"])
        s["r"].set_camera(_cameras(case, seed, [(W, H)])[0])
        s["rgba"] = torch.empty(H * W, 4, device="cuda")
        s["rgb8"] = torch.empty(H * W, 3, dtype=torch.uint8, device="cuda")
        return s
    if kind == "views":
        rng = random.Random(3)
        sizes = [rng.choice(VIEW_SIZES) if case["size"] == 0 else
                 (max(48, int(case["size"] * rng.uniform(0.4, 1))), max(48, int(case["size"] * rng.uniform(0.4, 1))))
                 for _ in range(case["views"])]
        opt = dict(lookahead=0, skip=0, preload=1)
        dev = bricks
    else:
        sizes = [(case["W"], case["H"])] * case["frames"]
        opt = dict(lookahead=case["lookahead"], skip=case["skip"], preload=0)
        dev = max(16, int(bricks * case["share"]))
    s["r"] = _renderer(case, fm, oc, sizes[0][0], sizes[0][1], dev, bricks, persistent=1, record_hits=0, **opt)
    s["stream"] = torch.cuda.Stream()
    s["out"] = [torch.empty(W * H, 3, dtype=torch.uint8, device="cuda") for W, H in sizes]
    s["views"] = []
    for cam, o in zip(_cameras(case, seed, sizes), s["out"]):
        v = vt.vt_view()
        v.cam, v.dev_rgba, v.dev_rgb8 = cam, None, o.data_ptr()
        s["views"].append(v)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        s["r"].updateVisibleCubes(s["rgba"], s["rgb8"])
        return [s["rgba"], s["rgb8"]]
    if kind == "views":
        s["r"].render_batch(s["views"], stream=s["stream"].cuda_stream)
        return s["out"]
    if kind == "path":
        if case["cold"]:
            s["r"].drop_cache()
        for i in range(0, case["frames"], case["batch"]):
            s["r"].render_batch(s["views"][i:i + case["batch"]], stream=s["stream"].cuda_stream)
        return s["out"]
    if kind == "octree":
        path = os.path.join(s["dir"].name, "v.oct")
        _build_octree(s["vol"], _iso(case), path)
        with open(path, "rb") as f:
            return [f.readinto(s["file"]), s["file"]]
    if kind == "train":
        b = case["batch"]
        for i in range(case["steps"]):
            s["net"].train_step(s["x"][i * b:(i + 1) * b], s["y"][i * b:(i + 1) * b], b, RATE, want_loss=False)
        return s["net"].weights()
    if kind == "forward":
        s["net"].forward(s["x"], case["batch"], s["p"])
        return s["p"]
    e = case["edge"]
    s["rc"].renderCube(s["cam"], s["cube"], s["min"], (e, e, e), (3, 3, 3), s["rgba"])
    return s["rgba"]


# ------------------------------------------------------------------ work
def work(case):
    """Frames: every pixel is written once, and a visible surface point costs
    the 8 voxels around it (at most the whole volume) and a sample, a normal
    and the shading (about 250 operations)."""
    kind = case["kind"]
    if kind in ("train", "forward"):
        h, o, b = case["hidden"], case["out"], case["batch"]
        par = 12 * h + h * h + h * o + 2 * h + o
        if kind == "forward":
            return {"bytes": 2 * par + 4 * b * (12 + o), "flops": 2 * b * par}
        # per step: masters and both moments read and written, inputs and targets read
        return {"bytes": case["steps"] * (24 * par + 4 * b * (12 + o)) + 4 * par, "flops": case["steps"] * 6 * b * par}
    if kind == "cube":
        pix = case["W"] * case["H"]
        return {"bytes": 16 * pix + 4 * (case["edge"] + 6) ** 3, "flops": 250 * pix}
    es = 1 if case["gen"] == "fractal" else 4
    vol = es * case["nx"] * case["ny"] * case["nz"]
    if kind == "octree":
        return {"bytes": vol, "flops": 8 * case["nx"] * case["ny"] * case["nz"]}
    if kind == "frame":
        pix, out = case["W"] * case["H"], 19
    elif kind == "views":
        side = 1024 * 1024 if case["size"] == 0 else 0.49 * case["size"] ** 2
        pix, out = int(case["views"] * side), 3
    else:
        pix, out = case["frames"] * case["W"] * case["H"], 3
    return {"bytes": out * pix + min(vol, 8 * es * pix), "flops": 250 * pix}


# ------------------------------------------------------------------ exact
def exact(case, seed):
    kind = case["kind"]
    if kind == "forward":
        d, layers, rng = _network(case, seed)
        return _net64(layers, torch.from_numpy(_poses(rng, case["batch"])).cuda().double())[-1]
    if kind == "train":
        return _train64(case, seed)
    if kind == "cube":
        return _cube64(case, seed)
    if kind == "frame" and case["gen"] == "sphere" and max(case["nx"], case["ny"], case["nz"]) <= 128 \
            and case["W"] * case["H"] <= 512 * 512 and not case["refine"]:
        return [_frame64(case, seed), None]
    return None     # bytes, or a picture that takes plain tensor code minutes


def _net64(layers, x):
    acts = [x]
    for l, (w, b) in enumerate(layers):
        w, b = (t if torch.is_tensor(t) else torch.from_numpy(t).cuda().double() for t in (w, b))
        z = acts[-1] @ w + b
        acts.append(torch.relu(z) if l < 2 else torch.sigmoid(z))
    return acts


def _train64(case, seed):
    """Adam (0.9, 0.999, 1e-8) on the mean over the batch of the summed
    binary cross-entropy."""
    d, layers, x, y = _train_data(case, seed)
    P = [torch.from_numpy(t).cuda().double() for wb in layers for t in wb]
    M, V = [torch.zeros_like(p) for p in P], [torch.zeros_like(p) for p in P]
    x, y = torch.from_numpy(x).cuda().double(), torch.from_numpy(y).cuda().double()
    b = case["batch"]
    for k in range(case["steps"]):
        xs, ys = x[k * b:(k + 1) * b], y[k * b:(k + 1) * b]
        acts = _net64([(P[0], P[1]), (P[2], P[3]), (P[4], P[5])], xs)
        G, dz = [None] * 6, (acts[3] - ys) / b
        for l in (2, 1, 0):
            G[2 * l], G[2 * l + 1] = acts[l].T @ dz, dz.sum(0)
            if l:
                dz = (dz @ P[2 * l].T) * (acts[l] > 0)
        for i, g in enumerate(G):
            M[i] = 0.9 * M[i] + 0.1 * g
            V[i] = 0.999 * V[i] + 0.001 * g * g
            P[i] = P[i] - RATE * (M[i] / (1 - 0.9 ** (k + 1))) / ((V[i] / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return [(P[0], P[1]), (P[2], P[3]), (P[4], P[5])]


def _rays64(c):
    f = lambda v: torch.tensor(list(v), dtype=torch.float64, device="cuda")  # noqa: E731
    i = torch.arange(c.H, dtype=torch.float64, device="cuda")[:, None, None]
    j = torch.arange(c.W, dtype=torch.float64, device="cuda")[None, :, None]
    d = f(c.look) * c.distance + f(c.up) * (-c.h / 2 + c.h / c.H * (i + 0.5)) + f(c.right) * (-c.w / 2 + c.w / c.W * (j + 0.5))
    d = d.reshape(-1, 3)
    return f(c.position), d / d.norm(dim=1, keepdim=True)


def _slab64(o, d, lo, hi):
    a, b = (lo - o) / d, (hi - o) / d
    tn, tf = torch.minimum(a, b).amax(-1), torch.maximum(a, b).amin(-1)
    return tn.clamp(min=0), tf, (tn <= tf) & (tf >= 0)


def _tri64(get, p):
    r = torch.trunc(p)
    f, i = p - r, r.long()
    v = 0
    for k in range(8):
        e = torch.tensor([(k >> 2) & 1, (k >> 1) & 1, k & 1], device=p.device)
        w = torch.where(e.bool(), f, 1 - f).prod(-1)
        v = v + w * get(i + e)
    return v


def _march64(get, o, d, tn, steps, iso, most):
    """first crossing along d from o + tn d in half-unit steps: (point, found)"""
    X = o + d * tn[:, None]
    last, at, found = _tri64(get, X), X.clone(), torch.zeros(len(X), dtype=torch.bool, device=X.device)
    alive = steps >= 0
    P = X.clone()
    for k in range(1, most + 1):
        X = X + 0.5 * d
        go = alive & ~found & (k <= steps)
        if not bool(go.any()):
            break
        v = _tri64(get, X)
        same = ((iso - last < 0) & (iso - v < 0)) | ((iso - last > 0) & (iso - v > 0))
        hit = go & ~same
        a = ((iso - last) / (v - last))[:, None]
        at = torch.where(hit[:, None], P * (1 - a) + X * a, at)
        found = found | hit
        P = torch.where((go & same)[:, None], X, P)
        last = torch.where(go & same, v, last)
    return at, found


def _shade64(get, X, scale):
    g = []
    for a in range(3):
        e = torch.zeros(3, dtype=torch.float64, device=X.device)
        e[a] = 1.0
        g.append((_tri64(get, X - e) - _tri64(get, X + e)) / 2)
    n = torch.stack(g, 1)
    n = n / n.norm(dim=1, keepdim=True)
    l = X - torch.tensor(LIGHT, dtype=torch.float64, device=X.device)
    dif = (n * l / l.norm(dim=1, keepdim=True)).sum(1).abs()
    a = X[:, 1] / scale
    return torch.stack([(1 - a) * dif, a * dif, 0 * dif, torch.ones_like(dif)], 1)


def _cube64(case, seed):
    v, cam, mn, iso = _cube(case, seed)
    e = case["edge"]
    D = e + 6
    flat = torch.from_numpy(v).cuda().double().reshape(-1)
    lo = torch.tensor(mn, dtype=torch.float64, device="cuda")

    def get(i):     # the brick's own linear addressing; zero outside its allocation
        k = i - (lo.long() - 3)
        q = k[:, 2] + k[:, 1] * D + k[:, 0] * D * D
        return torch.where((q >= 0) & (q < D ** 3), flat[q.clamp(0, D ** 3 - 1)], 0.0)
    o, d = _rays64(cam.c)
    tn, tf, hit = _slab64(o, d, lo, lo + e)
    out = torch.ones(len(d), 4, dtype=torch.float64, device="cuda")
    on = hit.nonzero()[:, 0]
    steps = torch.floor((tf - tn)[on] * 2)
    X, found = _march64(get, o, d[on], tn[on], steps, iso, int(steps.max()) if len(on) else 0)
    if bool(found.any()):
        out[on[found]] = _shade64(get, X[found], float(e))
    return out


def _frame64(case, seed):
    """Every ray against every candidate node of the surface, nearest first."""
    vol = _device_volume(case, seed).double()
    iso, dims = _iso(case), vol.shape
    levels = max(1, math.ceil(math.log2(max(dims))))
    N, pad = 1 << levels, 4
    full = torch.zeros([N + 2 * pad] * 3, dtype=torch.float64, device="cuda")
    full[pad:pad + dims[0], pad:pad + dims[1], pad:pad + dims[2]] = vol
    neg = (full[pad:, pad:, pad:] - iso) < 0
    cell = neg[:N, :N, :N]
    has = torch.zeros_like(cell)
    for k in range(1, 8):
        x, y, z = (k >> 2) & 1, (k >> 1) & 1, k & 1
        has |= neg[x:x + N, y:y + N, z:z + N] != cell
    node = min(case["node"], N // 2)
    m = N // node
    has = has.reshape(m, node, m, node, m, node).any(5).any(3).any(1)
    has[m // 2:, m // 2:, m // 2:] = False      # the file format leaves out each level's last node: no far octant
    lo = has.nonzero().double() * node

    def get(i):
        q = (i + pad).clamp(0, N + 2 * pad - 1)
        return full[q[:, 0], q[:, 1], q[:, 2]]
    o, dirs = _rays64(_cameras(case, seed, [(case["W"], case["H"])])[0])
    out = torch.ones(len(dirs), 4, dtype=torch.float64, device="cuda")
    for c0 in range(0, len(dirs), 4096):
        d = dirs[c0:c0 + 4096]
        tn, tf, hit = _slab64(o, d[:, None, :], lo[None], lo[None] + node)
        order = torch.where(hit, tn + 1e-9 * tf, torch.inf)
        k = min(int(hit.sum(1).max()), len(lo))
        if k == 0:
            continue
        key, idx = order.topk(k, dim=1, largest=False)
        done = torch.zeros(len(d), dtype=torch.bool, device="cuda")
        for q in range(k):
            on = (~done & torch.isfinite(key[:, q])).nonzero()[:, 0]
            if not len(on):
                break
            a = tn[on, idx[on, q]]
            steps = torch.ceil((tf[on, idx[on, q]] - a) * 2)
            X, found = _march64(get, o, d[on], a, steps, iso, int(steps.max()))
            if bool(found.any()):
                out[c0 + on[found]] = _shade64(get, X[found], 256.0)
                done[on[found]] = True
    return out
