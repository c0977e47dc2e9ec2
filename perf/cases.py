"""Performance cases of the ORB front-end: what a user's program calls, at the sizes it calls it with.

A case is one call (or the two or three calls that follow one another in a tracker) of the package's public entry
points, from single camera frames through batches of frames to the large descriptor searches.  The sizes are those
of this repository's benchmark and tests -- 640x480, 752x480, 1241x376 and 1280x720 frames with 1000 to 2000 features,
64-frame batches, a 50,000 x 200,000 kNN, a million map points, a vocabulary of ten children and six levels -- with odd
ones beside them; draw() spreads the same kinds over their ranges.

Every input comes from the seed.  Images are scenes of filled rectangles and ellipses under smoothed noise, second views
are small homographies or disparities of the first with noise, map points are noisy copies of frame features.
"""
import functools
import math

import numpy as np
import torch

from orb_slam2_detailed_comments_gb300 import (FRAME_MAPPOINT_DTYPE, FRUSTUM_FRAME_DTYPE, MAPPOINT_DTYPE, FrameView,
                                               ORBextractor, ORBmatcher, Vocabulary, compute_distinctive_descriptors,
                                               compute_stereo_matches, frustum_frame, is_in_frustum, search_by_bow)
from orb_slam2_detailed_comments_gb300 import synthetic
from orb_slam2_detailed_comments_gb300.batch import (BatchExtractor, BatchFrameProjection, BatchProjection, BatchStereo,
                                                     motion_struct)

DEV = "cuda"
SCALE, LEVELS = 1.2, 8
RESOLUTIONS = ((640, 480), (752, 480), (1241, 376), (1280, 720))
BF, FX = 386.1, 718.856  # stereo baseline times focal length, focal length


# ------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: one camera image on the host, keypoints and descriptors back on the host
        {"name": "frame_640x480", "kind": "frame", "w": 640, "h": 480, "nf": 1000, "ini": 20, "device": False},
        # monocular initialisation: the first two frames' level-0 keypoints within 100 px
        {"name": "init_640x480", "kind": "init", "w": 640, "h": 480, "nf": 1000, "window": 100},
        # one stereo frame of a car camera: both extractions on the device and the stereo matches
        {"name": "stereo_1241x376", "kind": "stereo", "w": 1241, "h": 376, "nf": 2000, "ini": 20},
        # one tracked frame: extraction, then the local map's 3000 points searched in it
        {"name": "track_1280x720", "kind": "track", "w": 1280, "h": 720, "nf": 2000, "ini": 20, "m": 3000},
        # a rig of five cameras with odd image sizes, each frame against its previous one (motion model)
        {"name": "rig_5_odd", "kind": "rig", "frames": 5, "sizes": "637x479,751x481,1239x375,611x457,853x479", "nf": 1201,
         "ini": 20},
        # many cameras at once: 64 frames of mixed sizes, 3000 map points searched in each
        {"name": "batch_64_mixed", "kind": "batch", "frames": 64, "sizes": "mixed", "nf": 0, "ini": 20, "m": 3000},
        # recorded stereo sequences: 32 pairs in one extraction, then all pairs' stereo matches
        {"name": "batch_stereo_32", "kind": "batch_stereo", "pairs": 32, "w": 1241, "h": 376, "nf": 2000, "ini": 20},
        # two frames' descriptors against each other, all pairs
        {"name": "knn_1999x2003", "kind": "knn", "nq": 1999, "nt": 2003, "algo": 0, "centres": 0},
        # a descriptor database: queries against a large clustered set, ratio test, the kernel left to the library
        {"name": "knn_50k_200k", "kind": "knn", "nq": 50000, "nt": 200000, "algo": -1, "centres": 2000},
        # a whole map's points: the distinctive descriptor of each
        {"name": "distinctive_1m", "kind": "distinctive", "m": 1000000, "mean": 6.0},
        # place recognition: the word and feature vectors of 64 frames, then 32 keyframe / frame pairs matched by node
        {"name": "bow_64x2000", "kind": "bow", "frames": 64, "per": 2000, "pairs": 32},
        # the local map of 64 frames tested against their view frusta
        {"name": "frustum_64x5000", "kind": "frustum", "frames": 64, "per": 5000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng):
    w = rng.randint(480, 1280)
    return w, min(720, max(240, int(w * rng.uniform(0.35, 0.75))))


def draw(rng):
    kind = rng.choice(("frame", "init", "stereo", "track", "rig", "batch", "batch_stereo", "knn", "distinctive", "bow",
                       "frustum"))
    w, h = _size(rng)
    nf, ini = rng.randint(800, 2000), rng.choice((20, 12))
    if kind == "frame":
        return {"kind": kind, "w": w, "h": h, "nf": nf, "ini": ini, "device": rng.random() < 0.5}
    if kind == "init":
        return {"kind": kind, "w": w, "h": h, "nf": nf, "window": rng.choice((10, 50, 100))}
    if kind == "stereo":
        return {"kind": kind, "w": w, "h": h, "nf": nf, "ini": ini}
    if kind == "track":
        return {"kind": kind, "w": w, "h": h, "nf": nf, "ini": ini, "m": _log(rng, 200, 4000)}
    if kind in ("rig", "batch"):
        n = rng.randint(2, 9) if kind == "rig" else _log(rng, 10, 64)
        sizes = ",".join("%dx%d" % _size(rng) for _ in range(min(n, 6)))
        return {"kind": kind, "frames": n, "sizes": sizes, "nf": nf, "ini": ini,
                **({"m": _log(rng, 300, 3000)} if kind == "batch" else {})}
    if kind == "batch_stereo":
        return {"kind": kind, "pairs": _log(rng, 3, 32), "w": w, "h": h, "nf": nf, "ini": ini}
    if kind == "knn":
        nq, nt = _log(rng, 500, 50000), _log(rng, 500, 200000)
        return {"kind": kind, "nq": nq, "nt": nt, "algo": rng.choice((0, -1)), "centres": rng.choice((0, 2000))}
    if kind == "distinctive":
        return {"kind": kind, "m": _log(rng, 2000, 1000000), "mean": round(rng.uniform(3.0, 6.0), 2)}
    if kind == "bow":
        frames = 2 * rng.randint(1, 32)
        return {"kind": kind, "frames": frames, "per": rng.randint(500, 2000), "pairs": frames // 2}
    return {"kind": kind, "frames": _log(rng, 1, 64), "per": _log(rng, 200, 5000)}


# ------------------------------------------------------------------------------------------------------ inputs
def _smooth3(a):
    p = torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="replicate")
    return torch.nn.functional.avg_pool2d(p, 3, 1)[0, 0]


def _scene(w, h, rng, gen, shapes=200, sigma=8.0):
    """A w x h uint8 image: filled rectangles and ellipses painted over one another, and smoothed noise."""
    half = max(8, min(w, h) // 6)
    c = torch.tensor(rng.uniform(0, 1, (shapes, 2)) * (w, h), dtype=torch.float32, device=DEV)
    a = torch.tensor(rng.uniform(3, half, (shapes, 2)), dtype=torch.float32, device=DEV)
    ellipse = torch.tensor(rng.random(shapes) < 0.5, device=DEV)[:, None, None]
    values = torch.tensor(np.concatenate([rng.integers(0, 256, 1 + shapes)]), dtype=torch.float32, device=DEV)
    x = ((torch.arange(w, device=DEV, dtype=torch.float32)[None] - c[:, :1]) / a[:, :1]).square()[:, None, :]
    y = ((torch.arange(h, device=DEV, dtype=torch.float32)[None] - c[:, 1:]) / a[:, 1:]).square()[:, :, None]
    top = torch.zeros((h, w), dtype=torch.int64, device=DEV)
    step = 40
    for s in range(0, shapes, step):
        inside = torch.where(ellipse[s:s + step], x[s:s + step] + y[s:s + step], torch.maximum(x[s:s + step], y[s:s + step])) <= 1
        order = torch.arange(s + 1, s + 1 + inside.shape[0], device=DEV)[:, None, None]
        top = torch.maximum(top, (inside * order).amax(0))
    noise = _smooth3(torch.randn((h, w), generator=gen, device=DEV) * sigma)
    return (values[top] + noise).round().clamp(0, 255).to(torch.uint8)


def _bilinear(img, sx, sy):
    h, w = img.shape
    sx, sy = sx.clamp(0, w - 1.001), sy.clamp(0, h - 1.001)
    x0, y0 = sx.floor().long(), sy.floor().long()
    fx, fy = sx - x0, sy - y0
    a = img.float()
    return (a[y0, x0] * (1 - fx) + a[y0, x0 + 1] * fx) * (1 - fy) + (a[y0 + 1, x0] * (1 - fx) + a[y0 + 1, x0 + 1] * fx) * fy


def _noisy(img, gen, sigma=2.0):
    return (img + torch.randn(img.shape, generator=gen, device=DEV) * sigma).round().clamp(0, 255).to(torch.uint8)


def _grid(h, w):
    return torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32), torch.arange(w, device=DEV, dtype=torch.float32),
                          indexing="ij")


def _second_view(img, rng, gen):
    """The image under a rotation of at most 3 degrees and a shift of at most 10 px, with noise."""
    h, w = img.shape
    th, (tx, ty) = math.radians(rng.uniform(-3, 3)), rng.uniform(-10, 10, 2)
    y, x = _grid(h, w)
    dx, dy = x - w / 2 - tx, y - h / 2 - ty
    return _noisy(_bilinear(img, math.cos(th) * dx + math.sin(th) * dy + w / 2, -math.sin(th) * dx + math.cos(th) * dy + h / 2),
                  gen)


def _right_view(img, rng, gen):
    """The image under a piecewise planar disparity of 5 to 80 px, with noise."""
    h, w = img.shape
    y, x = _grid(h, w)
    nb = int(rng.integers(3, 7))
    cuts = np.sort(rng.uniform(0, w, nb - 1))
    d = torch.zeros_like(x)
    for lo, hi in zip([0, *cuts], [*cuts, w]):
        plane = rng.uniform(5, 80) + rng.uniform(-0.03, 0.03) * (x - lo) + rng.uniform(-0.05, 0.05) * (y - h / 2)
        d = torch.where((x >= lo) & (x < hi), plane, d)
    return _noisy(_bilinear(img, x + d.clamp(5, 80), y), gen)


def _bits(shape, p, gen):
    """Bytes whose bits are set with probability p."""
    b = torch.rand((*shape, 8), generator=gen, device=DEV) < p
    return (b * torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], device=DEV)).sum(-1).to(torch.uint8)


def _random_bytes(shape, gen):
    return torch.randint(0, 256, shape, generator=gen, device=DEV, dtype=torch.uint8)


def _records(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).to(DEV)


def _map_points(kps, desc, m, rng, gen):
    """m map points seen near the frame's features: descriptors with 10 % of the bits flipped, positions off by 2 px."""
    k = kps.cpu().numpy()
    n = len(k)
    src = rng.integers(0, max(n, 1), m)
    mps = np.zeros(m, MAPPOINT_DTYPE)
    mps["proj_x"] = k[src, 0] + rng.normal(0, 2, m)
    mps["proj_y"] = k[src, 1] + rng.normal(0, 2, m)
    mps["proj_xr"] = -1
    mps["view_cos"] = 1.0
    mps["track_scale_level"] = k.view(np.int32)[src, 5]
    mps["track_in_view"] = 1
    return mps, desc[torch.from_numpy(src).to(DEV)] ^ _bits((m, 32), 0.1, gen)


def _previous_frame(kps, desc, w, h, rng, gen):
    """The frame before: its keypoints, map points and their descriptors, and the two poses."""
    k = kps.cpu().numpy()
    n = len(k)
    m = max(1, int(1.1 * n))
    src = rng.integers(0, max(n, 1), m)
    R, t = synthetic._rot(*rng.normal(0, 0.02, 3)), rng.normal(0, 0.3, 3)
    Rl = R @ synthetic._rot(*rng.normal(0, 0.005, 3))
    z = rng.uniform(3, 40, m)
    u, v = k[src, 0] + rng.normal(0, 1, m), k[src, 1] + rng.normal(0, 1, m)
    P = (np.stack([(u - w / 2) * z / FX, (v - h / 2) * z / FX, z], 1) - t) @ R
    mps = np.zeros(m, FRAME_MAPPOINT_DTYPE)
    mps["x"], mps["y"], mps["z"] = P[:, 0], P[:, 1], P[:, 2]
    flags = rng.random(m)
    mps["flags"] = np.where(flags < 0.1, 0, np.where(flags < 0.15, 3, np.where(flags < 0.27, 1, 5)))
    last = np.zeros((m, 7), np.float32)
    last[:, 3] = (k[src, 3] + 8 + rng.normal(0, 3, m)) % 360
    last.view(np.int32)[:, 5] = np.clip(k.view(np.int32)[src, 5] + rng.choice([-1, 0, 0, 0, 1], m), 0, LEVELS - 1)
    last.view(np.int32)[:, 6] = -1
    T = np.hstack([R, t[:, None]]).astype(np.float32)
    Tl = np.hstack([Rl, (-Rl @ (-R.T @ t))[:, None]]).astype(np.float32)
    motion = motion_struct(T, Tl, FX, FX, w / 2, h / 2, BF, BF / FX)
    return last, mps, desc[torch.from_numpy(src).to(DEV)] ^ _bits((m, 32), 0.08, gen), motion


def _frames(case, rng):
    """The sizes and feature budgets of a batch's frames."""
    n = case["frames"]
    if case["sizes"] == "mixed":
        pick = rng.integers(0, len(RESOLUTIONS), n)
        return [RESOLUTIONS[i] for i in pick], [int(v) for v in rng.choice((1000, 1500, 2000), n)]
    sizes = [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]
    return [sizes[i % len(sizes)] for i in range(n)], [case["nf"]] * n


def _batch(sizes, nfs):
    """A batch extractor for these frames; rows past a frame's keypoints are never written and stay 0."""
    b = BatchExtractor(len(sizes), max(s[0] for s in sizes), max(s[1] for s in sizes), max(nfs), SCALE, LEVELS)
    for t in (b.kps, b.desc, b.counts):
        t.zero_()
    return b


def _split(b, n):
    """The keypoints and descriptors of the batch's frames."""
    b.wait()
    cap = b.per_frame_capacity
    return [(b.kps[f * cap:f * cap + c], b.desc[f * cap:f * cap + c]) for f, c in enumerate(b.counts[:n].tolist())]


@functools.lru_cache(maxsize=1)
def _vocabulary():
    """The vocabulary a program loads once: ten children, six levels, a million words."""
    v = synthetic.vocabulary(10, 6, 2024)
    return v, Vocabulary.from_arrays(10, 6, 0, 0, v["parents"], v["is_leaf"], v["descriptors"], v["weights"])


def _bow_inputs(case, seed):
    """Descriptors of consecutive frames near words, 70 % of a frame's features shared with the frame before."""
    rng, gen = np.random.default_rng(seed), torch.Generator(DEV).manual_seed(seed)
    nf, per = case["frames"], case["per"]
    v, _ = _vocabulary()
    leaves = np.nonzero(v["is_leaf"])[0]
    words = torch.from_numpy(v["descriptors"][rng.choice(leaves, nf * per)]).to(DEV)
    desc = (words ^ _bits((nf * per, 32), 0.125, gen)).view(nf, per, 32)
    for f in range(1, nf):
        rows = torch.randperm(per, generator=gen, device=DEV)[:int(0.7 * per)]
        desc[f, rows] = desc[f - 1, rows] ^ _bits((len(rows), 32), 0.0625, gen)
    kps = torch.zeros((nf * per, 7), dtype=torch.float32, device=DEV)
    kps[:, 3] = torch.rand(nf * per, generator=gen, device=DEV) * 360
    return desc.reshape(nf * per, 32).contiguous(), kps


# ------------------------------------------------------------------------------------------------------ prepare and run
def _ready(*inputs):
    """The inputs, written: the library's handles work on streams of their own."""
    torch.cuda.current_stream().synchronize()
    return inputs[0] if len(inputs) == 1 else inputs


def prepare(case, seed):
    rng, gen = np.random.default_rng(seed), torch.Generator(DEV).manual_seed(seed)
    return {"kind": case["kind"], **_PREPARE[case["kind"]](case, seed, rng, gen)}


def run(state):
    return _RUN[state["kind"]](state)


def _room(n, device, **columns):
    """A program's own arrays for up to n rows of a frame's results, each frame's rows copied to their start."""
    make = functools.partial(torch.zeros, device=DEV) if device else np.zeros
    kinds = {"i": torch.int32, "f": torch.float32, "b": torch.uint8} if device else {"i": np.int32, "f": np.float32, "b": np.uint8}
    return {k: make((n, *shape), dtype=kinds[kind]) for k, (kind, *shape) in columns.items()}


def _keep(room, **rows):
    for k, r in rows.items():
        room[k][:len(r)] = r
    return room



def _prepare_frame(case, seed, rng, gen):
    img = _scene(case["w"], case["h"], rng, gen)
    ex = ORBextractor(case["nf"], SCALE, LEVELS, case["ini"], 7, case["w"], case["h"])
    return {"ex": ex, "image": img if case["device"] else img.cpu().numpy(), "device": case["device"],
            "room": _room(ex.capacity(), case["device"], keypoints=("i", 7), descriptors=("b", 32))}


def _run_frame(s):
    kps, desc = s["ex"](s["image"], device_out=s["device"])
    kps = kps.view(torch.int32) if s["device"] else kps.view(np.int32).reshape(-1, 7)
    return _keep(s["room"], keypoints=kps, descriptors=desc)


def _prepare_init(case, seed, rng, gen):
    w, h = case["w"], case["h"]
    first = _scene(w, h, rng, gen)
    second = _second_view(first, rng, gen)
    ex = ORBextractor(case["nf"], SCALE, LEVELS, 20, 7, w, h)
    views = [FrameView(*ex(i.cpu().numpy()), w, h, ex.GetScaleFactors()) for i in (first, second)]
    prev = np.stack([views[0].keypoints["x"], views[0].keypoints["y"]], 1)
    return {"matcher": ORBmatcher(0.9, True), "views": views, "prev": prev, "window": case["window"],
            "room": _room(ex.capacity(), False, matches=("i",), prev=("f", 2))}


def _run_init(s):
    n, matches, prev = s["matcher"].SearchForInitialization(*s["views"], s["prev"], s["window"])
    return {"n": n, **_keep(s["room"], matches=matches, prev=prev)}


def _prepare_stereo(case, seed, rng, gen):
    w, h = case["w"], case["h"]
    left = _scene(w, h, rng, gen)
    ex = [ORBextractor(case["nf"], SCALE, LEVELS, case["ini"], 7, w, h) for _ in range(2)]
    return {"images": (left, _right_view(left, rng, gen)), "ex": ex, "matcher": ORBmatcher(0.75, True),
            "scales": ex[0].GetScaleFactors(), "w": w, "h": h,
            "room": _room(ex[0].capacity(), True, left=("i", 7), right=("i", 7), left_desc=("b", 32), right_desc=("b", 32),
                          uright=("f",), depth=("f",))}


def _run_stereo(s):
    (kl, dl), (kr, dr) = (ex(i, device_out=True) for ex, i in zip(s["ex"], s["images"]))
    views = [FrameView(k, d, s["w"], s["h"], s["scales"]) for k, d in ((kl, dl), (kr, dr))]
    uright, depth = compute_stereo_matches(s["matcher"], *s["ex"], *views, BF, FX)
    return _keep(s["room"], left=kl.view(torch.int32), right=kr.view(torch.int32), left_desc=dl, right_desc=dr, uright=uright,
                 depth=depth)


def _prepare_track(case, seed, rng, gen):
    w, h = case["w"], case["h"]
    img = _scene(w, h, rng, gen)
    ex = ORBextractor(case["nf"], SCALE, LEVELS, case["ini"], 7, w, h)
    mps, mpd = _map_points(*ex(_ready(img), device_out=True), case["m"], rng, gen)
    return {"ex": ex, "image": img, "matcher": ORBmatcher(0.8, True), "mps": _records(mps), "mpd": mpd, "w": w, "h": h,
            "scales": ex.GetScaleFactors(),
            "room": _room(ex.capacity(), True, keypoints=("i", 7), descriptors=("b", 32), match=("i",))}


def _run_track(s):
    kps, desc = s["ex"](s["image"], device_out=True)
    view = FrameView(kps, desc, s["w"], s["h"], s["scales"])
    n, match = s["matcher"].SearchByProjection(view, s["mps"], s["mpd"], 3.0)
    return {"n": n, **_keep(s["room"], keypoints=kps.view(torch.int32), descriptors=desc, match=match)}


def _prepare_batch(case, seed, rng, gen):
    sizes, nfs = _frames(case, np.random.default_rng(case["frames"]))
    images = [_scene(w, h, rng, gen) for w, h in sizes]
    b = _batch(sizes, nfs)
    b.ini_th = case["ini"]
    frames = b.frames(images, nfs)
    _ready()
    b.extract(frames)
    views = _split(b, len(sizes))
    s = {"batch": b, "frames": frames}
    if case["kind"] == "batch":
        made = [_map_points(k, d, case["m"], rng, gen) for k, d in views]
        s |= {"search": BatchProjection(b, 0.8), "mps": _records(np.concatenate([m for m, _ in made])),
              "mpd": torch.cat([d for _, d in made]), "counts": [case["m"]] * len(sizes)}
    else:
        made = [_previous_frame(k, d, w, h, rng, gen) for (k, d), (w, h) in zip(views, sizes)]
        s |= {"search": BatchFrameProjection(b, True), "last": torch.from_numpy(np.concatenate([m[0] for m in made])).to(DEV),
              "mps": _records(np.concatenate([m[1] for m in made])), "mpd": torch.cat([m[2] for m in made]),
              "counts": [len(m[0]) for m in made], "motions": [m[3] for m in made]}
    return s


def _run_batch(s):
    kps, desc, counts = s["batch"].extract(s["frames"], wait=False)
    match, n = s["search"].search(s["mps"], s["mpd"], s["counts"], 6.0)
    return {"keypoints": kps.view(torch.int32), "descriptors": desc, "counts": counts, "match": match, "n": n}


def _run_rig(s):
    kps, desc, counts = s["batch"].extract(s["frames"], wait=False)
    match, n = s["search"].search(s["last"], s["mps"], s["mpd"], s["counts"], s["motions"], 15.0, True)
    return {"keypoints": kps.view(torch.int32), "descriptors": desc, "counts": counts, "match": match, "n": n}


def _prepare_batch_stereo(case, seed, rng, gen):
    w, h, n = case["w"], case["h"], case["pairs"]
    images = []
    for _ in range(n):
        left = _scene(w, h, rng, gen)
        images += [left, _right_view(left, rng, gen)]
    b = _batch([(w, h)] * 2 * n, [case["nf"]] * 2 * n)
    b.ini_th = case["ini"]
    st = BatchStereo(b)
    st.uright.zero_()
    st.depth.zero_()
    return {"batch": b, "frames": b.frames(images, [case["nf"]] * 2 * n), "stereo": st, "pairs": [(2 * p, 2 * p + 1) for p in range(n)]}


def _run_batch_stereo(s):
    kps, desc, counts = s["batch"].extract(s["frames"], wait=False)
    uright, depth = s["stereo"].compute(s["pairs"], BF, FX)
    return {"keypoints": kps.view(torch.int32), "descriptors": desc, "counts": counts, "uright": uright, "depth": depth}


def _prepare_knn(case, seed, rng, gen):
    if case["centres"]:
        centres = _random_bytes((case["centres"], 32), gen)
        q, t = (centres[torch.randint(0, case["centres"], (n,), generator=gen, device=DEV)] ^ _bits((n, 32), 0.1, gen)
                for n in (case["nq"], case["nt"]))
    else:
        q, t = _random_bytes((case["nq"], 32), gen), _random_bytes((case["nt"], 32), gen)
    return {"matcher": ORBmatcher(), "q": q, "t": t, "algo": case["algo"]}


def _run_knn(s):
    return s["matcher"].knn2(s["q"], s["t"], algo=s["algo"], ratio=0.8)


def _prepare_distinctive(case, seed, rng, gen):
    m = case["m"]
    lens = torch.log(torch.rand(m, generator=gen, device=DEV).clamp_min(1e-12)) / math.log(1 - 1 / case["mean"])
    lens = lens.floor().long().clamp(0, 63) + 1
    lens[torch.rand(m, generator=gen, device=DEV) < 0.02] = 0
    offsets = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    offsets[1:] = lens.cumsum(0)
    n = int(offsets[-1])
    of = torch.repeat_interleave(torch.arange(m, device=DEV), lens)
    pool = torch.empty((n, 32), dtype=torch.uint8, device=DEV)
    rows = torch.randperm(n, generator=gen, device=DEV)
    pool[rows] = _random_bytes((m, 32), gen)[of] ^ _bits((n, 32), 0.125, gen)
    rows = torch.where(torch.rand(n, generator=gen, device=DEV) < 0.05, -1, rows)
    return {"pool": pool, "offsets": offsets.int(), "rows": rows.int(),
            "descriptors": torch.zeros((m, 32), dtype=torch.uint8, device=DEV)}


def _run_distinctive(s):
    return {"best": compute_distinctive_descriptors(s["pool"], s["offsets"], s["rows"], s["descriptors"]),
            "descriptors": s["descriptors"]}


def _prepare_bow(case, seed, rng, gen):
    desc, kps = _bow_inputs(case, seed)
    nf, per = case["frames"], case["per"]
    return {"voc": _vocabulary()[1], "desc": desc, "kps": kps, "offsets": torch.arange(nf + 1, dtype=torch.int32, device=DEV) * per,
            "mp": (torch.rand(nf * per, generator=gen, device=DEV) < 0.9).to(torch.uint8),
            "pairs": [(2 * p, 2 * p + 1) for p in range(case["pairs"])],
            "place": torch.arange(per, device=DEV)[None], "shape": (nf, per)}


def _run_bow(s):
    v = s["voc"].transform(s["desc"], s["offsets"], 4)
    n, matches = search_by_bow(s["kps"], s["desc"], s["offsets"], v, s["mp"], s["pairs"])
    # a frame's word vector is its first bow_counts entries
    used = s["place"] < v["bow_counts"][:, None]
    words = torch.where(used, v["bow_words"].view(s["shape"]), -1)
    values = torch.where(used, v["bow_values"].view(s["shape"]), 0.0)
    return {"word": v["word"], "weight": v["weight"], "node": v["node"], "bow_counts": v["bow_counts"], "bow_words": words,
            "bow_values": values, "fv_counts": v["fv_counts"], "n": n, "matches": matches}


_CAMERAS = ((640, 480, 500.0), (1241, 376, 718.856), (752, 480, 458.7), (1280, 720, 900.0))


def _prepare_frustum(case, seed, rng, gen):
    nf, per = case["frames"], case["per"]
    frames, geometry = [], []
    for f in range(nf):
        w, h, fx = _CAMERAS[f % len(_CAMERAS)]
        T, g = synthetic.frustum_case(per, seed * 1000 + f, w, h, fx, SCALE, LEVELS)
        frames.append(frustum_frame(T, fx, fx, w / 2, h / 2, 40.0, 0.0, w, 0.0, h, SCALE, LEVELS))
        geometry.append(g)
    return {"frames": _records(np.array(frames, FRUSTUM_FRAME_DTYPE)),
            "offsets": torch.arange(nf + 1, dtype=torch.int32, device=DEV) * per,
            "geometry": torch.from_numpy(np.concatenate(geometry)).to(DEV),
            "mps": torch.zeros((nf * per, 8), dtype=torch.int32, device=DEV),
            "in_view": torch.zeros(nf, dtype=torch.int32, device=DEV)}


def _run_frustum(s):
    is_in_frustum(s["frames"], s["offsets"], s["geometry"], s["mps"], 0.5, s["in_view"])
    return {"mappoints": s["mps"], "in_view": s["in_view"]}


_PREPARE = {"frame": _prepare_frame, "init": _prepare_init, "stereo": _prepare_stereo, "track": _prepare_track,
            "rig": _prepare_batch, "batch": _prepare_batch, "batch_stereo": _prepare_batch_stereo, "knn": _prepare_knn,
            "distinctive": _prepare_distinctive, "bow": _prepare_bow, "frustum": _prepare_frustum}
_RUN = {"frame": _run_frame, "init": _run_init, "stereo": _run_stereo, "track": _run_track, "rig": _run_rig,
        "batch": _run_batch, "batch_stereo": _run_batch_stereo, "knn": _run_knn, "distinctive": _run_distinctive, "bow": _run_bow,
        "frustum": _run_frustum}


# ------------------------------------------------------------------------------------------------------ work and 64-bit values
def _frame_bytes(w, h, nf):
    """One extraction: the image read, the pyramid (a result of the extractor) written, 60 bytes a keypoint."""
    return w * h * (1 + sum(SCALE ** (-2 * l) for l in range(LEVELS))) + 60 * nf


def work(case):
    kind = case["kind"]
    flops = 0
    if kind == "frame":
        b = _frame_bytes(case["w"], case["h"], case["nf"])
    elif kind == "init":
        b = 2 * 60 * case["nf"] + 20 * case["nf"]
    elif kind == "stereo":
        b = 2 * _frame_bytes(case["w"], case["h"], case["nf"]) + 8 * case["nf"]
    elif kind == "track":
        b = _frame_bytes(case["w"], case["h"], case["nf"]) + 64 * case["m"] + 4 * case["nf"]
    elif kind in ("rig", "batch"):
        sizes, nfs = _frames(case, np.random.default_rng(case["frames"]))
        per = case["m"] * 64 if kind == "batch" else 1.1 * 76 * case["nf"]
        b = sum(_frame_bytes(w, h, n) + per + 4 * n for (w, h), n in zip(sizes, nfs))
    elif kind == "batch_stereo":
        b = case["pairs"] * (2 * _frame_bytes(case["w"], case["h"], case["nf"]) + 8 * case["nf"])
    elif kind == "knn":
        b = 32 * (case["nq"] + case["nt"]) + 17 * case["nq"]
        flops = 2 * 256 * case["nq"] * case["nt"]  # the dot products of the descriptors as +1 / -1 vectors
    elif kind == "distinctive":
        b = case["m"] * (4 + 36 * case["mean"] * 0.98 + 36)
    elif kind == "bow":
        b = case["frames"] * case["per"] * (32 + 28 + 16 + 32) + case["pairs"] * case["per"] * (2 * 36 + 4)
    else:
        b = case["frames"] * (160 + case["per"] * (32 + 24))
    return {"bytes": float(b), "flops": float(flops)}


def exact(case, seed):
    """The word vectors' values and the features' weights in 64 bits; the other kinds return whole numbers, bytes and records
    (compared bit for bit), or the results of a whole image pipeline."""
    if case["kind"] != "bow":
        return None
    desc, _ = _bow_inputs(case, seed)
    v, _ = _vocabulary()
    nf, per = case["frames"], case["per"]
    ones = torch.tensor([bin(i).count("1") for i in range(256)], dtype=torch.int16, device=DEV)
    table, first = torch.from_numpy(v["descriptors"]).to(DEV), 0
    at = torch.zeros(nf * per, dtype=torch.int64, device=DEV)  # the node's place in its level
    for level in range(1, 7):
        child = at[:, None] * 10 + torch.arange(10, device=DEV)
        dist = ones[(table[first + child] ^ desc[:, None]).long()].sum(-1)
        # the first child at the least distance
        at = child.gather(1, (dist * 16 + torch.arange(10, device=DEV)).argmin(1, keepdim=True))[:, 0]
        first += 10 ** level
    first -= 10 ** 6
    weight = torch.from_numpy(v["weights"]).to(DEV)[first + at].cpu().numpy()
    word = at.cpu().numpy()
    values = np.zeros((nf, per))
    for f in range(nf):
        w, u = word[f * per:(f + 1) * per], weight[f * per:(f + 1) * per]
        w, u = w[u > 0], u[u > 0]
        ids, place, count = np.unique(w, return_index=True, return_counts=True)
        total = u[place] * count
        values[f, :len(ids)] = total / total.sum()
    return {"weight": torch.from_numpy(weight), "bow_values": torch.from_numpy(values)}
