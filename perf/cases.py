"""Workloads of the dense-MVS library, one dict of plain values per workload.

A workload ("case") is one call sequence a user's program makes through the
public entry points, with the sizes, options and data it meets in earnest:

kind    call                                    direction / what is in hand
depth   mvs.estimate_depth                      one reference view, host buffers in and out
dense   mvs.run_mvs                             a whole model: host images -> fused cloud
stereo  DeviceScene.estimate (resident scene)   a batch of depth maps, device in and out
fuse    DeviceScene.fuse + points               depth maps -> fused cloud
sift    sift.extract_sift                       one decoded image -> keypoints, descriptors
match   sift.match_pairs                        descriptor sets -> mutual matches of pairs
train   ProposalNet.train_step                  network forward, backward, Adam step
resize  mvs.resize_view                         one decoded image -> working resolution

Stereo, fusion, SIFT and matching reproduce a serial f32/f64 algorithm bit
for bit (every abort, accept and tie decision depends on its rounding), so
their outputs have no separate 64-bit value; the training step does.
"""
import math

import numpy as np
import torch

from rustcolmap_b200 import MvsOptions, learned, mvs, scene, sift

# The (w, h) pool of a model whose views come from several cameras.
MIXED_SIZES = ((480, 360), (480, 270), (720, 540), (720, 405), (960, 720), (960, 540), (1440, 1080))

# Rows of the buffers that hold a fused cloud (a room at these voxel sizes
# fills fewer): outputs of a fixed shape, zeros after the last point.
CLOUD_ROWS = 600_000


def listed():
    return [
        # Smallest stereo call: a preview-sized reference view against two
        # neighbours, one sweep; launches and round trips, not arithmetic.
        {"name": "depth_small", "kind": "depth", "w": 96, "h": 72, "views": 4, "srcs": 2, "sweeps": 1, "hyps": 16,
         "k": 0.0},
        # A small model end to end with the reference's schedule (6 sweeps).
        {"name": "dense_corner", "kind": "dense", "w": 384, "h": 288, "views": 8, "srcs": 4, "sweeps": 6,
         "hyps": 64, "learned": False},
        # The headline use: 1080p views, K = 10, learned init + 4 passes,
        # from host images to the fused cloud (a 58-degree arc of the orbit).
        {"name": "dense_1080p", "kind": "dense", "w": 1920, "h": 1080, "views": 16, "srcs": 10, "sweeps": 3,
         "hyps": 64, "learned": True},
        # The reference's schedule on a resident scene, ordinary resolution.
        {"name": "stereo_960", "kind": "stereo", "w": 960, "h": 720, "views": 16, "srcs": 8, "sweeps": 6, "hyps": 64,
         "k": 0.0, "mixed": False},
        # Views of several cameras with radial distortion, the reference's
        # default schedule (4 sweeps, 48 hypotheses, 3 sources).
        {"name": "stereo_mixed", "kind": "stereo", "w": 1440, "h": 1080, "views": 12, "srcs": 3, "sweeps": 4,
         "hyps": 48, "k": -0.02, "mixed": True},
        # Fusion alone: depth maps that already exist (a re-run with other
        # fusion thresholds).
        {"name": "fuse_960", "kind": "fuse", "w": 960, "h": 720, "views": 24, "srcs": 8},
        # SIFT of one full-size photograph.
        {"name": "sift_1600", "kind": "sift", "w": 1600, "h": 1200, "channels": 3, "features": 2048},
        # SIFT of one small grey frame of odd sides (video).
        {"name": "sift_odd_grey", "kind": "sift", "w": 641, "h": 479, "channels": 1, "features": 1024},
        # Exhaustive matching of a small photo set.
        {"name": "match_set", "kind": "match", "frames": 12, "features": 2048, "ragged": False},
        # One pair of frames with few, unequal features.
        {"name": "match_pair", "kind": "match", "frames": 2, "features": 517, "ragged": True},
        # One optimiser step of the proposal network: a batch of 16
        # quarter-resolution 960x720 views.
        {"name": "train_16", "kind": "train", "n": 16, "w": 240, "h": 180},
        # Loading one 12-megapixel photograph at the working resolution.
        {"name": "resize_12mp", "kind": "resize", "w": 4000, "h": 3000, "channels": 3, "max_dim": 1920},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above, its sizes spread over their
    logarithm and usually odd."""
    kind = rng.choice(["depth", "dense", "dense", "stereo", "stereo", "fuse", "sift", "sift", "match", "match",
                       "train", "resize"])
    if kind == "depth":
        w = _log(rng, 80, 640)
        return {"kind": kind, "w": w, "h": max(60, int(w * rng.uniform(0.55, 1.0))), "views": rng.randint(3, 6),
                "srcs": rng.randint(2, 4), "sweeps": rng.randint(1, 4), "hyps": rng.choice([16, 32, 48, 64]),
                "k": rng.choice([0.0, 0.0, -0.03, 0.02])}
    if kind == "dense":
        learned_arm = rng.random() < 0.5
        w = _log(rng, 320, 1280)
        return {"kind": kind, "w": w, "h": int(w * rng.uniform(0.55, 0.8)), "views": rng.randint(6, 14),
                "srcs": rng.randint(3, 8), "sweeps": 3 if learned_arm else rng.randint(2, 6),
                "hyps": rng.choice([48, 64]), "learned": learned_arm}
    if kind == "stereo":
        mixed = rng.random() < 0.3
        w = _log(rng, 720 if mixed else 240, 1200)
        return {"kind": kind, "w": w, "h": int(w * rng.uniform(0.55, 0.8)), "views": rng.randint(4, 14),
                "srcs": rng.randint(2, 9), "sweeps": rng.randint(2, 6), "hyps": rng.choice([32, 48, 64]),
                "k": rng.choice([0.0, 0.0, -0.02, 0.015]), "mixed": mixed}
    if kind == "fuse":
        w = _log(rng, 320, 1300)
        return {"kind": kind, "w": w, "h": int(w * rng.uniform(0.55, 0.8)), "views": rng.randint(5, 24),
                "srcs": rng.randint(3, 10)}
    if kind == "sift":
        w = _log(rng, 200, 2000)  # above 1600 the extractor resizes first
        return {"kind": kind, "w": w, "h": int(w * rng.uniform(0.6, 1.0)), "channels": rng.choice([1, 3, 3, 4]),
                "features": rng.choice([512, 1024, 2048, 4096])}
    if kind == "match":
        return {"kind": kind, "frames": _log(rng, 2, 12), "features": _log(rng, 100, 2048),
                "ragged": rng.random() < 0.7}
    if kind == "train":
        w = _log(rng, 60, 300)
        return {"kind": kind, "n": rng.randint(2, 16), "w": w, "h": int(w * rng.uniform(0.55, 0.8))}
    w = _log(rng, 700, 4000)
    return {"kind": kind, "w": w, "h": int(w * rng.uniform(0.6, 0.8)), "channels": rng.choice([1, 3, 3, 4]),
            "max_dim": rng.choice([600, 900, 1280, 1920])}


# ------------------------------------------------------------------ inputs
def _scene(c, seed):
    """Rendered views of a furnished room with their sparse model; cameras a
    few degrees apart on an arc (3.6 degrees at 1080p, as 100 views on a full
    orbit stand; 8 degrees below)."""
    if c["w"] <= 400:
        return scene.corner_room(seed=seed, n_views=c["views"], w=c["w"], h=c["h"], f=c["w"] * 1.146,
                                 arc_deg=min(60.0, 12.0 * c["views"]), device=0)
    mixed = c.get("mixed", False)
    sizes = tuple(s for s in MIXED_SIZES if s[0] <= c["w"]) if mixed else ((c["w"], c["h"]),)
    return scene.orbit_room(seed=seed, n_views=c["views"], sizes=sizes, f_rel=1.15 if c["w"] >= 1400 else 1.1,
                            n_boxes=60 if c["w"] >= 1400 else 20, n_spheres=10 if c["w"] >= 1400 else 0,
                            device=0, size_choice="random" if mixed else None,
                            arc_deg=(3.6 if c["w"] >= 1400 else 8.0) * c["views"])


def _distort(sc, k):
    for v in sc.views:
        v.cam.k = k


def _dense_options(c):
    o = MvsOptions(max_dim=max(c["w"], c["h"]), num_sources=c["srcs"], sweeps=c["sweeps"], num_hyp=c["hyps"])
    if c["w"] >= 1400:  # the full-size model's fusion thresholds
        o.min_consistent, o.depth_diff, o.reproj_px = 3, 0.01, 1.0
    return learned.learned_options(o) if c["learned"] else o


def _jobs(sc, opts):
    srcs, zr, order = mvs.plan(sc.sparse, sc.views, opts)
    return [(i, srcs[i], zr[i, 0], zr[i, 1]) for i in range(len(sc.views)) if srcs[i]], order


def _image(c, seed):
    """One rendered photograph as decoded bytes (h, w[, channels])."""
    sc = scene.orbit_room(seed=seed, n_views=2, sizes=((c["w"], c["h"]),), f_rel=1.1, n_boxes=20, n_spheres=4,
                          device=0, per_view_sparse=10, arc_deg=8.0)
    g = sc.views[0].gray
    if c["channels"] == 1:
        return g
    rng = np.random.default_rng(seed)
    gain = rng.uniform(0.7, 1.0, size=3)  # a colour cast, so the channels differ
    img = np.empty(g.shape + (c["channels"],), np.uint8)
    for i in range(3):
        img[..., i] = g * gain[i]
    if c["channels"] == 4:
        img[..., 3] = 255
    return img


def _descriptors(c, seed):
    """SIFT-like unit descriptors (non-negative, clipped at 0.2 before the
    last normalisation); neighbouring frames share about a quarter of them up
    to noise, the rest are their own."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)

    def unit(x):
        x = x / x.norm(dim=1, keepdim=True)
        x = x.clamp(max=0.2)
        return x / x.norm(dim=1, keepdim=True)

    n = c["features"]
    base = torch.rand((2 * n, 128), device="cuda", generator=g) ** 3
    out = []
    for f in range(c["frames"]):
        m = int(rng.integers(max(n // 2, 2), n + 1)) if c["ragged"] else n
        own = torch.rand((m, 128), device="cuda", generator=g) ** 3
        shared = torch.randperm(2 * n, device="cuda", generator=g)[: m // 2]
        noise = torch.rand((m // 2, 128), device="cuda", generator=g)
        own[: m // 2] = base[shared] * (0.85 + 0.3 * noise)
        out.append(unit(own).cpu().numpy())
    return out


def _batch(c, seed):
    """A training batch: census cost volumes with a dip at the true plane,
    grey values, and labels (t, normal, valid, tolerance)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, h, w = c["n"], c["h"], c["w"]

    def rand(*s):
        return torch.rand(s, device="cuda", generator=g)

    lo = torch.rand((n, 1, max(h // 8, 2), max(w // 8, 2)), device="cuda", generator=g)
    t = torch.nn.functional.interpolate(lo, size=(h, w), mode="bilinear", align_corners=True)[:, 0]
    x = torch.zeros((n, h, w, learned.COSTVOL_C), device="cuda")
    bins = (torch.arange(32, device="cuda") + 0.5) / 32
    x[..., :32] = (0.42 + 0.08 * (rand(n, h, w, 32) - 0.5)
                   - 0.3 * torch.exp(-((bins - t[..., None]) / 0.04) ** 2))
    x[..., 32] = rand(n, h, w)
    lab = torch.zeros((n, h, w, learned.LABEL_C), device="cuda")
    nrm = rand(n, h, w, 3) - 0.5
    nrm[..., 2] += 1.2
    lab[..., 0] = t
    lab[..., 1:4] = nrm / nrm.norm(dim=-1, keepdim=True)
    lab[..., 4] = (rand(n, h, w) < 0.4).float()
    lab[..., 5] = 0.02 + 0.02 * t
    return x.to(torch.bfloat16).contiguous(), lab.contiguous()


def _buffers(s, shapes):
    s["buf"] = {k: np.zeros(sh, dt) for k, (sh, dt) in shapes.items()}
    s["rows"] = {k: 0 for k in shapes}


def _keep(s, key, parts):
    """`parts` (arrays) one after another in the state's buffer `key`, zeros
    after them."""
    buf, n = s["buf"][key], 0
    for a in parts:
        buf[n:n + len(a)] = a
        n += len(a)
    buf[n:s["rows"][key]] = 0
    s["rows"][key] = n
    return buf


def prepare(case, seed):
    c = dict(case)
    s = {"c": c}
    kind = c["kind"]
    if kind == "depth":
        sc = _scene(c, seed)
        _distort(sc, c["k"])
        s["opts"] = MvsOptions(max_dim=max(c["w"], c["h"]), num_sources=c["srcs"], sweeps=c["sweeps"],
                               num_hyp=c["hyps"])
        s["jobs"], _ = _jobs(sc, s["opts"])
        s["views"] = sc.views
        s["ctx"] = mvs.default_context()
    elif kind == "dense":
        sc = _scene(c, seed)
        s["views"], s["sparse"] = sc.views, sc.sparse
        s["opts"] = _dense_options(c)
        s["net"] = learned.ProposalNet(params=learned.load_weights()) if c["learned"] else None
        _buffers(s, {"xyz": ((CLOUD_ROWS, 3), np.float64), "rgb": ((CLOUD_ROWS, 3), np.uint8)})
    elif kind == "stereo":
        sc = _scene(c, seed)
        _distort(sc, c["k"])
        side = max(max(v.w, v.h) for v in sc.views)
        s["opts"] = MvsOptions(max_dim=side, num_sources=c["srcs"], sweeps=c["sweeps"], num_hyp=c["hyps"])
        s["jobs"], _ = _jobs(sc, s["opts"])
        s["scene"] = mvs.DeviceScene(sc.views)
        cap = max((a * b for a, b in MIXED_SIZES if a <= c["w"])) if c["mixed"] else c["w"] * c["h"]
        s["maps"] = torch.zeros((c["views"], cap), device="cuda")  # a row per view, its map first
    elif kind == "fuse":
        sc = _scene(c, seed)
        s["opts"] = MvsOptions(max_dim=max(c["w"], c["h"]), num_sources=c["srcs"], min_consistent=2,
                               depth_diff=0.01, reproj_px=1.0, voxel_rel=0.003)
        _, s["order"] = _jobs(sc, s["opts"])
        s["sparse"] = sc.sparse.xyz
        _buffers(s, {"xyz": ((CLOUD_ROWS, 3), np.float64), "rgb": ((CLOUD_ROWS, 3), np.uint8)})
        s["scene"] = mvs.DeviceScene(sc.views)
        rng = np.random.default_rng(seed)
        for i, d in enumerate(sc.gt_depth):
            # what the gate leaves of a depth map: a third of the pixels in
            # patches, with errors of up to about a percent
            gh, gw = -(-d.shape[0] // 24), -(-d.shape[1] // 24)
            keep = np.kron(rng.random((gh, gw)) < 0.35, np.ones((24, 24), bool))[: d.shape[0], : d.shape[1]]
            err = rng.standard_normal(d.shape, dtype=np.float32) * np.float32(0.004)
            s["scene"].set_depth(i, np.where(keep, d * (1 + err), 0).astype(np.float32))
    elif kind == "sift":
        s["img"] = _image(c, seed)
        s["opts"] = sift.SiftOptions(max_features=c["features"])
        n = c["features"]
        _buffers(s, {"pts": ((n, 2), np.float64), "desc": ((n, 128), np.float32), "colors": ((n, 3), np.uint8)})
    elif kind == "match":
        s["descs"] = _descriptors(c, seed)
        s["pairs"] = sift.job_pairs(len(s["descs"]))
        rows = len(s["pairs"]) * c["features"]
        _buffers(s, {"a": ((rows,), np.uint32), "b": ((rows,), np.uint32)})
    elif kind == "train":
        s["x"], s["lab"] = _batch(c, seed)
        s["net"] = learned.ProposalNet(params=learned.load_weights())
    elif kind == "resize":
        s["img"] = _image(c, seed)
        s["to"] = mvs.working_size(c["w"], c["h"], c["max_dim"])
    else:
        raise ValueError(kind)
    return s


def run(s):
    kind = s["c"]["kind"]
    if kind == "depth":
        ref, srcs, zmin, zmax = s["jobs"][0]
        m = mvs.estimate_depth(s["views"], ref, srcs, zmin, zmax, s["opts"], normals=True)
        return m.depth, m.cost, m.normal
    if kind == "dense":
        st, xyz, rgb = mvs.run_mvs(s["views"], s["sparse"], s["opts"], net=s["net"])
        return {"xyz": _keep(s, "xyz", [xyz]), "rgb": _keep(s, "rgb", [rgb]), "points": st.dense_points,
                "maps": st.views_with_depth, "candidates": st.fusion_candidates}
    if kind == "stereo":
        s["scene"].estimate(s["jobs"], s["opts"])
        for ref, _, _, _ in s["jobs"]:
            s["scene"].depth_to_device(ref, s["maps"][ref].data_ptr())
        return s["maps"]
    if kind == "fuse":
        n = s["scene"].fuse(s["order"], s["sparse"], s["opts"])
        xyz, rgb = s["scene"].points()
        return _keep(s, "xyz", [xyz]), _keep(s, "rgb", [rgb]), n
    if kind == "sift":
        f = sift.extract_sift(s["img"], opts=s["opts"])
        out = {"pts": f.pts, "desc": f.desc, "colors": f.colors}
        if len(f.pts) < s["c"]["features"]:
            out = {k: _keep(s, k, [v]) for k, v in out.items()}
        return {**out, "n": len(f.pts), "raw": f.n_raw}
    if kind == "match":
        m = sift.match_pairs(s["descs"], s["pairs"])
        return (_keep(s, "a", [a for a, _ in m]), _keep(s, "b", [b for _, b in m]),
                np.array([len(a) for a, _ in m]))
    if kind == "train":
        c = s["c"]
        loss, grads = s["net"].train_step(s["x"].data_ptr(), s["lab"].data_ptr(), c["n"], c["h"], c["w"], 1e-3,
                                          grads=True)
        return np.float32(loss), grads
    mw, mh = s["to"]
    return mvs.resize_view(s["img"], mw, mh)


def work(case):
    """Bytes: inputs once, outputs once.  Operations of stereo: about 40 per
    window term (geometry, divides, Hamming count), for the terms that no
    evaluation order avoids: one 5-term row per hypothesis and per random
    candidate, and the kept plane's 25 K terms."""
    c = dict(case)
    kind = c["kind"]
    if kind in ("depth", "dense", "stereo"):
        maps = 1 if kind == "depth" else c["views"]
        px = c["w"] * c["h"] * maps
        if c.get("mixed"):
            sizes = [a * b for a, b in MIXED_SIZES if a <= c["w"]]
            px = sum(sizes) / len(sizes) * maps
        seen = px / maps * (c["srcs"] + 1 if kind == "depth" else c["views"])
        passes = learned.LEARNED_PASSES if c.get("learned") else 2 * c["sweeps"]
        terms = 15 * passes + 25 * c["srcs"] + (0 if c.get("learned") else 5 * c["hyps"])
        out = {"depth": 20 * px, "dense": 0.02 * px * 27, "stereo": 4 * px}[kind]
        return {"bytes": seen * (4 if kind == "dense" else 1) + out, "flops": 40.0 * terms * px}
    if kind == "fuse":
        px = c["w"] * c["h"] * c["views"]
        # a depth and a colour per pixel; per kept pixel and view checked
        # about 60 f64 operations (two projections)
        return {"bytes": 7 * px + 0.03 * px * 27, "flops": 0.35 * px * c["srcs"] * 60}
    if kind == "sift":
        px = c["w"] * c["h"]
        wide = min(1.0, 1600 / max(c["w"], c["h"])) ** 2 * px
        # two separable blurs (11 and 19 taps) and the next octave, 26
        # comparisons, descriptors of about 1000 samples of 60 operations
        return {"bytes": px * c["channels"] + c["features"] * (16 + 512 + 3),
                "flops": wide * (44 + 4 / 3 * (76 + 26)) + c["features"] * 60000.0}
    if kind == "match":
        n = c["features"] * (0.75 if c["ragged"] else 1)
        pairs = c["frames"] * (c["frames"] - 1) / 2
        return {"bytes": c["frames"] * n * 512 + pairs * n * 0.25 * 8, "flops": pairs * n * n * 128 * 3}
    if kind == "train":
        px = c["n"] * c["w"] * c["h"]
        mac = 9 * (33 * 32 + 4 * 32 * 32 + 32 * 5)
        return {"bytes": px * (96 + 32) + 4 * 8 * 55472, "flops": 2.0 * px * (3 * mac - 9 * 33 * 32)}
    s = min(c["max_dim"] / max(c["w"], c["h"]), 1.0)
    out = c["w"] * s * c["h"] * s
    return {"bytes": c["w"] * c["h"] * c["channels"] + 4 * out,
            "flops": c["channels"] * 4.0 * (c["w"] * c["h"] + c["w"] * c["h"] * s)}


def exact(case, seed):
    if case["kind"] != "train":
        return None
    x, lab = _batch(dict(case), seed)
    return _gradients(learned.load_weights(), x, lab)


def _gradients(params, x, lab):
    """(loss, gradients) of the training step in 64 bits: six 3x3
    convolutions (zero padded, ReLU between), the loss |t - t*| +
    (1 - cos(n, n*)) + 0.1 BCE over valid cells, in the parameter layout
    W[9][cout][cin], b[cout] per layer; padded channels carry none."""
    cin, cout = [48, 32, 32, 32, 32, 32], [32, 32, 32, 32, 32, 16]
    cin_real, cout_real = [33, 32, 32, 32, 32, 32], [32, 32, 32, 32, 32, 5]
    p = torch.from_numpy(np.asarray(params, np.float64)).cuda()
    ws, bs, off = [], [], 0
    for ci, co in zip(cin, cout):
        ws.append(p[off:off + 9 * co * ci].reshape(9, co, ci).clone().requires_grad_())
        off += 9 * co * ci
        bs.append(p[off:off + co].clone().requires_grad_())
        off += co
    n_valid = max(int((lab[..., 4] > 0.5).sum()), 1)
    total = 0.0
    for i in range(x.shape[0]):  # one view at a time: the sums are over views
        a = x[i].double()
        h, w = a.shape[:2]
        for k in range(6):
            pad = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1))
            y = bs[k]
            for tap in range(9):
                y = y + pad[tap // 3:tap // 3 + h, tap % 3:tap % 3 + w] @ ws[k][tap].T
            a = torch.relu(y) if k < 5 else y
        lb = lab[i].double()
        ok = lb[..., 4] > 0.5
        a, lb = a[ok], lb[ok]
        dt = a[:, 0] - lb[:, 0]
        nv = a[:, 1:4]
        cos = (nv * lb[:, 1:4]).sum(1) / (nv.norm(dim=1) + 1e-6)
        hit = (dt.abs() < lb[:, 5]).double()
        bce = torch.nn.functional.binary_cross_entropy_with_logits(a[:, 4], hit, reduction="none")
        loss = (dt.abs() + (1 - cos) + 0.1 * bce).sum() / n_valid
        loss.backward()
        total += float(loss)
    grads = []
    for k in range(6):
        gw, gb = ws[k].grad, bs[k].grad
        gw[:, cout_real[k]:] = 0
        gw[:, :, cin_real[k]:] = 0
        gb[cout_real[k]:] = 0
        grads += [gw.reshape(-1), gb]
    return total, torch.cat(grads).cpu().numpy()
