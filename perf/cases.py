"""The work a user has this framework do, as cases that can be timed.

Every case calls the public entry points a program calls: a training step on
device tensors (``DeviceFrame``, ``autograd.render``), the host API of
``pale.Renderer``, batches of views of several scenes (``ViewBatch``), the
photon lookup and ray queries, and the BVH rebuild after density control or
optimizer steps.  Scenes are the synthetic box scenes of the benchmark: beta
surfels in a box of five walls and an area light, cameras on a ring.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from differentiablepointrendering_b200 import autograd
from differentiablepointrendering_b200.device import DeviceFrame, ViewBatch
from differentiablepointrendering_b200.pale import Renderer
from differentiablepointrendering_b200.scene import jitter_target, make_box_scene, make_surfels


def _train(**k):
    c = dict(kind="train", n=1000, views=1, res=64, passes=1, adjoint_passes=1, photons=10000, photon_passes=1,
             depth=4, radius=0.03, rng="decorrelated", estimator="reference", gradients="opacity")
    c.update(k)
    return c


def listed():
    return [
        # the throughput workload of the benchmark: one optimisation step over all views of a 200k-surfel scene
        _train(name="train-box200k", n=200000, views=8, res=512, passes=16, adjoint_passes=16, photons=1000000,
               depth=6, radius=0.01),
        # the benchmark's small configuration, as a differentiable torch operation inside a training loop
        _train(name="autograd-box10k", kind="autograd", n=10000, res=256, passes=4, adjoint_passes=4,
               photons=100000, depth=4, radius=0.02),
        # the smallest step: a preview-sized view at one pass, where launches and latency count
        _train(name="train-small", n=1000, res=64, photons=10000),
        # a gradient request: one 512x512 view at few passes, all seven gradient groups of the gathered image
        _train(name="request-512", n=200000, res=512, passes=4, adjoint_passes=4, photons=1000000, depth=6,
               radius=0.01, estimator="gather", gradients="all"),
        # ragged sizes: odd resolution and passes, seven bounces, all gradient groups of the adjoint, the
        # reference's seeding
        _train(name="train-odd", n=50001, views=3, res=333, passes=5, adjoint_passes=3, photons=300007, depth=7,
               radius=0.013, rng="reference", gradients="all"),
        # a script that leaves every setting at its default (6 x 1M photons, 6 passes, radius 0.01), host arrays
        _train(name="host-defaults", kind="host", n=20000, res=256, passes=6, adjoint_passes=6, photons=1000000,
               photon_passes=6, depth=6, radius=0.01, rng="reference"),
        # several scenes and views of uneven size and passes in one wavefront, forward and adjoint
        dict(name="views-3scenes", kind="views", scenes="30000,100000,250000", photons=500000, depth=6, radius=0.01,
             views="0:0:512:4:6 0:2:256:16:4 1:1:768:4:6 1:5:256:1:6 1:0:512:4:5 2:3:256:32:6 2:4:512:1:6 2:7:768:1:4",
             trace=True, backward=True),
        # one round of a server: forward requests on resident scenes and photon maps
        dict(name="serve-round", kind="views", scenes="10000,139000", photons=500000, depth=6, radius=0.01,
             views="0:0:128:8:6 0:1:512:1:6 0:3:256:2:6 1:2:128:16:6 1:6:256:4:6 1:0:128:1:6", trace=False,
             backward=False),
        # photon lookups at given points, a loaded photon map (fixed-map gradient checks, irradiance baking)
        dict(name="irradiance-100k", kind="irradiance", queries=100000, photons=1000000, radius=0.01),
        # closest-hit queries (picking, visibility, initialisation of new surfels)
        dict(name="rays-500k", kind="rays", n=200000, rays=500000),
        # the rebuild after optimizer steps moved the surfels, and the parameters a loop fetches after it
        dict(name="rebuild-300k", kind="rebuild", n=300000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "autograd", "host", "views", "views", "irradiance", "rays",
                       "rebuild"])
    if kind in ("train", "autograd", "host"):
        photons = _log_int(rng, 10000, 1000000)
        views = rng.choice([1, 1, 2, 3, 4, 6, 8]) if kind == "train" else rng.choice([1, 2])
        res = _log_int(rng, 48, 512)
        # at most an eighth of the largest listed case's camera paths
        most = max(1, min(16, (1 << 22) // (views * res * res)))
        return _train(kind=kind, n=_log_int(rng, 1000, 200000), views=views, res=res, passes=rng.randint(1, most),
                      adjoint_passes=rng.randint(1, most), photons=photons, photon_passes=rng.choice([1, 1, 2]),
                      depth=rng.randint(2, 8), radius=round(min(0.03, 0.01 * math.sqrt(1e6 / photons)), 4),
                      rng=rng.choice(["decorrelated", "decorrelated", "reference"]),
                      estimator=rng.choice(["reference", "reference", "gather"]),
                      gradients=rng.choice(["opacity", "all"]))
    if kind == "views":
        scenes = sorted(_log_int(rng, 5000, 250000) for _ in range(rng.randint(2, 4)))
        views = []
        for _ in range(rng.randint(3, 8)):
            res = _log_int(rng, 64, 640)
            most = max(1, min(16, (1 << 20) // (res * res)))
            views.append(f"{rng.randrange(len(scenes))}:{rng.randrange(8)}:{res}:{rng.randint(1, most)}:{rng.randint(2, 6)}")
        return dict(kind="views", scenes=",".join(map(str, scenes)), photons=_log_int(rng, 100000, 700000), depth=6,
                    radius=0.01, views=" ".join(views), trace=rng.random() < 0.5, backward=rng.random() < 0.6)
    if kind == "irradiance":
        photons = _log_int(rng, 20000, 1500000)
        return dict(kind="irradiance", queries=_log_int(rng, 500, 200000), photons=photons,
                    radius=round(min(0.04, 0.01 * math.sqrt(1e6 / photons)), 4))
    if kind == "rays":
        return dict(kind="rays", n=_log_int(rng, 500, 300000), rays=_log_int(rng, 500, 1000000))
    return dict(kind="rebuild", n=_log_int(rng, 500, 500000))


# ------------------------------------------------------------------ inputs
def _settings(c):
    return {"photons": c["photons"], "bounces": c["depth"], "forward_passes": c["photon_passes"],
            "gather_passes": c["passes"], "adjoint_bounces": c["depth"], "adjoint_passes": c["adjoint_passes"],
            "gather_radius": c["radius"], "seed": 42, "rng_mode": c["rng"], "estimator": c["estimator"],
            "gradients": c["gradients"]}


def _scene(c, points):
    return make_box_scene(c["n"], cameras=c["views"], resolution=c["res"], points=points)


def _parse_views(c):
    return [tuple(int(x) for x in v.split(":")) for v in c["views"].split()]


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("train", "autograd"):
        points = make_surfels(c["n"], seed)
        scene = _scene(c, points)
        # the target: a render of the cloud the optimisation should recover
        t = Renderer.from_scene(scene.with_points(jitter_target(points, seed + 1)), _settings(c))
        tf = DeviceFrame(t)
        target = tf.forward()[0][:, :3].clone()
        torch.cuda.synchronize()
        del tf
        t.close()
        r = Renderer.from_scene(scene, _settings(c))
        f = DeviceFrame(r)
        s = {"r": r, "frame": f, "target": target}
        if kind == "autograd":
            s["params"] = autograd.parameters(r)
        return s
    if kind == "host":
        points = make_surfels(c["n"], seed)
        r = Renderer.from_scene(_scene(c, points), _settings(c))
        rng = np.random.default_rng(seed + 2)
        # an L2 residual image per camera
        dldi = {k: (rng.normal(0.0, 0.1, (c["res"], c["res"], 3)) / (3 * c["res"] ** 2)).astype(np.float32)
                for k in r.get_camera_names()}
        return {"r": r, "dldi": dldi}
    if kind == "views":
        views = _parse_views(c)
        ns = [int(x) for x in c["scenes"].split(",")]
        rs, at = [], []
        for k, n in enumerate(ns):
            sizes = sorted({v[2] for v in views if v[0] == k}) or [64]
            at.append(sizes)
            st = {"photons": c["photons"], "bounces": c["depth"], "forward_passes": 1,
                  "gather_passes": max([v[3] for v in views if v[0] == k] + [1]),
                  "adjoint_bounces": c["depth"],
                  "adjoint_passes": max([v[3] for v in views if v[0] == k] + [1]),
                  "gather_radius": c["radius"], "seed": 42, "rng_mode": "decorrelated", "camera_seeds": "camera"}
            rs.append(Renderer.from_scene(make_box_scene(n, cameras=8, resolutions=sizes,
                                                         points=make_surfels(n, seed + 17 * k)), st))
        batch = ViewBatch(rs, [(s, pos * len(at[s]) + at[s].index(res), p, d) for s, pos, res, p, d in views])
        g = torch.Generator().manual_seed(seed)
        target = (0.25 + 0.1 * torch.randn(batch.pixels, 3, generator=g)).clamp_(0, 1).cuda()
        if not c["trace"]:
            batch.forward_loss()   # resident photon maps
        return {"r": rs, "batch": batch, "target": target, "trace": c["trace"], "backward": c["backward"]}
    rng = np.random.default_rng(seed)
    if kind == "irradiance":
        pos, direction, power, x, nrm = _photons(c, rng)
        r = Renderer.from_scene(make_box_scene(64, points=make_surfels(64, seed)),
                                {"photons": 1024, "bounces": 1, "gather_radius": c["radius"]})
        r.load_photons(pos, power, direction)
        return {"r": r, "x": x, "n": nrm}
    if kind == "rays":
        r = Renderer.from_scene(make_box_scene(c["n"], points=make_surfels(c["n"], seed)), {"photons": 1024})
        o, d = _rays(c, rng)
        return {"r": r, "o": o, "d": d}
    # rebuild: the surfels as an optimizer step left them on the device
    r = Renderer.from_scene(make_box_scene(c["n"], points=make_surfels(c["n"], seed)), {"photons": 1024})
    f = DeviceFrame(r)
    g = torch.Generator().manual_seed(seed)
    grads = {k: (1e-4 * torch.randn(v.shape, generator=g)).cuda() for k, v in f.grads.items()}
    r.optimizer_step({"optimizer_type": "adam"}, grads=grads)
    torch.cuda.synchronize()
    return {"r": r}


def _unit(rng, n):
    v = rng.normal(size=(n, 3))
    return (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)


def _photons(c, rng):
    """Photons on the walls and in the cloud, and lookups near them."""
    n, q = c["photons"], c["queries"]
    pos = rng.uniform(-0.4, 0.4, (n, 3))
    wall = rng.random(n) < 0.5
    axis = rng.integers(0, 3, n)
    pos[wall] *= 0.499 / 0.4
    pos[wall, axis[wall]] = np.where(rng.random(int(wall.sum())) < 0.5, -0.499, 0.499)
    x = pos[rng.integers(0, n, q)] + rng.normal(0.0, 0.5 * c["radius"], (q, 3))
    power = rng.gamma(2.0, 0.5, (n, 3)) / n
    return (pos.astype(np.float32), _unit(rng, n), power.astype(np.float32), x.astype(np.float32), _unit(rng, q))


def _rays(c, rng):
    """Half from inside the box (secondary rays), half from around it."""
    n = c["rays"]
    o = rng.uniform(-0.45, 0.45, (n, 3))
    d = _unit(rng, n)
    out = rng.random(n) < 0.5
    k = int(out.sum())
    e = _unit(rng, k).astype(np.float64) * 1.5
    a = rng.uniform(-0.4, 0.4, (k, 3)) - e
    o[out] = e
    d[out] = (a / np.linalg.norm(a, axis=1, keepdims=True)).astype(np.float32)
    return o.astype(np.float32), d


# --------------------------------------------------------------- one pass
def run(state):
    s = state
    if "params" in s:
        image = autograd.render(s["frame"], s["params"])
        loss = 0.5 * (image[:, :3] - s["target"]).square().mean()
        g = torch.autograd.grad(loss, [s["params"][k] for k in autograd.FIELDS])
        return {"image": image.detach(), "loss": loss.detach(), "grads": g}
    if "frame" in s:
        f = s["frame"]
        loss = f.forward_loss(s["target"])
        g = f.backward()
        return {"ldr": f.ldr, "raw": f.raw, "dldi": f.dldi, "loss": loss, "grads": g}
    if "dldi" in s:
        images = s["r"].render_forward()
        g, _ = s["r"].render_backward(s["dldi"])
        return {"images": images, "grads": g}
    if "batch" in s:
        b = s["batch"]
        if not s["backward"]:
            b.forward_loss(trace_photons=s["trace"])
            return {"ldr": b.ldr, "raw": b.raw}
        loss = b.forward_loss(s["target"], trace_photons=s["trace"])
        return {"ldr": b.ldr, "loss": loss, "grads": [g["opacity"] for g in b.backward()]}
    if "x" in s:
        return s["r"].gather_irradiance(s["x"], s["n"])
    if "o" in s:
        inst, prim, t, alpha, pos = s["r"].trace_rays(s["o"], s["d"])
        return {"inst": inst, "prim": prim, "t": t, "alpha": alpha, "pos": pos}
    s["r"].rebuild_bvh()
    return {"order": s["r"].get_point_order(), "params": s["r"].get_point_parameters()}


# ------------------------------------------------------------------- work
def work(case):
    """Inputs read once and outputs written once; per path at least one
    descent through a binary tree over the surfels (a 20-flop box test per
    level) and one 60-flop surfel test."""
    c, kind = case, case["kind"]
    per = lambda n: 20.0 * math.log2(max(2, n)) + 60.0
    if kind in ("train", "autograd", "host"):
        pix = c["views"] * c["res"] ** 2
        adj = c["adjoint_passes"] if c["estimator"] == "reference" else 0
        paths = pix * (c["passes"] + adj) + c["photons"] * c["photon_passes"]
        return {"bytes": 2.0 * 68 * c["n"] + pix * (12.0 + 48.0), "flops": paths * per(c["n"])}
    if kind == "views":
        views = _parse_views(c)
        ns = [int(x) for x in c["scenes"].split(",")]
        pix = sum(v[2] ** 2 for v in views)
        paths = sum(v[2] ** 2 * v[3] * (2 if c["backward"] else 1) for v in views)
        paths += len(ns) * c["photons"] if c["trace"] else 0
        return {"bytes": 68.0 * sum(ns) * (2 if c["backward"] else 1) + pix * 32.0, "flops": paths * per(max(ns))}
    if kind == "irradiance":
        return {"bytes": 36.0 * c["photons"] + 36.0 * c["queries"], "flops": 10.0 * 25 * c["queries"]}
    if kind == "rays":
        return {"bytes": 68.0 * c["n"] + 52.0 * c["rays"], "flops": c["rays"] * per(c["n"])}
    n = c["n"]
    return {"bytes": 68.0 * n * 2 + 64.0 * n + 4.0 * n, "flops": 60.0 * n}


# ------------------------------------------------- the answers in 64 bits
def exact(case, seed):
    """The lookups and the closest hits in 64-bit arithmetic; the renders
    (Monte Carlo paths through the whole scene) have none."""
    if case["kind"] == "irradiance":
        return _exact_irradiance(case, np.random.default_rng(seed))
    if case["kind"] == "rays" and case["rays"] * float(case["n"]) <= 1.1e11:
        return _exact_rays(case, seed)
    return None


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _exact_irradiance(c, rng):
    pos, direction, power, x, nrm = (torch.from_numpy(a).to(_dev()).double() for a in _photons(c, rng))
    r2 = float(np.float32(c["radius"]) * np.float32(c["radius"]))
    radius = float(np.float32(c["radius"]))
    by_x = torch.argsort(pos[:, 0])
    pos, direction, power = pos[by_x], direction[by_x], power[by_x]
    order = torch.argsort(x[:, 0])
    out = torch.zeros_like(x)
    for part in torch.split(order, 256):
        q, m = x[part], nrm[part]
        lo = int(torch.searchsorted(pos[:, 0].contiguous(), q[:, 0].min() - 1.001 * radius))
        hi = int(torch.searchsorted(pos[:, 0].contiguous(), q[:, 0].max() + 1.001 * radius))
        d2 = (q[:, None, 0] - pos[None, lo:hi, 0]) ** 2
        for a in (1, 2):
            d2 += (q[:, None, a] - pos[None, lo:hi, a]) ** 2
        ok = (d2 <= r2) & (m @ direction[lo:hi].T <= 0.0)
        out[part] = ok.double() @ power[lo:hi] / (math.pi * r2)
    return out.cpu().numpy()


def _exact_rays(c, seed):
    o, d = (torch.from_numpy(a).to(_dev()).double() for a in _rays(c, np.random.default_rng(seed)))
    p = {k: torch.from_numpy(v).to(_dev()).double() for k, v in make_surfels(c["n"], seed).items()}
    unit = lambda v: v / v.norm(dim=1, keepdim=True)
    tu, tv = unit(p["tangent_u"]), unit(p["tangent_v"])
    nrm = unit(torch.linalg.cross(tu, unit(tv - (tv * tu).sum(1, keepdim=True) * tu)))
    tu, tv = tu / p["scale"][:, :1], tv / p["scale"][:, 1:]
    np_, up, vp = ((a * p["position"]).sum(1) for a in (nrm, tu, tv))
    best = torch.full((c["rays"],), math.inf, dtype=torch.float64, device=o.device)
    prim = torch.zeros(c["rays"], dtype=torch.int64, device=o.device)
    step = max(1, min(c["rays"], int(2e8 / c["n"])))
    for a in range(0, c["rays"], step):
        oo, dd = o[a:a + step], d[a:a + step]
        t = (np_ - oo @ nrm.T) / (dd @ nrm.T)
        r2 = (oo @ tu.T + t * (dd @ tu.T) - up).square_()
        r2 += (oo @ tv.T + t * (dd @ tv.T) - vp).square_()
        t.masked_fill_(~((t > 1e-5) & (r2 < 1.0)), math.inf)
        best[a:a + step], prim[a:a + step] = t.min(1)
    # the walls and the light: axis-aligned rectangles (axis, offset, half sizes)
    for ax, off, h in ((2, -0.5, 0.5), (2, 0.5, 0.5), (1, 0.5, 0.5), (0, -0.5, 0.5), (0, 0.5, 0.5), (2, 0.499, 0.125)):
        t = (off - o[:, ax]) / d[:, ax]
        x = o + t[:, None] * d
        others = [k for k in range(3) if k != ax]
        hit = (t > 1e-4) & (x[:, others].abs() <= h).all(1) & (t < best)
        best = torch.where(hit, t, best)
        prim = torch.where(hit, torch.full_like(prim, -1), prim)
    miss = torch.isinf(best)
    x = o + torch.where(miss, torch.zeros_like(best), best)[:, None] * d
    k = prim.clamp(min=0)
    rel = x - p["position"][k]
    r2 = (tu[k] * rel).sum(1) ** 2 + (tv[k] * rel).sum(1) ** 2
    alpha = (1.0 - r2).clamp(min=0.0) ** (4.0 * torch.exp(p["beta"][k]))
    alpha = torch.where((prim < 0) | miss, torch.zeros_like(alpha), alpha)
    t = torch.where(miss, torch.full_like(best, 3.402823466e+38), best)
    pos = torch.where(miss[:, None], torch.zeros_like(x), x)
    return {"inst": None, "prim": None, "t": t.cpu().numpy(), "alpha": alpha.cpu().numpy(), "pos": pos.cpu().numpy()}
