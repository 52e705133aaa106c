"""The camera gather's photon lookups (lookups without a photon in reach,
short and long ones; records in queue order and grouped by grid cell).

- Images of scenes whose visible surfels and walls are lit by given photons
  against the oracle, over the values that photons contribute to.
- Lookups at known points with known numbers of photons: the camera's
  results equal gather_irradiance's bit for bit (every form of the lookup
  adds the same 32 partial sums in the same way), and both the sums of the
  accepted powers.
"""
import dataclasses
import math

import numpy as np
import pytest

from differentiablepointrendering_b200.pale import Renderer
from differentiablepointrendering_b200.scene import make_box_scene, look_at
from oracle_lib import OracleRenderer

pytestmark = pytest.mark.gpu


def _visible(oracle, scene, n, rng):
    """Closest hits of camera 0 that are not the light's."""
    inv = scene.camera_inv_view[0].astype(np.float64)
    tan = math.tan(math.radians(0.5 * float(scene.camera_fovy[0])))
    d = np.concatenate([tan * rng.uniform(-0.9, 0.9, (n, 2)), -np.ones((n, 1))], 1) @ inv[:3, :3].T
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    inst, _, _, _, x = oracle.trace_rays(np.tile(inv[:3, 3], (n, 1)).astype(np.float32), d.astype(np.float32))
    return x[(inst >= 0) & (inst != len(scene.instance_mesh) - 1)].astype(np.float64)


def _photons(kind, rng, hits):
    if kind == "none":
        pos = hits[:1]                                       # one photon: nearly every lookup finds none
    elif kind == "short":
        pos = hits[rng.integers(0, len(hits), 20000)]        # a few photons per lookup
    elif kind == "edge":
        pos = hits[rng.integers(0, 100, 100 * 200)]          # clusters of about 200 photons: on both sides of 256
    else:
        pos = hits[rng.integers(0, 80, 80 * 4000)]           # thousands per lookup, and photons on the grid's rim
    pos = pos + rng.normal(size=pos.shape) * 0.006
    if kind == "long":
        pos[:500] = rng.choice([-0.5, 0.5], (500, 3))
    d = rng.normal(size=pos.shape)
    return (pos.astype(np.float32), rng.uniform(0.0, 1e-4, pos.shape).astype(np.float32),
            (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))


# 64^2 x 2 paths stay in queue order, 160^2 x 2 are grouped by cell
@pytest.mark.parametrize("res", [64, 160])
@pytest.mark.parametrize("kind", ["none", "short", "edge", "long"])
def test_gather_lookups_match_oracle(gpu, kind, res):
    scene = make_box_scene(1500, cameras=1, resolution=res)
    st = {"photons": 1000, "bounces": 1, "forward_passes": 1, "gather_passes": 2, "gather_radius": 0.02}
    g, o = Renderer.from_scene(scene, st), OracleRenderer(scene, st)
    g.render_forward()
    o.render_forward()
    rng = np.random.default_rng(5)
    photons = _photons(kind, rng, _visible(o, scene, 4000, rng))
    dark = (photons[0], np.zeros_like(photons[1]), photons[2])
    o.load_photons(*dark)
    base = o.render_gather()["camera0_raw"][..., :3]         # the light and nothing else
    g.load_photons(*photons)
    o.load_photons(*photons)
    a = g.render_gather()["camera0_raw"][..., :3] - base
    b = o.render_gather()["camera0_raw"][..., :3] - base
    g.close()
    o.close()
    lit = (b != 0) & (base == 0)                             # values of photons alone
    assert lit.sum() >= (3 if kind == "none" else 600), lit.sum()
    assert np.all(a[(b == 0) & (base == 0)] == 0) or np.mean((a != 0) != (b != 0)) < 1e-3
    # a lookup's sum is within 1e-5 of the oracle's; the layers' weights add
    # the powf of either side (1e-4)
    err, scale = np.abs(a - b)[lit], np.maximum(np.abs(b[lit]), 1e-3 * float(np.abs(b[lit]).mean()))
    assert np.median(err / scale) < 1e-4
    assert np.mean(err / scale < 1e-3) > 0.95
    assert abs(a[lit].mean() - b[lit].mean()) <= 1e-2 * b[lit].mean()


R = 0.02
COUNTS = [0, 1, 2, 7, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 200, 255, 256, 257, 258, 300, 511, 512, 513, 1000, 4095,
          4096, 9000]


def _floor_points(shift):
    """Points on the floor 0.09 apart, the first four in its corners (off the
    diagonal between its two triangles)."""
    c = 0.4985
    pts = [(-c, -c + 0.002), (c, -c + 0.002), (-c, c - 0.002), (c, c - 0.002)]
    pts += [(0.09 * (k % 8) - 0.33 + 0.003 * k, 0.09 * (k // 8) - 0.3) for k in range(len(COUNTS) - 4)]
    return np.array([(x, y, -0.5) for x, y in pts]), np.roll(COUNTS, shift)


def _point_scene(pts, res):
    """The box with a camera per point whose view is the point itself (its
    field of view is below the rounding of the ray's direction)."""
    scene = make_box_scene(0, cameras=1, resolution=res)
    inv, fwd = [], []
    for p in pts:
        off = np.array([-0.5 if p[0] > 0 else 0.5, -0.45 if p[1] > 0 else 0.45, 0.74])
        m = np.linalg.inv(look_at(p + 0.3 * off / np.linalg.norm(off), p, (0.0, 0.0, 1.0)))
        inv.append(m)
        fwd.append(-m[:3, 2])
    n = len(pts)
    return dataclasses.replace(
        scene, camera_inv_view=np.asarray(inv, np.float32), camera_forward=np.asarray(fwd, np.float32),
        camera_fovy=np.full(n, 1e-7, np.float32), camera_size=np.full((n, 2), res, np.uint32),
        camera_names=[f"p{k}" for k in range(n)], camera_adjoint=np.ones(n, bool))


def _clusters(pts, counts, rng):
    """counts[k] photons within 0.9 R of point k, none near its sphere."""
    pos, owner = [], []
    for k, (p, m) in enumerate(zip(pts, counts)):
        v = rng.normal(size=(m, 3))
        v *= 0.9 * R * rng.uniform(0.0, 1.0, (m, 1)) ** (1 / 3) / np.linalg.norm(v, axis=1, keepdims=True)
        pos.append(p + v)
        owner.append(np.full(m, k))
    pos, owner = np.concatenate(pos), np.concatenate(owner)
    order = rng.permutation(len(pos))
    d = rng.normal(size=pos.shape)
    d[:, 2] = np.sign(d[:, 2]) * np.maximum(np.abs(d[:, 2]), 0.1)   # no photon along the floor
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    power = rng.gamma(2.0, 0.5, pos.shape) / len(pos)
    return (pos[order].astype(np.float32), power.astype(np.float32), d.astype(np.float32)), owner[order]


def _expected(renderer, pts, photons, owner):
    """gather_irradiance at the points, checked against the sums of the
    accepted powers, and the radiance a camera sees there."""
    E = renderer.gather_irradiance(pts.astype(np.float32), np.tile(np.float32([[0, 0, 1]]), (len(pts), 1)))
    down = photons[2][:, 2] < 0
    want = np.zeros((len(pts), 3))
    np.add.at(want, owner[down], photons[1][down].astype(np.float64))
    want /= math.pi * float(np.float32(R) * np.float32(R))
    # 9000 positive terms in 32 running sums of at most 282: 300 roundings of 2^-24
    np.testing.assert_allclose(E, want, rtol=2e-5, atol=0)
    floor = np.float32(0.8) * np.float32(0.318309886183790671538)
    return floor * E


# 27 points x 16^2 paths stay in queue order, x 40^2 are grouped by cell
@pytest.mark.parametrize("res", [16, 40])
def test_lookups_at_known_points_are_the_same_in_every_form(gpu, res):
    import torch
    from differentiablepointrendering_b200.device import ViewBatch

    st = {"photons": 1000, "bounces": 1, "forward_passes": 1, "gather_passes": 1, "gather_radius": R,
          "camera_seeds": "camera"}
    rs, want = [], []
    try:
        for k in range(2):
            pts, counts = _floor_points(5 * k)
            r = Renderer.from_scene(_point_scene(pts, res), st)
            rs.append(r)
            r.render_forward()
            photons, owner = _clusters(pts, counts, np.random.default_rng(11 + k))
            r.load_photons(*photons)
            want.append(_expected(r, pts, photons, owner))
            assert (want[k].max(axis=1) > 0).sum() >= len(pts) - 2
            images = r.render_gather()
            for c in range(len(pts)):
                np.testing.assert_array_equal(
                    images[f"p{c}_raw"][..., :3], np.broadcast_to(want[k][c], (res, res, 3)), err_msg=str(counts[c]))
        # both scenes in one call
        n = len(want[0])
        batch = ViewBatch(rs, [(k, c, 1, 0) for c in range(n) for k in (1, 0)])
        batch.forward_loss(trace_photons=False)
        torch.cuda.synchronize()
        for i, img in enumerate(batch.split(batch.raw)):
            np.testing.assert_array_equal(img[..., :3].cpu().numpy(),
                                          np.broadcast_to(want[1 - i % 2][i // 2], (res, res, 3)))
    finally:
        for r in rs:
            r.close()
