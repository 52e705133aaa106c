"""Closest hits through the traversal nodes against the oracle for the
directions and positions where the node test could lose one: axis-parallel
and nearly parallel rays, negative zeros, every octant, clouds away from the
origin and of another size, few surfels and leaves of several."""
import dataclasses

import numpy as np
import pytest

from differentiablepointrendering_b200.pale import Renderer
from differentiablepointrendering_b200.scene import make_box_scene, make_surfels
from oracle_lib import OracleRenderer

pytestmark = pytest.mark.gpu


def _rays(n, rng, centre, size):
    o = centre + size * rng.uniform(-0.6, 0.6, (n, 3))
    d = rng.normal(size=(n, 3))
    k = n // 2
    a = rng.integers(0, 3, k)
    d[:k] = rng.choice([0.0, -0.0, 1e-7, -1e-7, 1e-5], (k, 3))
    d[np.arange(k), a] = rng.choice([-1.0, 1.0], k)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o.astype(np.float32), d.astype(np.float32)


@pytest.mark.parametrize("leaf", [1, 4])
@pytest.mark.parametrize("n,centre,size", [(1, 0.0, 1.0), (3, 0.0, 1.0), (4000, 0.0, 1.0), (4000, 7.3, 1.0),
                                           (4000, -20.0, 40.0)])
def test_closest_hits_match_oracle(gpu, n, centre, size, leaf):
    pts = make_surfels(n, 3)
    pts["position"] = (centre + size * pts["position"]).astype(np.float32)
    pts["scale"] = (np.float32(2.0 * size) * pts["scale"]).astype(np.float32)
    scene = make_box_scene(n, points=pts)
    st = {"photons": 64, "bounces": 1, "gather_radius": 0.2 * max(size, 1.0), "leaf_size": leaf}
    g, o = Renderer.from_scene(scene, st), OracleRenderer(scene, st)
    rays = _rays(20000, np.random.default_rng(1), centre, size)
    gi, gp, gt, ga, gx = g.trace_rays(*rays)
    oi, op, ot, oa, ox = o.trace_rays(*rays)
    go, oo = g.get_point_order(), o.get_point_order()
    g.close()
    o.close()
    assert np.mean(gi == oi) >= 0.9995
    s = (gi == oi) & (gi == scene.instance_mesh.shape[0])
    assert s.any() or n < 10
    assert not s.any() or np.mean(go[gp[s]] == oo[op[s]]) >= 0.9995
    hit = (gi == oi) & (gi >= 0)
    np.testing.assert_allclose(gt[hit], ot[hit], rtol=1e-5, atol=1e-6 * max(1.0, size))


def test_hits_on_the_planes_of_boxes_away_from_the_origin(gpu):
    # surfels whose box has an x bound that half precision holds exactly, and
    # rays along z whose origin lies on that plane, within the box in y and z:
    # the plane's distance is zero, and an error of o / d must not make it
    # negative
    h = np.arange(16.0, 64.0, 0.125, dtype=np.float32)
    h = np.concatenate([h, -h])
    side = np.where(np.arange(h.size) % 2 == 0, np.float32(1), np.float32(-1))
    x = (h - side * np.float32(0.0035)).astype(np.float32)
    s = (np.abs(h - x) * np.float32(1.00003)).astype(np.float32)
    assert np.array_equal((x + side * (np.float32(1.0001) * s)).astype(np.float32), h)
    n = h.size
    y = np.linspace(-0.4, 0.4, n)
    pts = make_surfels(n, 3)
    pts["position"] = np.stack([x, y, np.zeros(n)], 1).astype(np.float32)
    pts["tangent_u"] = np.tile(np.float32([[1, 0, 0]]), (n, 1))
    pts["tangent_v"] = np.tile(np.float32([[0, 1, 0]]), (n, 1))
    pts["scale"] = np.stack([s, np.full(n, 5e-4, np.float32)], 1)
    scene = make_box_scene(n, points=pts)
    st = {"photons": 64, "bounces": 1, "gather_radius": 2.0, "leaf_size": 1}
    g, o = Renderer.from_scene(scene, st), OracleRenderer(scene, st)
    rays = (np.stack([h, y, np.full(n, -5e-4)], 1).astype(np.float32), np.tile(np.float32([[0, 0, 1]]), (n, 1)))
    gi, gp, gt, _, _ = g.trace_rays(*rays)
    oi, op, ot, _, _ = o.trace_rays(*rays)
    go, oo = g.get_point_order(), o.get_point_order()
    g.close()
    o.close()
    assert np.all(oi == scene.instance_mesh.shape[0]) and np.array_equal(oo[op], np.arange(n))
    np.testing.assert_array_equal(gi, oi)
    np.testing.assert_array_equal(go[gp], oo[op])
    np.testing.assert_array_equal(gt, ot)


@pytest.mark.parametrize("instances", [31, 32, 33, 65, 100])
def test_meshes_of_many_instances_match_oracle(gpu, instances):
    # instances are taken 32 at a time: boxes first, then each ray its own
    rng = np.random.default_rng(instances)
    scene = make_box_scene(200, points=make_surfels(200, 3))
    m = np.tile(np.eye(4), (instances, 1, 1))
    for k in range(instances):
        q = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        m[k, :3, :3] = q * rng.uniform(0.02, 0.3)
        m[k, :3, 3] = rng.uniform(-0.5, 0.5, 3)
    m[-1] = scene.object_to_world[-1]                      # the light
    first = [0] * (instances - 1)
    scene = dataclasses.replace(
        scene, instance_mesh=np.asarray(first + [scene.instance_mesh[-1]], np.uint32),
        instance_material=np.asarray(first + [scene.instance_material[-1]], np.uint32),
        object_to_world=m.astype(np.float32), world_to_object=np.linalg.inv(m).astype(np.float32), instance_names=[])
    st = {"photons": 64, "bounces": 1, "gather_radius": 0.1}
    g, o = Renderer.from_scene(scene, st), OracleRenderer(scene, st)
    rays = _rays(20000, rng, 0.0, 1.0)
    gi, gp, gt, _, _ = g.trace_rays(*rays)
    oi, op, ot, _, _ = o.trace_rays(*rays)
    g.close()
    o.close()
    assert len(np.unique(oi)) > instances // 2
    assert np.mean(gi == oi) >= 0.9995
    hit = (gi == oi) & (gi >= 0)
    np.testing.assert_allclose(gt[hit], ot[hit], rtol=1e-5, atol=1e-6)
