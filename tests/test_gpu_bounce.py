"""Photon and adjoint bounces (mesh pass, surfel walk, shading; rays in queue
order and grouped for the walk) against the oracle, at queue sizes around a
tile, around the grouping threshold and above it."""
import numpy as np
import pytest

from differentiablepointrendering_b200.pale import Renderer
from differentiablepointrendering_b200.scene import make_box_scene
from oracle_lib import OracleRenderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("surfels", [0, 1, 700])
@pytest.mark.parametrize("photons", [1, 257, 16383, 16384, 40000])
def test_photon_pass_matches_oracle(gpu, photons, surfels):
    scene = make_box_scene(surfels, cameras=1, resolution=16)
    st = {"photons": photons, "bounces": 3, "forward_passes": 2, "gather_passes": 1, "gather_radius": 0.05}
    g, o = Renderer.from_scene(scene, st), OracleRenderer(scene, st)
    g.render_forward()
    o.render_forward()
    a, b = g.get_photons(), o.get_photons()
    sg, so = g.stats(), o.stats()
    g.close()
    o.close()
    # the paths agree up to the ulps of sin, cos and pow, which can send a
    # rare path another way (then its later photons shift in the list)
    assert abs(sg["photon_segments"] - so["photon_segments"]) <= 1e-3 * so["photon_segments"]
    n = min(len(a["position"]), len(b["position"]))
    assert abs(len(a["position"]) - len(b["position"])) <= 1 + 1e-3 * n
    first = n // 4          # the first bounces' photons, before any shift
    close = np.abs(a["position"][:first] - b["position"][:first]).max(axis=1, initial=0.0) < 1e-4
    assert first == 0 or close.mean() > 0.99


@pytest.mark.parametrize("photons", [(1 << 19) - 1, 1 << 19, (1 << 19) + 33])
def test_walk_of_many_rays_matches_oracle(gpu, photons):
    # on both sides of the queue size from which the walk has its own build
    test_photon_pass_matches_oracle(gpu, photons, 700)


@pytest.mark.parametrize("gradients", ["opacity", "all"])
# 512, 16200, 33282 and 135200 adjoint paths (the last: lookups apart from the transport)
@pytest.mark.parametrize("res", [16, 90, 129, 260])
def test_adjoint_matches_oracle(gpu, res, gradients):
    scene = make_box_scene(900, cameras=1, resolution=res)
    st = {"photons": 20000, "bounces": 3, "forward_passes": 1, "gather_passes": 1, "adjoint_bounces": 4,
          "adjoint_passes": 2, "gather_radius": 0.04, "rng_mode": "decorrelated", "gradients": gradients}
    g, o = Renderer.from_scene(scene, st), OracleRenderer(scene, st)
    ig = g.render_forward()
    o.render_forward()
    raw = ig["camera0_raw"][..., :3]
    dl = {"camera0": ((raw - 0.5 * raw.mean()) / raw.size).astype(np.float32)}
    gg, _ = g.render_backward(dl)
    go, _ = o.render_backward(dl)
    assert abs(g.stats()["gradient_events"] - o.stats()["gradient_events"]) <= 1e-2 * o.stats()["gradient_events"] + 2
    groups = ("opacity",) if gradients == "opacity" else ("opacity", "beta", "albedo", "scale", "position", "tangent_u",
                                                          "tangent_v")
    for k in groups:
        a, b = np.empty_like(gg[k]), np.empty_like(go[k])
        a[g.get_point_order()] = gg[k]
        b[o.get_point_order()] = go[k]
        a, b = a.reshape(-1).astype(np.float64), b.reshape(-1).astype(np.float64)
        cos = a @ b / (np.linalg.norm(a) * np.linalg.norm(b))
        # one ray that goes another way reshuffles its job's later random
        # numbers; the first passes hold few rays
        assert cos >= 0.99, (k, cos)
    g.close()
    o.close()
