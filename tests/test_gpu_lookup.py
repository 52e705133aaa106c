"""The camera gather's photon lookups (lookups without a photon in reach,
short and long ones; records in queue order and grouped by grid cell)
against the oracle on identical photons."""
import numpy as np
import pytest

from differentiablepointrendering_b200.pale import Renderer
from differentiablepointrendering_b200.scene import make_box_scene
from oracle_lib import OracleRenderer

pytestmark = pytest.mark.gpu


def _photons(kind, rng):
    if kind == "none":
        n, pos = 1, np.array([[0.45, 0.45, -0.45]])          # one photon, far from most of the view
    elif kind == "short":
        n = 40000                                            # a few photons per lookup
        pos = rng.uniform(-0.5, 0.5, (n, 3))
    elif kind == "edge":
        n = 120000                                           # around the boundary between short and long lookups
        pos = rng.normal(size=(n, 3)) * 0.08
    else:
        n = 150000                                           # thousands per lookup, and photons on the grid's rim
        pos = rng.normal(size=(n, 3)) * 0.03
        pos[:500] = rng.choice([-0.5, 0.5], (500, 3))
    d = rng.normal(size=(n, 3))
    return (pos.astype(np.float32), rng.uniform(0.0, 1e-4, (n, 3)).astype(np.float32),
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
    photons = _photons(kind, np.random.default_rng(5))
    g.load_photons(*photons)
    o.load_photons(*photons)
    a = g.render_gather()["camera0_raw"][..., :3]
    b = o.render_gather()["camera0_raw"][..., :3]
    g.close()
    o.close()
    # a lookup's sum is within 1e-5 of the oracle's; the layers' weights add
    # the powf of either side (1e-4)
    err, scale = np.abs(a - b), np.maximum(np.abs(b), 1e-3 * max(1e-3, float(np.abs(b).mean())))
    assert np.median(err / scale) < 1e-4
    assert np.mean(err / scale < 1e-3) > 0.95
    assert abs(a.mean() - b.mean()) <= 1e-2 * abs(b.mean()) + 1e-12
