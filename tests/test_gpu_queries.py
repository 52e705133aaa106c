"""Ray and lookup queries with host arrays: through the pinned stage that a
render left and through pageable memory, a large query and then a small one
on the same handle, and the device memory they hold afterwards."""
import numpy as np
import pytest

from differentiablepointrendering_b200.pale import Renderer
from differentiablepointrendering_b200.scene import make_box_scene

pytestmark = pytest.mark.gpu

ST = {"photons": 50000, "bounces": 3, "forward_passes": 1, "gather_passes": 1, "gather_radius": 0.03}


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    return (rng.uniform(-0.45, 0.45, (n, 3)).astype(np.float32),
            (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))


def test_a_large_query_gives_its_buffer_back(gpu):
    import torch

    r = Renderer.from_scene(make_box_scene(500, cameras=1, resolution=16), ST)
    try:
        r.trace_rays(*_rays(1000, 1))
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        r.trace_rays(*_rays(4_000_000, 2))     # 208 MB on the device
        assert before - torch.cuda.mem_get_info()[0] < 64 << 20
        o, d = _rays(1_200_000, 3)             # 62 MB: kept for the next call
        r.trace_rays(o, d)
        assert before - torch.cuda.mem_get_info()[0] <= 66 << 20
    finally:
        r.close()


def test_queries_through_the_stage_a_render_left(gpu):
    # two images of 512^2 pixels leave a stage of 8 MB; 250k rays are 6 MB in
    # and 7 MB out, 200k lookups 4.8 MB in; then a few of each
    scene = make_box_scene(3000, cameras=1, resolution=512)
    staged, plain = Renderer.from_scene(scene, ST), Renderer.from_scene(scene, ST)
    rng = np.random.default_rng(4)
    n, m = 50000, 200000
    photons = (rng.uniform(-0.5, 0.5, (n, 3)).astype(np.float32), rng.uniform(0, 1e-4, (n, 3)).astype(np.float32),
               _rays(n, 5)[1])
    try:
        staged.render_forward()
        for r in (staged, plain):
            r.load_photons(*photons)
        for k in (250000, 100, 250000):
            rays, (x, nrm) = _rays(k, k), _rays(min(k, m), k + 1)
            for a, b in zip(staged.trace_rays(*rays), plain.trace_rays(*rays)):
                np.testing.assert_array_equal(a, b)
            for a, b in zip(staged.trace_transmittance(*rays), plain.trace_transmittance(*rays)):
                np.testing.assert_array_equal(a, b)
            e = staged.gather_irradiance(x, nrm)
            np.testing.assert_array_equal(e, plain.gather_irradiance(x, nrm))
            assert (e > 0).any()
        # and against a handle's first, small query of the same rays
        rays = _rays(250000, 250000)
        whole = staged.trace_rays(*rays)
        for lo in (0, 123456, 249000):
            part = plain.trace_rays(rays[0][lo:lo + 1000], rays[1][lo:lo + 1000])
            for a, b in zip(whole, part):
                np.testing.assert_array_equal(a[lo:lo + 1000], b)
    finally:
        staged.close()
        plain.close()
