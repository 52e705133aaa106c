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
