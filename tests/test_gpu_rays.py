"""Caller rays at the batch sizes where lux_trace_rays changes its way: one ray, a warp and one more,
one ray per warp of the grid and one more, the last batch that is spread over the warps and the next,
a full grid, and the sizes around which the copies go through page-locked staging (4 MB of rays, then
of hits), with a remainder of one ray. Rays are independent, so a batch's hits equal those of the
same rays traced in other, small batches (lux_trace_rays_static, whose hits the parity suite
holds against the oracle), word for word.
"""
import numpy as np
import pytest

import luxion_b200 as lx
from luxion_b200 import _ffi
from luxion_b200._ffi import default_options

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[_ffi.BVH_SINGLE_LEVEL, _ffi.BVH_TWO_LEVEL], ids=["single", "two"])
def renderer(request):
    s = lx.random_scene(seed=3, total_tris=30_000, num_instances=12, min_tris=500, max_tris=6000, num_textures=4,
                        texture_size=64, env_width=0, env_height=0, width=64, height=64)
    for k in range(0, s.desc.num_materials, 3):  # some hits are decided by texture alpha
        m = s.desc.materials[k]
        m.albedo_tex, m.alpha_mode, m.alpha_cutoff = 3, _ffi.ALPHA_BLEND, 0.5
    r = lx.Renderer(s, default_options(bvh_layout=request.param))
    yield r
    r.close()


@pytest.mark.parametrize("n", [1, 33, 4144, 4145, 33152, 33153, 131072, 131073, 209716, 262145])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_batches_equal_their_slices(renderer, n, mode):
    g = np.random.default_rng(n + mode)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = g.uniform((-12, 0.2, -12), (12, 8, 12), (n, 3))
    d = g.normal(size=(n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 3] = g.uniform(1.0, 40.0, n)
    rays[:, 7] = np.arange(n, dtype=np.int32).view(np.float32)
    got = renderer.trace_rays(rays, mode, 7)
    step = 50_021
    want = np.concatenate([renderer.trace_rays_static(rays[i:i + step], mode, 7) for i in range(0, n, step)])
    assert np.array_equal(got, want)
    assert np.array_equal(got, renderer.trace_rays(rays, mode, 7))
