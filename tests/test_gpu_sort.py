"""Ray sorting's radix passes at the sizes where a tile, a warp or a look-back chain ends.

The sort permutes a bounce's queue; every path is computed as without it, so the image of a
sorted render equals the unsorted one bit for bit exactly when the sorted queue is a permutation
of the queue. The sizes put the first bounce's queue (width * height * samples items) at one
item, at a tile of 4096 items and one to either side, at several tiles with a remainder, and at
more tiles than the launch has blocks; later bounces give smaller queues, an empty one included.
"""
import numpy as np
import pytest

import luxion_b200 as lx
from luxion_b200._ffi import default_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (33, 1, 1), (65, 63, 1), (64, 64, 1), (17, 241, 1), (91, 45, 3),
                                              (255, 257, 2), (1280, 720, 3)])
def test_sorted_render_equals_unsorted(width, height, spp):
    scene = lx.random_scene(seed=5, total_tris=20_000, num_instances=8, min_tris=500, max_tris=8000, num_textures=2,
                            texture_size=64, env_width=64, env_height=32, width=width, height=height, trace_depth=6)
    images = []
    for sort in (0, 1):
        r = lx.Renderer(scene, default_options(env_importance_sampling=1, ray_sorting=sort, spp_per_wave=spp))
        r.render(3, spp)
        r.render(3 + spp, spp)  # the counters are cleared for a second wave
        images.append(r.image_sum())
        counts = r.wave_counts(6)
        r.close()
        images.append(np.array(counts))
    assert np.array_equal(images[0].view(np.uint32), images[2].view(np.uint32))
    assert np.array_equal(images[1], images[3])
