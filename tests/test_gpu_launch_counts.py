"""The launch counts of a call of more waves than the wave table holds (4096), which runs in chunks:
each chunk ends with its own attempts to hand the last wave's bounces to the whole-path kernel
(before bounces 1 to 3, while two bounces or more are to come)."""
import pytest

import luxion_b200 as lx
from luxion_b200._ffi import default_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waves,chunks", [(5, 1), (4096, 1), (4097, 2)])
@pytest.mark.parametrize("depth,attempts", [(3, 1), (8, 3)])
def test_every_chunk_counts_its_hand_over(waves, chunks, depth, attempts):
    s = lx.random_scene(seed=3, total_tris=4000, num_instances=4, min_tris=500, max_tris=1500, num_emissive=1,
                        num_textures=1, texture_size=16, env_width=16, env_height=8, width=4, height=2, trace_depth=depth)
    r = lx.Renderer(s, default_options(direct_light_sampling=1, spp_per_wave=1))
    r.render(1, waves)
    st = r.stats()
    r.close()
    # a radiance and a shadow launch for each shading launch, and the attempts
    assert st["launches_trace"] == 2 * st["launches_shade"] + chunks * attempts
    assert st["kernel_launches"] == sum(st[k] for k in ("launches_camera", "launches_trace", "launches_shade",
                                                        "launches_accum", "launches_sort"))
